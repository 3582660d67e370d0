// Nearest-code search (nearest.cu).
#pragma once
#include "common.cuh"

namespace ncmb {
// idx_out[(r / out_tlen) * out_stride + out_off + r % out_tlen] = argmin_j |x_r - E_j|^2 (lowest index among equals).
// x [rows][D], E [V][D], all device memory. E is a model weight: its prepared copies are kept, keyed by address.
void nearest_codes(const float *x, const float *E, int64_t rows, int V, int D, int *idx_out, int out_tlen, int out_stride, int out_off);
void nearest_forget_weights();
void nearest_forget_range(const void *p, size_t bytes);
} // namespace ncmb
