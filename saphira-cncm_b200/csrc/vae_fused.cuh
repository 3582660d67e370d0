// The VQ-VAE's transformer stacks in one kernel (vae_fused.cu).
#pragma once
#include "common.cuh"

namespace ncmb {
struct VaeStackIO {
    const int *ids = nullptr; const float *wte = nullptr;    // token rows [B][T] (device) embedded with wte, or ...
    const float *x = nullptr;                                // ... latents [B][T][64]
    const float *wpe = nullptr;                              // optional position rows [T][64]
    const float *lnf = nullptr;                              // gain of the final LayerNorm, or null for none
    float *y = nullptr;                                      // latents out [B][T][64], or ...
    const float *out_w = nullptr; int V = 0; int *tok = nullptr;   // ... argmax over the V <= 64 rows of out_w
};
// whether the stack (embedding width D, `heads` heads, rows of T tokens, no attention window) runs as one kernel
bool vae_stack_supported(const std::vector<BlockWeights> &layers, int D, int heads, int T, int window);
void vae_stack(const std::vector<BlockWeights> &layers, int heads, int B, int T, const VaeStackIO &io);
} // namespace ncmb
