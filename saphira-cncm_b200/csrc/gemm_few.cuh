// Products of a weight matrix with few rows (gemm_few.cu): decode steps and the first levels of a generate.
#pragma once
#include "common.cuh"

namespace ncmb {

// y = act(x W^T + bias) for 2 to 640 rows of x. With `part` set, K may be cut into slices whose raw sums go to part[slice][row][N] (no
// bias, no activation); the consumer adds them in slice order.
//   Up to FEW_F32_ROWS rows: fp32 multiply-adds. x1 and y are fp32 (x2, y_lo null); W is streamed as it is, or as its exact bf16 copy W16
//     where there is one; glu: gate rows, then up rows, y (or the columns of part, in pairs) per unit.
//   More: x is an fp16 pair, W its pair in the cache of the fp16-pair engine, y fp32 (y_lo null) or a pair; glu: W holds interleaved
//     gate / up rows and y has N / 2 columns.
constexpr int FEW_F32_ROWS = 16;
struct FewGemm {
    const void *x1, *x2; int64_t ldx;        // elements
    const float *W; int M, N, K;
    const unsigned short *W16 = nullptr;
    const float *bias = nullptr; int act = ACT_NONE, glu = 0;
    float *y = nullptr, *y_lo = nullptr; int64_t ldy = 0;
    float *part = nullptr; int max_slices = 1;
};
// Five 128-row tiles: up to there the K slices and the folded reductions win over 128 x N tiles that leave SMs idle (config 2, 38 rows
// x 16 tokens: 4% of a generate; a Qwen2 decode step of 300 rows 3.81 -> 2.31 ms, of 600 rows 5.10 -> 3.60); at 1216 rows they are even,
// at 3000 they lose 10%.
constexpr int FEW_MAX_ROWS = 640;
bool gemm_few_supported(int64_t M, int N, int K, const void *W);
int gemm_few_slices(int M, int N, int K, int max_slices);      // slices gemm_few() will use for a call with `part`
void gemm_few(const FewGemm &g);
// y = x W^T + bias with many columns (a vocabulary): up to 64 rows on gemm_few(), more on the fp16-pair engine's wide tiles
// (128 rows x 151936 columns of 896: 178 us against 368)
void few_head(const void *x1, const void *x2, int rows, const float *W, const unsigned short *W16, const float *bias, int N, int K, float *y);

// x[row] += bias + sum_s part[s][row] (S slices of rows x C), then norm(x) as an fp16 pair, or in fp32 where y2 is null (ln_kind 0: no
// norm; 1 LayerNorm; 2 RMSNorm). S = 0: only the norm.
void few_reduce_norm(float *x, const float *part, int S, const float *bias, int rows, int C, int ln_kind, const float *ln_w, const float *ln_b,
                     float eps, void *y1, void *y2);

// An up-projection with so few 128-row tiles that most SMs would idle is cut into slices too (GPT-2's 3072 rows are 24 tiles:
// 15.5 us at 64 tokens against 8 with the kernel that adds the slices); 1 = store the result directly.
int few_up_slices(int M, int N, int K, int max_slices);
void few_reduce_act(const float *part, int S, int rows, int N, const float *bias, int act, int glu, void *y1, void *y2);

// q | k | v = bias + sum_s part[s][row], rotated (tables may be null), q to q[row * ldq], k | v to q as well (kv_self) and / or
// to the cache row kv + (row / rps) * seq_pitch + (row % rps) * pitch + *step_d * step
struct FewQkv {
    const float *part; int S, rows, H, Hkv; const float *bias;
    const float *cos_t = nullptr, *sin_t = nullptr; const int *pos = nullptr, *step_d = nullptr; int64_t pos_step = 0;
    float *q; int64_t ldq; int kv_self = 0;
    float *kv = nullptr; int rps = 1; int64_t seq_pitch = 0, pitch = 0, step = 0;
    int hd = 64;
};
void few_reduce_qkv(const FewQkv &a);

// Decode attention that takes q and the new token's k | v from the slices itself and appends k | v to the cache
// (attention_decode.cu): one query per row, cached keys only, head dim 64, up to eight query heads per kv head.
bool attention_fused_supported(const AttnArgs &a);
void attention_fused(const AttnArgs &a, const FewQkv &q);

// the fp16 pair of a static weight matrix [N][K], its scale and whether the second half is all zero (gemm_h3.cu)
struct H3Weights { const unsigned short *v1, *v2; float scale; bool v2_zero; };
H3Weights gemm_h3_weights(const float *W, int64_t n);

} // namespace ncmb
