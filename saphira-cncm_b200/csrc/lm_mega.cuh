// Persistent decode-step kernel of the decoder LMs (lm_mega.cu).
#pragma once
#include "common.cuh"

namespace ncmb {

struct MegaLayer { const float *ln1w, *ln1b, *qkvb, *ob, *ln2w, *ln2b, *fcb, *pb; float *kv; };

// What the kernel needs of a model, laid out once: every CTA's weight rows of all layers, in the order it uses them, as one
// stream (bf16 where every matrix holds bf16 values, else fp32).
struct MegaModel {
    bool ready = false, w16 = false;
    int grid = 0;
    void *stream_w = nullptr;             // [CTA][layer][qkv pairs | o rows | up pairs or rows | down rows]
    long long *stream_off = nullptr;      // device: byte offset of each CTA's stream
    const void *head_w = nullptr;         // vocabulary projection [V][C], fp32 or bf16
};
struct MegaShape { int B, C, H, nkv, I, NL, V; int gated; };
bool lm_mega_supported(const MegaShape &s, int hd, bool qk_norm);
int lm_mega_ring_need(const MegaShape &s, int esz, int g);       // host arithmetic only
void lm_mega_pack(MegaModel &m, const MegaShape &s, const std::vector<BlockWeights> &blocks, const float *wte, const unsigned short *wte16);
void lm_mega_free(MegaModel &m);

struct MegaArgs {
    MegaShape s;
    int norm;                             // 1 LayerNorm, 2 RMSNorm
    int act;
    float eps, eps_f;                     // block norms / final norm
    const MegaLayer *layers;              // device array [NL]
    const float *wte, *wpe, *lnfw, *lnfb, *cosb, *sinb;
    float *logits;
    const int *ids, *posmat;
    const int *step_d;                    // tokens finalised so far (v); this step's position is posmat[v + pos_base]
    int pos_base;
    uint2 *ll;                            // exchange buffers, zeroed before the first step of a generate: lm_mega_exchange_words() words
    int *err;
};
size_t lm_mega_exchange_words(const MegaShape &s);
void lm_mega_enable(int on);
bool lm_mega_enabled();
void lm_mega_launch(const MegaModel &m, const MegaArgs &a);     // on stream(); fatal when the cooperative launch is refused

} // namespace ncmb
