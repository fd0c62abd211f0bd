// hx_gpt2_step.cuh -- the layers of one GPT-2 token in one launch (hx_gpt2_step.cu).
#pragma once
#include "hx_common.cuh"

struct HxGpt2LayerDev {                     // one layer, in device memory; order: qkv, proj, c_fc, second proj
    const uint8_t* t16[4];                  // A-fragment order (hx_repack_t16)
    const float* bias[4]; float ts[4];
    const float *ln1g, *ln1b, *ln2g, *ln2b;
};
struct HxGpt2Step {
    const HxGpt2LayerDev* layers; int n_layers;
    const float *emb, *wpe; const int *tok, *pos;           // token at *pos
    float *kc, *vc; int cap;                                // [layer][head][cap][64]
    float* x_out;                                           // [d_model] residual stream behind the last layer
    float eps, scale;
    int* err;                                               // set when a bounded wait ran out
    unsigned wait_ns; int stall;                            // limit of a wait; 1: begin with a wait for something that nothing does (tests)
};
bool hx_gpt2_step_fits(const hx_config& c, int kv_cap);
int hx_gpt2_step_launch(const HxGpt2Step& p, int d_model, cudaStream_t st, bool pdl);
