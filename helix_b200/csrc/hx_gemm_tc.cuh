// hx_gemm_tc.cuh -- interface of the tcgen05 block-scaled NVFP4 GEMMs: raw E2M1 columns (hx_gemm_tc.cu) and the digit columns of
// the chunk paths (hx_gemm_dig.cu).
#pragma once
#include "hx_common.cuh"

#define HX_T128_CELL 18432         // one (128-row tile, 256-column group) cell of A: 16384 B codes + 4 x 512 B scales
#define HX_TC_STAGES 4
#define HX_TC_MAX_SK 8             // raw GEMM: 64-column steps per ring stage (4 or 8)
#define HX_TC_RES_CELLS 16         // digit cells of a (part of K, token group) that a CTA keeps at most (as many as fit beside the ring of weight cells)
#define HX_TC_DIGITS 8             // base-13 digits of a 29-bit signed integer per activation, digit values 0, 1, 2, 3, 4, 6, 8 and their negatives
#define HX_TC_MAX_TOK 26           // tokens per group at most: digit d of token t is column 16 (t / 2) + 2 d + t % 2, up to 208 columns per MMA
// Bytes of a digit cell: 1024 per token (8 swizzled rows of 128), then the column scales of the first and of the second 128 columns of K: 512 bytes
// per 128 digit columns each.
#define HX_TC_DSF(G) ((G) > 16 ? 1024 : 512)
#define HX_TC_DCELL(G) ((G) * 1024 + ((G) > 16 ? 2048 : 1024))
#define HX_TC_DIGIT_UNIT 134217728.0f      // 2^27: the integer is |x| / (scale of the block) * 2^27 <= 2^28

struct HxGemmTC {                  // raw GEMM
    const uint8_t* a;              // T128 cells, [tile][kstep]
    const uint8_t* b;              // B cells, [256-column group of K]: ncols x 128 B swizzled codes + 4 x 512 B scale chunks
    float* y;                      // [rows][ncols]
    int rows, ntiles, ksteps, ncols, stage_ksteps;
    int* err;                      // set when a bounded wait ran out
};
int hx_gemm_tc_launch(const HxGemmTC& g, cudaStream_t st);
size_t hx_gemm_tc_smem(int ncols, int stage_ksteps);

// A linear of a chunk: out[t * ld_out + row] = resid ? out + y : y with
//   y = act(col_scale[t] * ts(row) * 13^7 * sum_d 13^-d D_d[row][t] + bias[row])
struct HxGemmDig {
    const uint8_t* a;              // T128 weight cells [tile][cell of 256 columns]
    const uint8_t* b;              // digit cells [cell of 256 columns][token group] of HX_TC_DCELL(tokens of a group) bytes
    int rows, ntiles, kcells, ntok;
    const float* col_scale;        // [ntok] scale of each token's digits (a power of two)
    float* out; int ld_out;        // token-major output
    float* acc;                    // K in more than one block: the sums so far of residual linears (shape of out) and of SwiGLU ([ntok][ntiles * 128])
    int resid;                     // 1: add to out instead of storing
    float ts[3]; int bound0, bound1;   // per-row tensor scale: rows < bound0 ts[0], < bound1 ts[1], else ts[2]
    int pair64;                    // 1: ts[0] for rows with (row % 128) < 64, ts[1] for the others (gate/up tiles)
    int swiglu;                    // 1: tiles hold 64 gate + 64 up rows; out[t][tile * 64 + r] = silu(gate_r) * up_r, rows = hidden size
    const float* bias;             // [rows] or null; gelu: gelu_new after it (plain linears)
    int gelu;
    int* err;                      // set when a bounded wait ran out
    int group, groups, nblk, res, stages;  // filled in by the launch: tokens per group, groups, blocks of K, resident digit cells, ring of weight cells
};
// Tokens per group of a chunk of n tokens: as few groups as possible, all of the same size (even: columns of an MMA come in
// sixteens).  With groups of the full size a remainder costs as much as a whole group: 64 tokens are three of 22, not 26 + 26 + 12.
inline int hx_gemm_dig_group(int n) {
    const int k = (n + HX_TC_MAX_TOK - 1) / HX_TC_MAX_TOK;
    return ((n + k - 1) / k + 1) & ~1;
}
int hx_gemm_dig_launch(HxGemmDig g, cudaStream_t st);
int hx_gemm_dig_prepare();         // kernel attributes; call once outside stream capture
