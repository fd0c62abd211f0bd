// hx_gemm_tc.cuh -- interface of the tcgen05 block-scaled NVFP4 GEMMs: raw E2M1 columns (hx_gemm_tc.cu) and the digit columns of
// the chunk paths (hx_gemm_dig.cu).
#pragma once
#include "hx_common.cuh"

#define HX_T128_CELL 18432         // one (128-row tile, 256-column group) cell of A: 16384 B codes + 4 x 512 B scales
#define HX_TC_STAGES 4
#define HX_TC_MAX_SK 8             // raw GEMM: 64-column steps per ring stage (4 or 8)
#define HX_TC_RES_CELLS 4          // digit cells of a (part of K, token group) that fit beside the ring of weight cells
#define HX_TC_DIGITS 10            // balanced base-9 digits (-4 .. 4, all E2M1 values) of a 30-bit magnitude per activation
#define HX_TC_MAX_TOK 24           // tokens per group: digit d of token t is column 24 d + t, 240 columns per MMA
#define HX_TC_GROUP_COLS (HX_TC_DIGITS * HX_TC_MAX_TOK)
#define HX_TC_DIGIT_UNIT 536870912.0f      // 2^29: the integer a digit vector spells is |x| / scale * 2^29 < 2^30 < (9^10 - 1) / 2

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
//   y = act(col_scale[t] * ts(row) * sum_d 9^(9-d) D[row][group of t][24 d + t % 24] + bias[row])
struct HxGemmDig {
    const uint8_t* a;              // T128 weight cells [tile][cell of 256 columns]
    const uint8_t* b;              // digit cells [cell of 256 columns][token group]: 240 rows of 128 swizzled bytes
    int rows, ntiles, kcells, ntok;
    const float* col_scale;        // [ntok] scale of each token's digit integer (a power of two)
    float* out; int ld_out;        // token-major output
    float* acc;                    // K in more than one block: the sums so far of residual linears (shape of out) and of SwiGLU ([ntok][ntiles * 128])
    int resid;                     // 1: add to out instead of storing
    float ts[3]; int bound0, bound1;   // per-row tensor scale: rows < bound0 ts[0], < bound1 ts[1], else ts[2]
    int pair64;                    // 1: ts[0] for rows with (row % 128) < 64, ts[1] for the others (gate/up tiles)
    int swiglu;                    // 1: tiles hold 64 gate + 64 up rows; out[t][tile * 64 + r] = silu(gate_r) * up_r, rows = hidden size
    const float* bias;             // [rows] or null; gelu: gelu_new after it (plain linears)
    int gelu;
    int* err;                      // set when a bounded wait ran out
    int groups, nblk;              // filled in by the launch: token groups, blocks of K
};
int hx_gemm_dig_launch(HxGemmDig g, cudaStream_t st);
int hx_gemm_dig_prepare();         // kernel attributes; call once outside stream capture
