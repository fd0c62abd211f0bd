// hx_gpt2_step.cu -- the layers of one GPT-2 token in one launch: a cluster of sixteen CTAs, vectors exchanged through
// distributed shared memory.
//
// Replaces, for one token, the launch sequence of forward_layer_gpt2 (helixc/runtime/gpt2_infer.c:1131-1193) with a KV cache:
// LayerNorm -> qkv (+bias) -> attention -> proj (+bias, residual) -> LayerNorm -> c_fc (+bias, gelu_new) -> proj (+bias,
// residual).  The lm_head follows as a launch of its own over all SMs.
//
// What bounds a token of this size (48 MB of packed weights in the layers, L2-resident between tokens) is the chain of
// sixty dependent exchanges.  Seventy-two launches cost 4 us each; a hand-over between CTAs through L2 costs about 1.2 us; a
// store into the shared memory of another CTA of the cluster arrives in about 0.3.  A layer at D = 768 takes 25 500
// cycles (13 us) on sixteen SMs: 12 000 for the rows, 8000 for LayerNorms and f16 terms, 5500 for attention; the hand-overs that more
// SMs would put through L2 cost more than their arithmetic saves, so the layers run on one cluster:
//  * every CTA owns a sixteenth of the rows of each linear; its weights stream through two shared-memory buffers by bulk
//    copies, a phase ahead;
//  * a warp takes sixteen rows and 256 columns at a time: codes decoded by cvt.f16x2.e2m1x2, times their scale (exact in
//    f16), mma.sync m16n8k16 against the input as three f16 terms (33 bits of the largest element) in three of the eight
//    columns.  The decode engines' tcgen05 form needs 128-row tiles: eighteen of them do not share out over sixteen CTAs.
//    (A half-warp per row in f32 was bound by the f16 -> f32 conversions: 20 000 of a layer's 38 000 cycles.)
//  * results leave as 8-byte (value, epoch) pairs stored into all sixteen CTAs (q, k, v: into the head's CTA), and the
//    reader polls its own shared memory until the epoch of the layer shows up.  An aligned 8-byte store is single-copy
//    atomic, so a matching epoch proves the value.  No buffer is written for the next layer before every CTA has read this
//    layer's: each phase needs rows of all CTAs, so nobody is more than a phase ahead;
//  * attention: one CTA per head.
// Waits are bounded; after one that ran out the CTA goes on with what is there, raises *err and the call reports it.
#include "hx_tc.cuh"
#include "hx_kernels.cuh"
#include "hx_persist.cuh"
#include "hx_gpt2_step.cuh"
#include <cuda_fp16.h>

using namespace hxtc;

namespace {

constexpr int G2_CTAS = 16, G2_WARPS = 16, G2_CT = G2_WARPS * 32, G2_THREADS = G2_CT + 32;
constexpr int G2_CAP = 2048;                          // cached positions at most (scores in shared memory)

__device__ __forceinline__ void g2_sync() { asm volatile("bar.sync 1, %0;" :: "n"(G2_CT) : "memory"); }
__device__ __forceinline__ void g2_send(uint32_t addr, float v, unsigned ep) {
    const unsigned long long w = ((unsigned long long)ep << 32) | (unsigned long long)__float_as_uint(v);
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" :: "r"(addr), "l"(w) : "memory");
}
__device__ __forceinline__ float g2_wait(const unsigned long long* p, unsigned ep, volatile int* ab, unsigned limit_ns) {
    unsigned long long w = 0;
    const uint32_t a = s_u32(p);
    (void)mb_bounded([&] {
        asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(w) : "r"(a) : "memory");
        return (unsigned)(w >> 32) == ep || *ab != 0;
    }, ab, limit_ns);
    return __uint_as_float((unsigned)w);
}
__device__ __forceinline__ float g2_gelu(float x) {   // gpu_gelu_stable_kernel.hx:15-28
    const float inner = 0.7978846f * (x + (0.044715f * (x * x * x))), two = 2.0f * inner;
    const float sgn = inner < 0.0f ? -1.0f : 1.0f;
    const float e = __expf(-(sgn * two));
    const float th = sgn * ((1.0f - e) / (1.0f + e));
    return 0.5f * x * (1.0f + th);
}
__device__ __forceinline__ void g2_cvt8(uint32_t w, uint32_t (&h)[4]) {       // eight codes -> four pairs of halves
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\tmov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\tcvt.rn.f16x2.e2m1x2 %1, b1;\n\tcvt.rn.f16x2.e2m1x2 %2, b2;\n\tcvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3]) : "r"(w));
}
__device__ __forceinline__ uint32_t g2_scale2(uint32_t s) { uint32_t h; asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"((unsigned short)s)); return h; }
__device__ __forceinline__ uint32_t g2_mul2(uint32_t a, uint32_t b) { uint32_t d; asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ void g2_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint2 b) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b.x), "r"(b.y));
}
// where the first term of element k of the input lies among the halves (the next two 16 and 32 behind): a B fragment of an
// MMA is eight consecutive bytes per lane (hx_repack_t16 pairs the elements of two blocks the same way)
__device__ __forceinline__ int g2_place(int k) {
    const int e = k & 127, blk = e >> 4, j = e & 15, m = (blk & ~1) | (j >> 3);
    return ((k >> 7) * 8 + m) * 48 + (((j >> 2) & 1) << 1 | (blk & 1)) + (j & 3) * 4;
}
// sixteen rows times `n` cells of 128 columns (T16: 1024 bytes of codes in A-fragment order, eight scales per row).  A weight
// is code times scale, exact in f16; the input is three f16 terms in columns 0 .. 2.
__device__ __forceinline__ void g2_cells(const uint8_t* cell, int n, const __half* x, float& lo, float& hi) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    float c[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 2
    for (int i = 0; i < n; i++, cell += HX_T16_CELL, x += 8 * 48) {
        const uint4 qa = *reinterpret_cast<const uint4*>(cell + lane * 16), qb = *reinterpret_cast<const uint4*>(cell + 512 + lane * 16);
        const uint2 sa = *reinterpret_cast<const uint2*>(cell + 1024 + g * 8), sb = *reinterpret_cast<const uint2*>(cell + 1024 + (g + 8) * 8);
        const uint32_t wa[4] = {qa.x, qa.y, qa.z, qa.w}, wb[4] = {qb.x, qb.y, qb.z, qb.w};
#pragma unroll
        for (int p = 0; p < 4; p++) {
            uint32_t a[4], b[4];
            g2_cvt8(wa[p], a); g2_cvt8(wb[p], b);
            const uint32_t sA = g2_scale2((p < 2 ? sa.x : sa.y) >> (16 * (p & 1))), sB = g2_scale2((p < 2 ? sb.x : sb.y) >> (16 * (p & 1)));
            uint2 x0 = make_uint2(0u, 0u), x1 = make_uint2(0u, 0u);
            if (g < 3) {
                x0 = *reinterpret_cast<const uint2*>(x + (2 * p * 3 + g) * 16 + t * 4);
                x1 = *reinterpret_cast<const uint2*>(x + ((2 * p + 1) * 3 + g) * 16 + t * 4);
            }
            g2_mma(c, g2_mul2(a[0], sA), g2_mul2(b[0], sB), g2_mul2(a[1], sA), g2_mul2(b[1], sB), x0);
            g2_mma(d, g2_mul2(a[2], sA), g2_mul2(b[2], sB), g2_mul2(a[3], sA), g2_mul2(b[3], sB), x1);
        }
    }
    // columns 0 and 1 of rows g, g + 8 are with the lanes t == 0, column 2 with t == 1
#pragma unroll
    for (int q = 0; q < 4; q++) c[q] += d[q];
    const float n0 = __shfl_down_sync(0xffffffffu, c[0], 1), n2 = __shfl_down_sync(0xffffffffu, c[2], 1);
    constexpr float k1 = 1.0f / 2048.0f, k2 = k1 * k1;
    lo = c[0] + c[1] * k1 + n0 * k2;
    hi = c[2] + c[3] * k1 + n2 * k2;
}

template <int NB> struct G2Smem {
    static constexpr int D = 256 * NB;
    static constexpr int WB = 36 * D * D / 256;       // bytes of the largest phase: 4 D / 16 rows of D, or D / 16 rows of 4 D
    uint8_t w[2][WB];
    unsigned long long xa[D], xb[D], ctx[D], h[4 * D], qkv[192];
    static constexpr int XS = 6 * D > G2_CAP + 1216 ? 6 * D : G2_CAP + 1216;
    // input of a linear: three halves per element (then, for inputs of D elements, the K parts of its rows and the rows);
    // attention: scores, from G2_CAP on [warp][64] partial outputs, then q, k and v of the position
    float xs[XS];
    float xres[D / 16];                               // this CTA's rows of the residual stream
    float part[256];                                  // K parts of the second projection
    float red[4][G2_WARPS];
    uint64_t full[2], empty[2], never;
    int loads;                                        // copies issued, for a launch that gives up
    volatile int abort_flag;
};

template <int NB>
__global__ void __launch_bounds__(G2_THREADS, 1) k_gpt2_layers(const __grid_constant__ HxGpt2Step P) {
    constexpr int D = 256 * NB, ROWS = D / 16;        // rows of a D-row linear per CTA
    extern __shared__ __align__(128) uint8_t smem_raw[];
    G2Smem<NB>& S = *reinterpret_cast<G2Smem<NB>*>(smem_raw);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31, cta = (int)cl_rank();
    volatile int* ab = &S.abort_flag;
    hx_grid_dep_launch();
    if (tid == 0) {
        for (int i = 0; i < 2; i++) { mb_init(&S.full[i], 1); mb_init(&S.empty[i], G2_WARPS); }
        mb_init(&S.never, 1);
        S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int i = tid; i < D; i += G2_THREADS) S.xa[i] = S.xb[i] = S.ctx[i] = 0ull;
    for (int i = tid; i < 4 * D; i += G2_THREADS) S.h[i] = 0ull;
    for (int i = tid; i < 192; i += G2_THREADS) S.qkv[i] = 0ull;
    cl_sync();

    if (warp == G2_WARPS) {
        // ------------------------------ weights: a phase ahead ------------------------------
        if (lane == 0) {
            bool ok = !P.stall || mb_wait(&S.never, 0, ab, P.wait_ns);
            int n = 0;
            for (int L = 0; L < P.n_layers && ok; L++)
                for (int ph = 0; ph < 4 && ok; ph++, n++) {
                    const HxGpt2LayerDev& ly = P.layers[L];
                    const uint32_t rows = ph == 0 ? 3 * ROWS : (ph == 2 ? 4 * ROWS : ROWS), kb = ph == 3 ? 4 * D : D;
                    const uint32_t bytes = rows * kb / 16 * 9;
                    const int b = n & 1;
                    if (n >= 2 && !mb_wait(&S.empty[b], (uint32_t)((n >> 1) - 1) & 1u, ab, P.wait_ns)) { ok = false; break; }
                    mb_expect(&S.full[b], bytes);
                    bulk_load(S.w[b], ly.t16[ph] + (size_t)cta * bytes, bytes, &S.full[b]);
                }
            S.loads = n;
        }
    } else {
        const int g = lane >> 2, t = lane & 3;
        // What every CTA needs is sent to CTA w by warp w, consecutive rows by consecutive lanes: whole lines through the
        // cluster's network (the sixteen lanes of a row each to another CTA took 4500 cycles for the 192 rows of c_fc).
        static_assert(G2_WARPS == G2_CTAS, "a warp per destination");
        const uint32_t base = cl_map(s_u32(smem_raw), (uint32_t)warp), me = s_u32(smem_raw);
        const uint32_t d_xa = base + s_u32(S.xa) - me, d_xb = base + s_u32(S.xb) - me, d_h = base + s_u32(S.h) - me, d_ctx = base + s_u32(S.ctx) - me;
        hx_grid_dep_wait();                                        // the token and the position come from the launch before
        const int pos = __ldcg(P.pos), tok = __ldcg(P.tok);
        __half* dig = reinterpret_cast<__half*>(S.xs);
        float* part = S.xs + 3 * D / 2;                            // [NB][rows] of a linear with D inputs
        float* yrow = part + NB * 4 * ROWS;
        int n = 0;                                                 // weight phases so far
        auto take = [&]() { (void)mb_wait(&S.full[n & 1], (uint32_t)(n >> 1) & 1u, ab, P.wait_ns); __syncwarp(); };      // the phase's weights are complete
        auto give = [&]() { __syncwarp(); if (lane == 0) mb_arrive(&S.empty[n & 1]); n++; };
        // The phase's input (elements tid, tid + 512, ... of K) scaled to at most one by a power of two, as three f16 terms
        // (33 bits); returns the power.  Every thread is past its use of xs when the first barrier lets go.
        auto split = [&](const auto& v, int K, int slot) {
            constexpr int N = sizeof(v) / sizeof(float);
            float mx = 0.0f;
#pragma unroll
            for (int i = 0; i < N; i++) if (tid + i * G2_CT < K) mx = fmaxf(mx, fabsf(v[i]));
            mx = hx_warp_max(mx);
            if (lane == 0) S.red[slot][warp] = mx;
            g2_sync();
            mx = 0.0f;
#pragma unroll
            for (int i = 0; i < G2_WARPS; i++) mx = fmaxf(mx, S.red[slot][i]);
            float sx = 1.0f;
            if (mx > 0.0f && mx < INFINITY) sx = __uint_as_float(min((__float_as_uint(mx) >> 23) + 1u, 254u) << 23);
            const float inv = 1.0f / sx;
#pragma unroll
            for (int i = 0; i < N; i++) {
                const int k = tid + i * G2_CT;
                if (k >= K) continue;
                const float x = v[i] * inv;
                const __half a = __float2half_rn(x);
                const float r = (x - __half2float(a)) * 2048.0f;
                const __half b = __float2half_rn(r);
                __half* to = dig + g2_place(k);
                to[0] = a; to[16] = b; to[32] = __float2half_rn((r - __half2float(b)) * 2048.0f);
            }
            g2_sync();
            return sx;
        };
        // `rows` rows of D inputs: a warp takes (sixteen rows, 256 columns) at a time
        auto linear = [&](int rows) {
            take();
            #pragma unroll 1
            for (int u = warp; u < rows / 16 * NB; u += G2_WARPS) {
                const int tile = u / NB, pt = u - tile * NB;
                float lo, hi;
                g2_cells(S.w[n & 1] + u * 2 * HX_T16_CELL, 2, dig + pt * 2 * 384, lo, hi);
                if (t == 0) { part[pt * rows + tile * 16 + g] = lo; part[pt * rows + tile * 16 + g + 8] = hi; }
            }
            give();
            g2_sync();
        };
        auto row_sum = [&](int rows, int rl) {
            float s = part[rl];
#pragma unroll
            for (int i = 1; i < NB; i++) s += part[i * rows + rl];
            return s;
        };
        // LayerNorm of the values this thread fetched (elements tid and tid + 512), this CTA's rows of them to xres; the result's terms to xs
        constexpr int PT = (D + G2_CT - 1) / G2_CT;
        auto layer_norm = [&](const float (&v)[PT], const float (&gg)[PT], const float (&bb)[PT]) {
            float s = 0.0f;
#pragma unroll
            for (int i = 0; i < PT; i++) if (tid + i * G2_CT < D) s += v[i];
            s = hx_warp_sum(s);
            if (lane == 0) S.red[0][warp] = s;
            g2_sync();                                             // (every warp has sent its rows: xres may change)
#pragma unroll
            for (int i = 0; i < PT; i++) { const int e = tid + i * G2_CT - cta * ROWS; if (e >= 0 && e < ROWS) S.xres[e] = v[i]; }
            float mean = 0.0f;
#pragma unroll
            for (int i = 0; i < G2_WARPS; i++) mean += S.red[0][i];
            mean /= (float)D;
            s = 0.0f;
#pragma unroll
            for (int i = 0; i < PT; i++) if (tid + i * G2_CT < D) s += (v[i] - mean) * (v[i] - mean);
            s = hx_warp_sum(s);
            if (lane == 0) S.red[1][warp] = s;
            g2_sync();
            float var = 0.0f;
#pragma unroll
            for (int i = 0; i < G2_WARPS; i++) var += S.red[1][i];
            const float inv = rsqrtf(var / (float)D + P.eps);
            float y[PT];
#pragma unroll
            for (int i = 0; i < PT; i++) y[i] = gg[i] * ((v[i] - mean) * inv) + bb[i];
            return split(y, D, 2);
        };
        #pragma unroll 1
        for (int L = 0; L < P.n_layers; L++) {
            const HxGpt2LayerDev& ly = P.layers[L];
            const unsigned ep = (unsigned)L + 1u;
            float* kc = P.kc + (size_t)L * (D / 64) * P.cap * 64;
            float* vc = P.vc + (size_t)L * (D / 64) * P.cap * 64;
            // ---- LayerNorm, qkv ----
            {
                float v[PT], gg[PT], bb[PT];
#pragma unroll
                for (int i = 0; i < PT; i++) { const int e = tid + i * G2_CT; gg[i] = e < D ? __ldg(ly.ln1g + e) : 0.0f; bb[i] = e < D ? __ldg(ly.ln1b + e) : 0.0f; }
                const float bias = tid < 3 * ROWS ? __ldg(ly.bias[0] + cta * 3 * ROWS + tid) : 0.0f;
#pragma unroll
                for (int i = 0; i < PT; i++) {
                    const int e = tid + i * G2_CT;
                    v[i] = e >= D ? 0.0f : (L == 0 ? __ldg(P.emb + (size_t)tok * D + e) + __ldg(P.wpe + (size_t)pos * D + e) : g2_wait(&S.xb[e], (unsigned)L, ab, P.wait_ns));
                }
                const float sc = layer_norm(v, gg, bb) * ly.ts[0];
                linear(3 * ROWS);
                if (tid < 3 * ROWS) {
                    const int row = cta * 3 * ROWS + tid, sec = row / D, r = row - sec * D;
                    g2_send(cl_map(s_u32(&S.qkv[sec * 64 + (r & 63)]), (uint32_t)(r >> 6)), row_sum(3 * ROWS, tid) * sc + bias, ep);
                }
                g2_sync();                                         // (the head's own attention writes over the parts)
            }
            // ---- attention of head `cta` ----
            if (cta < D / 64) {
                const float* kb = kc + (size_t)cta * P.cap * 64;
                const float* vb = vc + (size_t)cta * P.cap * 64;
                const int kp = tid & 3, c4 = tid & 15, kg = tid >> 4;
                // Passes of 256 keys: a thread holds a quarter of two K rows, later a chunk of eight V rows.  The first pass of K
                // travels while q is on its way, the first of V during the softmax.
                float4 kr[8];
                auto load_k = [&](int k0) {
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const int key = k0 + (tid >> 2) + 128 * p;
#pragma unroll
                        for (int c = 0; c < 4; c++) kr[4 * p + c] = key < pos ? __ldcg(reinterpret_cast<const float4*>(kb + (size_t)key * 64 + (kp + 4 * c) * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                };
                auto load_v = [&](int k0) {
#pragma unroll
                    for (int i = 0; i < 8; i++) { const int key = k0 + kg + 32 * i; kr[i] = key < pos ? __ldcg(reinterpret_cast<const float4*>(vb + (size_t)key * 64 + c4 * 4)) : make_float4(0.f, 0.f, 0.f, 0.f); }
                };
                float* sq = S.xs + G2_CAP + 1024;                 // q, k, v of the position
                load_k(0);
                if (tid < 192) {
                    const float x = g2_wait(&S.qkv[tid], ep, ab, P.wait_ns);
                    sq[tid] = x;
                    if (tid >= 64) (tid < 128 ? kc : vc)[((size_t)cta * P.cap + pos) * 64 + (tid & 63)] = x;
                }
                g2_sync();
                float4 q4[4];
#pragma unroll
                for (int c = 0; c < 4; c++) q4[c] = *reinterpret_cast<const float4*>(sq + (kp + 4 * c) * 4);
                float* sc = S.xs;
                float* pv = S.xs + G2_CAP;
                float mx = -INFINITY;
                for (int k0 = 0; k0 <= pos; k0 += 256) {
                    if (k0 > 0) load_k(k0);
#pragma unroll
                    for (int p = 0; p < 2; p++) {
                        const int key = k0 + (tid >> 2) + 128 * p;
                        float d = 0.0f;
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const float4 k4 = key == pos ? *reinterpret_cast<const float4*>(sq + 64 + (kp + 4 * c) * 4) : kr[4 * p + c];
                            d = fmaf(q4[c].x, k4.x, d); d = fmaf(q4[c].y, k4.y, d); d = fmaf(q4[c].z, k4.z, d); d = fmaf(q4[c].w, k4.w, d);
                        }
                        d += __shfl_xor_sync(0xffffffffu, d, 1); d += __shfl_xor_sync(0xffffffffu, d, 2);
                        d *= P.scale;
                        if (key <= pos) { mx = fmaxf(mx, d); if (kp == 0) sc[key] = d; }
                    }
                }
                load_v(0);
                mx = hx_warp_max(mx);
                if (lane == 0) S.red[2][warp] = mx;
                g2_sync();
                mx = -INFINITY;
#pragma unroll
                for (int i = 0; i < G2_WARPS; i++) mx = fmaxf(mx, S.red[2][i]);
                float ls = 0.0f;
                for (int key = tid; key <= pos; key += G2_CT) { const float p = __expf(sc[key] - mx); sc[key] = p; ls += p; }
                ls = hx_warp_sum(ls);
                if (lane == 0) S.red[3][warp] = ls;
                g2_sync();
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                for (int k0 = 0; k0 <= pos; k0 += 256) {
                    if (k0 > 0) load_v(k0);
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const int key = k0 + kg + 32 * i;
                        if (key > pos) break;
                        const float p = sc[key];
                        const float4 v4 = key == pos ? *reinterpret_cast<const float4*>(sq + 128 + c4 * 4) : kr[i];
                        acc.x = fmaf(p, v4.x, acc.x); acc.y = fmaf(p, v4.y, acc.y); acc.z = fmaf(p, v4.z, acc.z); acc.w = fmaf(p, v4.w, acc.w);
                    }
                }
                acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16); acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
                acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16); acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
                if (lane < 16) *reinterpret_cast<float4*>(pv + warp * 64 + c4 * 4) = acc;
                g2_sync();
                float lsum = 0.0f;
#pragma unroll
                for (int i = 0; i < G2_WARPS; i++) lsum += S.red[3][i];
                const int dim = tid >> 3, p8 = tid & 7;
                float o = pv[p8 * 64 + dim] + pv[(p8 + 8) * 64 + dim];
                o += __shfl_xor_sync(0xffffffffu, o, 1); o += __shfl_xor_sync(0xffffffffu, o, 2); o += __shfl_xor_sync(0xffffffffu, o, 4);
                if (p8 == 0) sq[dim] = o / lsum;                   // (q has been used)
                g2_sync();
#pragma unroll
                for (int i = 0; i < 64; i += 32) g2_send(d_ctx + (uint32_t)(cta * 64 + i + lane) * 8, sq[i + lane], ep);
            }
            // ---- proj + residual ----
            {
                constexpr int RL = (ROWS + 31) / 32;
                float bias[RL], cv[PT];
#pragma unroll
                for (int i = 0; i < RL; i++) bias[i] = lane + 32 * i < ROWS ? __ldg(ly.bias[1] + cta * ROWS + lane + 32 * i) : 0.0f;
#pragma unroll
                for (int i = 0; i < PT; i++) cv[i] = tid + i * G2_CT < D ? g2_wait(&S.ctx[tid + i * G2_CT], ep, ab, P.wait_ns) : 0.0f;
                const float sc = split(cv, D, 0) * ly.ts[1];
                linear(ROWS);
#pragma unroll
                for (int i = 0; i < RL; i++) {
                    const int rl = lane + 32 * i;
                    if (rl < ROWS) g2_send(d_xa + (uint32_t)(cta * ROWS + rl) * 8, S.xres[rl] + (row_sum(ROWS, rl) * sc + bias[i]), ep);
                }
            }
            // ---- LayerNorm, c_fc, gelu ----
            {
                float v[PT], gg[PT], bb[PT];
#pragma unroll
                for (int i = 0; i < PT; i++) { const int e = tid + i * G2_CT; gg[i] = e < D ? __ldg(ly.ln2g + e) : 0.0f; bb[i] = e < D ? __ldg(ly.ln2b + e) : 0.0f; }
                const float bias = tid < 4 * ROWS ? __ldg(ly.bias[2] + cta * 4 * ROWS + tid) : 0.0f;
#pragma unroll
                for (int i = 0; i < PT; i++) v[i] = tid + i * G2_CT < D ? g2_wait(&S.xa[tid + i * G2_CT], ep, ab, P.wait_ns) : 0.0f;
                const float sc = layer_norm(v, gg, bb) * ly.ts[2];
                linear(4 * ROWS);
                if (tid < 4 * ROWS) yrow[tid] = g2_gelu(row_sum(4 * ROWS, tid) * sc + bias);
                g2_sync();
#pragma unroll
                for (int i = 0; i < 4 * ROWS; i += 32) g2_send(d_h + (uint32_t)(cta * 4 * ROWS + i + lane) * 8, yrow[i + lane], ep);
            }
            // ---- second projection + residual: WT warps per sixteen rows, each every WT-th part of 256 columns ----
            {
                constexpr int WT = G2_WARPS / NB, RL = (ROWS + 31) / 32;
                float hv[4 * PT], bias[RL];
#pragma unroll
                for (int i = 0; i < RL; i++) bias[i] = lane + 32 * i < ROWS ? __ldg(ly.bias[3] + cta * ROWS + lane + 32 * i) : 0.0f;
#pragma unroll
                for (int i = 0; i < 4 * PT; i++) hv[i] = tid + i * G2_CT < 4 * D ? g2_wait(&S.h[tid + i * G2_CT], ep, ab, P.wait_ns) : 0.0f;
                const float sc = split(hv, 4 * D, 0) * ly.ts[3];
                take();
                const int tile = warp % NB, j = warp / NB;
                if (j < WT) {
                    float lo = 0.0f, hi = 0.0f;
                    #pragma unroll 1
                    for (int pt = j; pt < 4 * NB; pt += WT) {
                        float a, b;
                        g2_cells(S.w[n & 1] + (tile * 8 * NB + pt * 2) * HX_T16_CELL, 2, dig + pt * 2 * 384, a, b);
                        lo += a; hi += b;
                    }
                    if (t == 0) { S.part[j * ROWS + tile * 16 + g] = lo; S.part[j * ROWS + tile * 16 + g + 8] = hi; }
                }
                give();
                g2_sync();
#pragma unroll
                for (int i = 0; i < RL; i++) {
                    const int rl = lane + 32 * i, row = cta * ROWS + rl;
                    if (rl >= ROWS) continue;
                    float s = S.part[rl];
#pragma unroll
                    for (int q = 1; q < WT; q++) s += S.part[q * ROWS + rl];
                    const float y = S.xres[rl] + (s * sc + bias[i]);
                    if (L + 1 < P.n_layers) g2_send(d_xb + (uint32_t)row * 8, y, ep);
                    else if (warp == 0) P.x_out[row] = y;
                }
            }
        }
    }
    __syncthreads();
    if (S.abort_flag && tid == 0) {
        // given up: the CTA must not end with a copy of its own in flight
        for (int i = S.loads > 2 ? S.loads - 2 : 0; i < S.loads; i++) mb_drain(&S.full[i & 1], (uint32_t)(i >> 1) & 1u);
        *P.err = 1;
    }
    cl_sync();      // nobody leaves while a CTA of the cluster may still write into its shared memory
}

template <int NB> int g2_launch(const HxGpt2Step& p, cudaStream_t st, bool pdl) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G2_CTAS); cfg.blockDim = dim3(G2_THREADS); cfg.dynamicSmemBytes = sizeof(G2Smem<NB>); cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = G2_CTAS; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = pdl ? 2 : 1;
    HX_CUDA(cudaLaunchKernelEx(&cfg, k_gpt2_layers<NB>, p));
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}

template <int NB> bool g2_fits() {
    static_assert(sizeof(G2Smem<NB>) <= 227 * 1024, "shared memory");
    if (cudaFuncSetAttribute(k_gpt2_layers<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(G2Smem<NB>)) != cudaSuccess ||
        cudaFuncSetAttribute(k_gpt2_layers<NB>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) { (void)cudaGetLastError(); return false; }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G2_CTAS); cfg.blockDim = dim3(G2_THREADS); cfg.dynamicSmemBytes = sizeof(G2Smem<NB>);
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = G2_CTAS; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_gpt2_layers<NB>, &cfg) != cudaSuccess) { (void)cudaGetLastError(); return false; }
    return n >= 1;
}

}  // namespace

// d_model 256, 512 or 768 with heads of 64, hidden size 4 d_model and a cache of at most G2_CAP positions, on a device that
// holds a cluster of sixteen such CTAs.  Everything else keeps the per-op graph.
bool hx_gpt2_step_fits(const hx_config& c, int kv_cap) {
    if (c.head_dim != 64 || c.d_ff != 4 * c.d_model || kv_cap > G2_CAP || c.d_model % 256 || c.d_model > 768) return false;
    return c.d_model == 256 ? g2_fits<1>() : c.d_model == 512 ? g2_fits<2>() : g2_fits<3>();
}

int hx_gpt2_step_launch(const HxGpt2Step& p, int d_model, cudaStream_t st, bool pdl) {
    return d_model == 256 ? g2_launch<1>(p, st, pdl) : d_model == 512 ? g2_launch<2>(p, st, pdl) : g2_launch<3>(p, st, pdl);
}
