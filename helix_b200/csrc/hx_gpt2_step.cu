// hx_gpt2_step.cu -- the layers of one GPT-2 token in one launch: a cluster of sixteen CTAs, vectors exchanged through
// distributed shared memory.
//
// Replaces, for one token, the launch sequence of forward_layer_gpt2 (helixc/runtime/gpt2_infer.c:1131-1193) with a KV cache:
// LayerNorm -> qkv (+bias) -> attention -> proj (+bias, residual) -> LayerNorm -> c_fc (+bias, gelu_new) -> proj (+bias,
// residual).  The lm_head follows as a launch of its own over all SMs.
//
// What bounds a token of this size (48 MB of packed weights in the layers, L2-resident between tokens) is the chain of
// sixty dependent exchanges.  Seventy-two launches cost 4 us each; a hand-over between CTAs through L2 costs about 1.2 us; a
// store into the shared memory of another CTA of the cluster arrives in about 0.3.  Sixteen SMs are enough for the
// arithmetic (5 us of a layer at D = 768), so the layers run on one cluster:
//  * every CTA owns a sixteenth of the rows of each linear; its weights stream through two shared-memory buffers by bulk
//    copies, a phase ahead;
//  * a half-warp takes a row: its lanes hold the (normed) input in registers, 16 * NB elements each (D = 256 * NB), decode
//    the codes with cvt.f16x2.e2m1x2 and multiply in f32; the second projection (K = 4 D) is cut into four K quarters over
//    the warps;
//  * results leave as 8-byte (value, epoch) pairs stored into all sixteen CTAs (q, k, v: into the head's CTA), and the
//    reader polls its own shared memory until the epoch of the layer shows up.  An aligned 8-byte store is single-copy
//    atomic, so a matching epoch proves the value.  No buffer is written for the next layer before every CTA has read this
//    layer's: each phase needs rows of all CTAs, so nobody is more than a phase ahead;
//  * attention: one CTA per head.
// Waits are bounded; after one that ran out the CTA goes on with what is there, raises *err and the call reports it.
#include "hx_tc.cuh"
#include "hx_kernels.cuh"
#include "hx_gpt2_step.cuh"
#include <cuda_fp16.h>

using namespace hxtc;

namespace {

constexpr int G2_CTAS = 16, G2_WARPS = 16, G2_CT = G2_WARPS * 32, G2_THREADS = G2_CT + 32;
constexpr int G2_CAP = 2048;                          // cached positions at most (scores in shared memory)

__device__ __forceinline__ void g2_sync() { asm volatile("bar.sync 1, %0;" :: "n"(G2_CT) : "memory"); }
__device__ __forceinline__ int g2_pad(int e) { return (e >> 4) * 20 + (e & 15); }      // blocks of sixteen 20 words apart: no bank conflicts
__device__ __forceinline__ void g2_send(uint32_t addr, float v, unsigned ep) {
    const unsigned long long w = ((unsigned long long)ep << 32) | (unsigned long long)__float_as_uint(v);
    asm volatile("st.relaxed.cluster.shared::cluster.u64 [%0], %1;" :: "r"(addr), "l"(w) : "memory");
}
__device__ __forceinline__ float g2_wait(const unsigned long long* p, unsigned ep, volatile int* ab) {
    unsigned long long w = 0;
    const uint32_t a = s_u32(p);
    (void)mb_bounded([&] {
        asm volatile("ld.relaxed.cluster.shared::cta.u64 %0, [%1];" : "=l"(w) : "r"(a) : "memory");
        return (unsigned)(w >> 32) == ep || *ab != 0;
    }, ab);
    return __uint_as_float((unsigned)w);
}
__device__ __forceinline__ float g2_gelu(float x) {   // gpu_gelu_stable_kernel.hx:15-28
    const float inner = 0.7978846f * (x + (0.044715f * (x * x * x))), two = 2.0f * inner;
    const float sgn = inner < 0.0f ? -1.0f : 1.0f;
    const float e = __expf(-(sgn * two));
    const float th = sgn * ((1.0f - e) / (1.0f + e));
    return 0.5f * x * (1.0f + th);
}
// sum of sixteen products with the codes of one block
__device__ __forceinline__ float g2_dot16(uint2 c, const float* x) {
    float a = 0.0f, b = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t p0, p1, p2, p3;
        asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\tmov.b32 {b0, b1, b2, b3}, %4;\n\t"
            "cvt.rn.f16x2.e2m1x2 %0, b0;\n\tcvt.rn.f16x2.e2m1x2 %1, b1;\n\tcvt.rn.f16x2.e2m1x2 %2, b2;\n\tcvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
            : "=r"(p0), "=r"(p1), "=r"(p2), "=r"(p3) : "r"(h ? c.y : c.x));
        const float* y = x + 8 * h;
        float2 f;
        f = __half22float2(*reinterpret_cast<__half2*>(&p0)); a = fmaf(y[0], f.x, a); b = fmaf(y[1], f.y, b);
        f = __half22float2(*reinterpret_cast<__half2*>(&p1)); a = fmaf(y[2], f.x, a); b = fmaf(y[3], f.y, b);
        f = __half22float2(*reinterpret_cast<__half2*>(&p2)); a = fmaf(y[4], f.x, a); b = fmaf(y[5], f.y, b);
        f = __half22float2(*reinterpret_cast<__half2*>(&p3)); a = fmaf(y[6], f.x, a); b = fmaf(y[7], f.y, b);
    }
    return a + b;
}
__device__ __forceinline__ float g2_scale(uint32_t byte) {
    uint32_t h;
    asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h) : "h"((unsigned short)byte));
    return __half2float(__ushort_as_half((unsigned short)h));
}
// row . x over NB blocks per lane: lane l of the half-warp owns blocks l, l + 16, ...; every lane of the half gets the sum
template <int NB>
__device__ __forceinline__ float g2_row(const uint8_t* codes, const uint8_t* scales, const float (&x)[16 * NB], int l) {
    float s = 0.0f;
#pragma unroll
    for (int j = 0; j < NB; j++) {
        const uint2 c = *reinterpret_cast<const uint2*>(codes + (l + 16 * j) * 8);
        s = fmaf(g2_dot16(c, x + 16 * j), g2_scale(scales[l + 16 * j]), s);
    }
#pragma unroll
    for (int d = 1; d < 16; d <<= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    return s;
}

template <int NB> struct G2Smem {
    static constexpr int D = 256 * NB;
    static constexpr int WB = 36 * D * D / 256;       // bytes of the largest phase: 4 D / 16 rows of D, or D / 16 rows of 4 D
    uint8_t w[2][WB];
    unsigned long long xa[D], xb[D], ctx[D], h[4 * D], qkv[192];
    static constexpr int XS = 5 * D > G2_CAP + 1024 ? 5 * D : G2_CAP + 1024;
    float xs[XS];                                     // input of the phase, padded; attention: scores, then [warp][64] partial outputs from G2_CAP on
    float xres[D];                                    // residual stream
    float part[4 * (D / 16)];                         // K quarters of the second projection
    float red[4][G2_WARPS];
    float q[64], k[64], v[64];
    uint64_t full[2], empty[2];
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
            bool ok = true;
            int n = 0;
            for (int L = 0; L < P.n_layers && ok; L++)
                for (int ph = 0; ph < 4 && ok; ph++, n++) {
                    const HxGpt2LayerDev& ly = P.layers[L];
                    const uint32_t rows = ph == 0 ? 3 * ROWS : (ph == 2 ? 4 * ROWS : ROWS), kb = ph == 3 ? 4 * D : D;
                    const uint32_t cb = rows * kb / 2, sb = rows * kb / 16;
                    const int b = n & 1;
                    if (n >= 2 && !mb_wait(&S.empty[b], (uint32_t)((n >> 1) - 1) & 1u, ab)) { ok = false; break; }
                    mb_expect(&S.full[b], cb + sb);
                    bulk_load(S.w[b], ly.codes[ph] + (size_t)cta * cb, cb, &S.full[b]);
                    bulk_load(S.w[b] + cb, ly.scales[ph] + (size_t)cta * sb, sb, &S.full[b]);
                }
            for (int i = n > 2 ? n - 2 : 0; i < n && !ok; i++) mb_drain(&S.full[i & 1], (uint32_t)(i >> 1) & 1u);
        }
    } else {
        const int l = lane & 15, hw = warp * 2 + (lane >> 4);      // half-warp of the CTA
        // where this lane's stores go: CTA l of the cluster
        const uint32_t base = cl_map(s_u32(smem_raw), (uint32_t)l), me = s_u32(smem_raw);
        const uint32_t d_xa = base + s_u32(S.xa) - me, d_xb = base + s_u32(S.xb) - me, d_h = base + s_u32(S.h) - me, d_qkv = base + s_u32(S.qkv) - me;
        hx_grid_dep_wait();                                        // the token and the position come from the launch before
        const int pos = __ldcg(P.pos), tok = __ldcg(P.tok);
        float xr[16 * NB];
        int n = 0;                                                 // weight phases so far
        auto take = [&](int slice) {                               // the phase's input into registers, its weights complete
            const float* src = S.xs + slice * (D / 16) * 20;
#pragma unroll
            for (int j = 0; j < NB; j++)
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const float4 v = *reinterpret_cast<const float4*>(src + (l + 16 * j) * 20 + c * 4);
                    xr[16 * j + 4 * c] = v.x; xr[16 * j + 4 * c + 1] = v.y; xr[16 * j + 4 * c + 2] = v.z; xr[16 * j + 4 * c + 3] = v.w;
                }
            (void)mb_wait(&S.full[n & 1], (uint32_t)(n >> 1) & 1u, ab);
            __syncwarp();
        };
        auto give = [&]() { __syncwarp(); if (lane == 0) mb_arrive(&S.empty[n & 1]); n++; };
        // LayerNorm of the values this thread fetched (elements tid and tid + 512), result to xs, the values to xres
        constexpr int PT = (D + G2_CT - 1) / G2_CT;
        auto layer_norm = [&](const float (&v)[PT], const float (&gg)[PT], const float (&bb)[PT]) {
            float s = 0.0f;
#pragma unroll
            for (int i = 0; i < PT; i++) if (tid + i * G2_CT < D) { s += v[i]; S.xres[tid + i * G2_CT] = v[i]; }
            s = hx_warp_sum(s);
            if (lane == 0) S.red[0][warp] = s;
            g2_sync();
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
#pragma unroll
            for (int i = 0; i < PT; i++) if (tid + i * G2_CT < D) S.xs[g2_pad(tid + i * G2_CT)] = gg[i] * ((v[i] - mean) * inv) + bb[i];
            g2_sync();
        };
        #pragma unroll 1
        for (int L = 0; L < P.n_layers; L++) {
            const HxGpt2LayerDev& ly = P.layers[L];
            const unsigned ep = (unsigned)L + 1u;
            float* kc = P.kc + (size_t)L * (D / 64) * P.cap * 64;
            float* vc = P.vc + (size_t)L * (D / 64) * P.cap * 64;
            // ---- LayerNorm, qkv ----
            {
                float v[PT], gg[PT], bb[PT], bias[(3 * ROWS + 31) / 32];
#pragma unroll
                for (int i = 0; i < PT; i++) { const int e = tid + i * G2_CT; gg[i] = e < D ? __ldg(ly.ln1g + e) : 0.0f; bb[i] = e < D ? __ldg(ly.ln1b + e) : 0.0f; }
#pragma unroll
                for (int i = 0; i < (3 * ROWS + 31) / 32; i++) bias[i] = hw + 32 * i < 3 * ROWS ? __ldg(ly.bias[0] + cta * 3 * ROWS + hw + 32 * i) : 0.0f;
#pragma unroll
                for (int i = 0; i < PT; i++) {
                    const int e = tid + i * G2_CT;
                    v[i] = e >= D ? 0.0f : (L == 0 ? __ldg(P.emb + (size_t)tok * D + e) + __ldg(P.wpe + (size_t)pos * D + e) : g2_wait(&S.xb[e], (unsigned)L, ab));
                }
                layer_norm(v, gg, bb);
                take(0);
                const uint8_t* w = S.w[n & 1];
                const float ts = ly.ts[0];
#pragma unroll
                for (int i = 0; i < (3 * ROWS + 31) / 32; i++) {
                    const int rl = min(hw + 32 * i, 3 * ROWS - 1);
                    const float y = g2_row<NB>(w + rl * (D / 2), w + 3 * ROWS * (D / 2) + rl * (D / 16), xr, l) * ts + bias[i];
                    const int row = cta * 3 * ROWS + rl, sec = row / D, r = row - sec * D;
                    if (hw + 32 * i < 3 * ROWS && l == (r >> 6)) g2_send(d_qkv + (uint32_t)(sec * 64 + (r & 63)) * 8, y, ep);
                }
                give();
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
                load_k(0);
                if (tid < 192) {
                    const float x = g2_wait(&S.qkv[tid], ep, ab);
                    (tid < 64 ? S.q : (tid < 128 ? S.k : S.v))[tid & 63] = x;
                    if (tid >= 64) (tid < 128 ? kc : vc)[((size_t)cta * P.cap + pos) * 64 + (tid & 63)] = x;
                }
                g2_sync();
                float4 q4[4];
#pragma unroll
                for (int c = 0; c < 4; c++) q4[c] = *reinterpret_cast<const float4*>(S.q + (kp + 4 * c) * 4);
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
                            const float4 k4 = key == pos ? *reinterpret_cast<const float4*>(S.k + (kp + 4 * c) * 4) : kr[4 * p + c];
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
                        const float4 v4 = key == pos ? *reinterpret_cast<const float4*>(S.v + c4 * 4) : kr[i];
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
                o /= lsum;
                const uint32_t off = s_u32(&S.ctx[cta * 64 + dim]);
                g2_send(cl_map(off, (uint32_t)p8), o, ep);
                g2_send(cl_map(off, (uint32_t)p8 + 8u), o, ep);
            }
            // ---- proj + residual ----
            {
                float bias[(ROWS + 31) / 32];
#pragma unroll
                for (int i = 0; i < (ROWS + 31) / 32; i++) bias[i] = hw + 32 * i < ROWS ? __ldg(ly.bias[1] + cta * ROWS + hw + 32 * i) : 0.0f;
                float cv[PT];
#pragma unroll
                for (int i = 0; i < PT; i++) cv[i] = tid + i * G2_CT < D ? g2_wait(&S.ctx[tid + i * G2_CT], ep, ab) : 0.0f;
                g2_sync();                                         // (the head's own attention has used xs)
#pragma unroll
                for (int i = 0; i < PT; i++) if (tid + i * G2_CT < D) S.xs[g2_pad(tid + i * G2_CT)] = cv[i];
                g2_sync();
                take(0);
                const uint8_t* w = S.w[n & 1];
                const float ts = ly.ts[1];
#pragma unroll
                for (int i = 0; i < (ROWS + 31) / 32; i++) {
                    const int rl = min(hw + 32 * i, ROWS - 1), row = cta * ROWS + rl;
                    const float y = S.xres[row] + (g2_row<NB>(w + rl * (D / 2), w + ROWS * (D / 2) + rl * (D / 16), xr, l) * ts + bias[i]);
                    if (hw + 32 * i < ROWS) g2_send(d_xa + (uint32_t)row * 8, y, ep);
                }
                give();
            }
            // ---- LayerNorm, c_fc, gelu ----
            {
                float v[PT], gg[PT], bb[PT], bias[(4 * ROWS + 31) / 32];
#pragma unroll
                for (int i = 0; i < PT; i++) { const int e = tid + i * G2_CT; gg[i] = e < D ? __ldg(ly.ln2g + e) : 0.0f; bb[i] = e < D ? __ldg(ly.ln2b + e) : 0.0f; }
#pragma unroll
                for (int i = 0; i < (4 * ROWS + 31) / 32; i++) bias[i] = hw + 32 * i < 4 * ROWS ? __ldg(ly.bias[2] + cta * 4 * ROWS + hw + 32 * i) : 0.0f;
#pragma unroll
                for (int i = 0; i < PT; i++) v[i] = tid + i * G2_CT < D ? g2_wait(&S.xa[tid + i * G2_CT], ep, ab) : 0.0f;
                layer_norm(v, gg, bb);
                take(0);
                const uint8_t* w = S.w[n & 1];
                const float ts = ly.ts[2];
#pragma unroll
                for (int i = 0; i < (4 * ROWS + 31) / 32; i++) {
                    const int rl = min(hw + 32 * i, 4 * ROWS - 1);
                    const float y = g2_gelu(g2_row<NB>(w + rl * (D / 2), w + 4 * ROWS * (D / 2) + rl * (D / 16), xr, l) * ts + bias[i]);
                    if (hw + 32 * i < 4 * ROWS) g2_send(d_h + (uint32_t)(cta * 4 * ROWS + rl) * 8, y, ep);
                }
                give();
            }
            // ---- second projection + residual: K quarter warp & 3, rows (warp >> 2) * 2 + half, + 8, ... ----
            {
                float hv[4 * PT];
#pragma unroll
                for (int i = 0; i < 4 * PT; i++) hv[i] = tid + i * G2_CT < 4 * D ? g2_wait(&S.h[tid + i * G2_CT], ep, ab) : 0.0f;
#pragma unroll
                for (int i = 0; i < 4 * PT; i++) if (tid + i * G2_CT < 4 * D) S.xs[g2_pad(tid + i * G2_CT)] = hv[i];
                g2_sync();
                const int sl = warp & 3, r0 = (warp >> 2) * 2 + (lane >> 4);
                take(sl);
                const uint8_t* w = S.w[n & 1];
                const float ts = ly.ts[3];
#pragma unroll
                for (int i = 0; i < ROWS / 8; i++) {
                    const int rl = r0 + 8 * i;
                    const float y = g2_row<NB>(w + rl * (2 * D) + sl * (D / 2), w + ROWS * (2 * D) + rl * (D / 4) + sl * (D / 16), xr, l);
                    if (l == 0) S.part[sl * ROWS + rl] = y;
                }
                give();
                g2_sync();
                for (int i = tid; i < ROWS * 16; i += G2_CT) {     // (i & 15 is this lane's l: the row goes to CTA l)
                    const int rl = i >> 4, row = cta * ROWS + rl;
                    const float y = S.xres[row] + (((S.part[rl] + S.part[ROWS + rl]) + (S.part[2 * ROWS + rl] + S.part[3 * ROWS + rl])) * ts + __ldg(ly.bias[3] + row));
                    if (L + 1 < P.n_layers) g2_send(d_xb + (uint32_t)row * 8, y, ep);
                    else if (l == 0) P.x_out[row] = y;
                }
            }
        }
    }
    __syncthreads();
    if (S.abort_flag && tid == 0) *P.err = 1;
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
