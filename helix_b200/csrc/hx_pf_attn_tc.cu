// hx_pf_attn_tc.cu -- causal attention of a prompt chunk over the KV cache on the tensor cores (tcgen05, head_dim 128).
//
// Replaces the per-head Q K^T / softmax / P V of forward_layer_llama (helixc/runtime/gpt2_infer.c:1242-1265).
//
// f32 accuracy from bf16 operands: every f32 value is the sum of three bf16 terms (24 bits: hi + mid + lo, exact), and a
// product keeps the six term pairs above 2^-25 of it (hi hi, hi mid, mid hi, hi lo, mid mid, lo hi); sums are f32 in TMEM.
// Six MMAs of 8192 multiply-adds per cycle and SM replace 128 FMA lanes: 10 x the f32 rate of the CUDA cores before any
// overhead.
//
// A CTA takes one kv head and 128 query rows (all query heads of the kv head times 128 / group tokens, so K and V serve
// the whole group) and walks through tiles of 128 keys.  The terms of K and V^T are prepared once per launch by
// k_pf_kv_split as shared-memory images (128 rows x 128 swizzled bytes = a 16 KB piece per term and half of the inner
// dimension); one thread streams the pieces through a ring with bulk copies, least significant term first, so that slots
// come free while the products of the more significant terms still run.  Per tile: S = Q K^T (48 MMAs, N = 128) -> eight
// softmax warps read S, two threads per row, keep the running maximum and sum, write P as three bf16 terms back to TMEM ->
// P V (48 MMAs, A operand from TMEM) -> the same warps add it to the output rows, which live in registers.
// The steps of a tile are serial (about 3000 + 2500 + 3000 cycles); what overlaps is the loading.
// Waits are bounded; after one that ran out the CTA writes nothing and raises *err.
#include "hx_tc.cuh"
#include "hx_prefill.cuh"
#include <cuda_bf16.h>

using namespace hxtc;

namespace {

constexpr int AT_DH = 128, AT_KT = 128;
constexpr uint32_t AT_PIECE = 16384;                  // 128 rows x 64 bf16
constexpr int AT_RING = 7;
constexpr int AT_THREADS = 320;                       // warp 0 loads, warp 1 issues the MMAs, warps 2-9 softmax
constexpr uint32_t AT_HDR = 4096;
constexpr uint32_t TM_S = 0, TM_PV = 128, TM_P = 256; // TMEM columns: S, P V, three terms of P (64 columns each)

struct AtSmem {
    uint64_t full[AT_RING], empty[AT_RING], q_ready, s_full, p_ready, pv_full;
    uint32_t tmem_base;
    volatile int abort_flag;
    float ex[2][2][128];                              // row maxima / sums exchanged between the two halves of a row
};
static_assert(sizeof(AtSmem) <= AT_HDR, "header");

// x = hi + mid + lo with bf16 terms, two values at a time (x0 in the low half)
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(h) : "f"(x1), "f"(x0));
    x0 -= __uint_as_float(h << 16); x1 -= __uint_as_float(h & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(m) : "f"(x1), "f"(x0));
    x0 -= __uint_as_float(m << 16); x1 -= __uint_as_float(m & 0xFFFF0000u);
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(l) : "f"(x1), "f"(x0));
}
// eight values -> one 16-byte chunk per term
__device__ __forceinline__ void split8(const float (&v)[8], uint4& h, uint4& m, uint4& l) {
    split2(v[0], v[1], h.x, m.x, l.x); split2(v[2], v[3], h.y, m.y, l.y); split2(v[4], v[5], h.z, m.z, l.z); split2(v[6], v[7], h.w, m.w, l.w);
}

// K and V^T of one kv head and tile of 128 keys as term pieces: [kv head][tile][K: lo0 lo1 mid0 mid1 hi0 hi1 | V: the same].
// K piece half h: row = key, 64 dims from 64 h.  V piece half h: row = dim, 64 keys from 64 h.  Keys beyond the context are 0.
// Bound by HBM / L2: 8 bytes read and 12 written per (key, dim).
__global__ void __launch_bounds__(256) k_pf_kv_split(const float* __restrict__ kc, const float* __restrict__ vc, HxPfWhere wh, int n_tok, int cap, uint8_t* __restrict__ dst) {
    const int tile = blockIdx.x, kvh = blockIdx.y, part = blockIdx.z, isv = part >> 1;
    hx_grid_dep_launch();
    hx_grid_dep_wait();
    const int ctx = __ldcg(wh.posp) + n_tok, k0 = tile * AT_KT;
    const size_t seq_off = wh.seqp ? (size_t)__ldcg(wh.seqp) * wh.seq_stride : 0;
    const float* src = (isv ? vc : kc) + seq_off + ((size_t)kvh * cap) * AT_DH;
    uint8_t* out = dst + (((size_t)kvh * gridDim.x + tile) * 2 + isv) * 6 * AT_PIECE;
#pragma unroll
    for (int n = 0; n < 4; n++) {
        const int i = (part & 1) * 1024 + n * 256 + threadIdx.x;
        float v[8];
        int row, c;                                       // row of the piece, 8-element chunk of its inner dimension
        if (!isv) {
            row = i >> 4; c = i & 15;
            const bool in = k0 + row < ctx;
            const float4* p = reinterpret_cast<const float4*>(src + (size_t)(k0 + row) * AT_DH + c * 8);
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), a = in ? __ldcg(p) : z, b = in ? __ldcg(p + 1) : z;
            v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        } else {
            row = i & 127; c = i >> 7;
#pragma unroll
            for (int e = 0; e < 8; e++) { const int key = k0 + c * 8 + e; v[e] = key < ctx ? __ldcg(src + (size_t)key * AT_DH + row) : 0.0f; }
        }
        uint4 h, m, l;
        split8(v, h, m, l);
        uint8_t* o = out + (size_t)(c >> 3) * AT_PIECE + row * 128 + (((c & 7) ^ (row & 7)) << 4);
        *reinterpret_cast<uint4*>(o) = l; *reinterpret_cast<uint4*>(o + 2 * AT_PIECE) = m; *reinterpret_cast<uint4*>(o + 4 * AT_PIECE) = h;
    }
}

__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tm_ld16(uint32_t (&r)[16], uint32_t a) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(a));
}
__device__ __forceinline__ void tm_st8(uint32_t a, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
                 :: "r"(a), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

// grid (kv heads, row tiles): the last row tiles, which see the most keys, start first
__global__ void __launch_bounds__(AT_THREADS, 1) k_pf_attn_tc(const float* __restrict__ qkv, int ld, HxPfWhere wh, int n_tok, int GRP, const uint8_t* __restrict__ pieces,
                                                              int ktiles, float scale, float* __restrict__ ctx, int ld_ctx, int* err) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    uint8_t* base = smem_raw + (((s_u32(smem_raw) + 1023u) & ~1023u) - s_u32(smem_raw));
    AtSmem& S = *reinterpret_cast<AtSmem*>(base);
    uint8_t* sq = base + AT_HDR;                              // Q terms: [hi, mid, lo][half]
    uint8_t* ring = sq + 6 * AT_PIECE;
    hx_grid_dep_launch();
    hx_grid_dep_wait();
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int kvh = blockIdx.x, TPT = 128 / GRP, t0 = ((int)gridDim.y - 1 - (int)blockIdx.y) * TPT;
    const int pos0 = __ldcg(wh.posp), tlast = min(n_tok, t0 + TPT) - 1;
    const int ntile = (pos0 + tlast + AT_KT) / AT_KT;         // key tiles that the last token sees
    volatile int* ab = &S.abort_flag;

    if (tid == 0) {
        for (int i = 0; i < AT_RING; i++) { mb_init(&S.full[i], 1); mb_init(&S.empty[i], 1); }
        mb_init(&S.q_ready, 8); mb_init(&S.s_full, 1); mb_init(&S.p_ready, 8); mb_init(&S.pv_full, 1);
        S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(s_u32(&S.tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;

    if (warp == 0) {
        if (lane == 0) {
            const uint8_t* src = pieces + (size_t)kvh * ktiles * 12 * AT_PIECE;
            uint32_t slot = 0, round = 0;
            bool ok = true;
            for (int i = 0; i < ntile * 12 && ok; i++) {
                if (round > 0 && !mb_wait(&S.empty[slot], (round - 1) & 1, ab)) { ok = false; break; }
                mb_expect(&S.full[slot], AT_PIECE);
                bulk_load(ring + slot * AT_PIECE, src + (size_t)i * AT_PIECE, AT_PIECE, &S.full[slot]);
                if (++slot == AT_RING) { slot = 0; round++; }
            }
            if (!ok)
                for (int i = 0; i < AT_RING; i++) {
                    const uint32_t uses = round + ((uint32_t)i < slot ? 1u : 0u);
                    if (uses > 0) mb_drain(&S.full[i], (uses - 1) & 1);
                }
        }
    } else if (warp == 1) {
        // bf16 x bf16 -> f32, K-major both, M = 128, N = 128, K = 16
        constexpr uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | (8u << 24);
        const uint64_t dR = smem_desc(s_u32(ring), 16, 1024, SW128), dQ = smem_desc(s_u32(sq), 16, 1024, SW128);
        uint32_t slot = 0, par = 0;
        bool ok = warp_wait(&S.q_ready, 0, ab);
        tc_fence_after();
        for (int j = 0; j < ntile && ok; j++) {
#pragma unroll
            for (int ph = 0; ph < 2; ph++) {
                if (ph == 1) { ok = warp_wait(&S.p_ready, (uint32_t)j & 1u, ab); if (!ok) break; tc_fence_after(); }
#pragma unroll
                for (int pc = 0; pc < 6; pc++) {              // lo0 lo1 mid0 mid1 hi0 hi1
                    if (ok) ok = warp_wait(&S.full[slot], par, ab);
                    if (!ok) break;
                    tc_fence_after();
                    const int half = pc & 1, terms = (pc >> 1) + 1;      // lo meets hi; mid meets hi, mid; hi meets all three
                    const uint64_t b = dR + (uint64_t)(slot * (AT_PIECE >> 4));
                    if (tc_elect()) {
#pragma unroll
                        for (int st = 0; st < 4; st++)
#pragma unroll
                            for (int t = 0; t < terms; t++) {
                                const uint32_t acc = (pc > 0 || st > 0) ? 1u : 0u;
                                if (ph == 0) mma_ss(tmem + TM_S, dQ + (uint64_t)((t * 2 + half) * (AT_PIECE >> 4) + st * 2), b + (uint64_t)(st * 2), idesc, acc);
                                else mma_ts(tmem + TM_PV, tmem + TM_P + (uint32_t)(t * 64 + half * 32 + st * 8), b + (uint64_t)(st * 2), idesc, acc);
                            }
                        tc_commit(&S.empty[slot]);
                        if (pc == 5) tc_commit(ph == 0 ? &S.s_full : &S.pv_full);
                    }
                    __syncwarp();
                    if (++slot == AT_RING) { slot = 0; par ^= 1u; }
                }
            }
        }
    } else {
        const int sub = warp & 3, half = (warp - 2) >> 2, row = sub * 32 + lane, st = tid - 64;
        // ---- Q rows of the tile (query head of the group fastest) as terms ----
#pragma unroll 2
        for (int n = 0; n < 8; n++) {
            const int i = n * 256 + st, r = i >> 4, c = i & 15, tok = t0 + r / GRP;
            float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (r < TPT * GRP && tok < n_tok) {
                const float4* p = reinterpret_cast<const float4*>(qkv + (size_t)tok * ld + (size_t)(kvh * GRP + r % GRP) * AT_DH + c * 8);
                const float4 a = __ldcg(p), b = __ldcg(p + 1);
                v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
            }
            uint4 h, m, l;
            split8(v, h, m, l);
            uint8_t* o = sq + (size_t)(c >> 3) * AT_PIECE + r * 128 + (((c & 7) ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(o) = h; *reinterpret_cast<uint4*>(o + 2 * AT_PIECE) = m; *reinterpret_cast<uint4*>(o + 4 * AT_PIECE) = l;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mb_arrive(&S.q_ready);

        const int tok = t0 + row / GRP;
        const bool valid = row < TPT * GRP && tok < n_tok;
        const int nk = pos0 + min(tok, tlast) + 1;            // keys this row sees
        const uint32_t tl = tmem + ((uint32_t)(sub * 32) << 16);
        float m_run = -100000000.0f, l_run = 0.0f, r_prev = 1.0f;      // seeded like fused_decode_attn_kernel.hx:74-102
        float acc[64];
#pragma unroll
        for (int d = 0; d < 64; d++) acc[d] = 0.0f;
        auto add_pv = [&]() {                                  // acc = acc * r_prev + P V of the tile before
#pragma unroll
            for (int b = 0; b < 4; b++) {
                uint32_t r[16];
                tm_ld16(r, tl + TM_PV + (uint32_t)(half * 64 + b * 16));
                tc_wait_ld();
#pragma unroll
                for (int d = 0; d < 16; d++) acc[b * 16 + d] = fmaf(acc[b * 16 + d], r_prev, __uint_as_float(r[d]));
            }
        };
        bool ok = true;
        for (int j = 0; j < ntile; j++) {
            // (The P V before it is complete too: the pipe works in order.)  After a wait that ran out the warp keeps to the
            // barriers that it shares with its partner and touches nothing.
            ok = ok && warp_wait(&S.s_full, (uint32_t)j & 1u, ab);
            tc_fence_after();
            float s[64];
            float tm = -INFINITY;
            const int lim = nk - (j * AT_KT + half * 64);      // keys of this half that the row sees
#pragma unroll
            for (int b = 0; b < 4; b++) {
                uint32_t r[16];
                if (ok) { tm_ld16(r, tl + TM_S + (uint32_t)(half * 64 + b * 16)); tc_wait_ld(); }
                else {
#pragma unroll
                    for (int e = 0; e < 16; e++) r[e] = 0u;
                }
#pragma unroll
                for (int e = 0; e < 16; e++) {
                    const int k = b * 16 + e;
                    s[k] = k < lim ? __uint_as_float(r[e]) * scale : -INFINITY;
                    tm = fmaxf(tm, s[k]);
                }
            }
            S.ex[j & 1][half][row] = tm;
            asm volatile("bar.sync %0, 64;" :: "r"(1 + sub) : "memory");      // the two warps that share these rows
            const float mn = fmaxf(m_run, fmaxf(tm, S.ex[j & 1][half ^ 1][row]));
            if (j > 0 && ok) add_pv();
            r_prev = __expf(m_run - mn);
            m_run = mn;
            float ls = 0.0f;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                uint32_t h[8], m[8], l[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const float p0 = __expf(s[b * 16 + 2 * e] - mn), p1 = __expf(s[b * 16 + 2 * e + 1] - mn);
                    ls += p0 + p1;
                    split2(p0, p1, h[e], m[e], l[e]);
                }
                const uint32_t c = tl + TM_P + (uint32_t)(half * 32 + b * 8);
                if (ok) { tm_st8(c, h); tm_st8(c + 64, m); tm_st8(c + 128, l); }
            }
            l_run = l_run * r_prev + ls;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive(&S.p_ready);
        }
        ok = ok && warp_wait(&S.pv_full, (uint32_t)(ntile - 1) & 1u, ab);
        if (ok) {
            tc_fence_after();
            add_pv();
        }
        S.ex[ntile & 1][half][row] = l_run;
        asm volatile("bar.sync %0, 64;" :: "r"(1 + sub) : "memory");
        const float inv_l = l_run + S.ex[ntile & 1][half ^ 1][row];
        if (ok && valid && !S.abort_flag) {
            float4* o = reinterpret_cast<float4*>(ctx + (size_t)tok * ld_ctx + (size_t)(kvh * GRP + row % GRP) * AT_DH + half * 64);
#pragma unroll
            for (int d = 0; d < 16; d++) o[d] = make_float4(acc[4 * d] / inv_l, acc[4 * d + 1] / inv_l, acc[4 * d + 2] / inv_l, acc[4 * d + 3] / inv_l);
        }
        tc_fence_before();
    }
    __syncthreads();
    if (S.abort_flag && tid == 0 && err) *err = 1;
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
    }
}

}  // namespace

// Bytes of the term pieces for a context of `ctx` positions.
size_t hx_pf_attn_tc_bytes(int ctx, int NKV) { return (size_t)NKV * ((ctx + AT_KT - 1) / AT_KT) * 12 * AT_PIECE; }

// head_dim 128 and a group that shares a row tile
bool hx_pf_attn_tc_takes(int NH, int NKV, int DH) { return DH == AT_DH && NH % NKV == 0 && NH / NKV <= 8; }

// Whether a chunk of n_tok tokens that ends at position ctx should go this way (if it can).  A row tile costs about 4.5 us per key
// tile however few of its rows exist and the key runs are not split over CTAs, while the vector kernel (hx_pf_attn) costs about
// 1.5 ns per (token, key) of eight kv heads plus 8 us and splits them: it keeps the small windows at a long context.  Prompts on 8
// layers of the 8B shape, this kernel / the vector kernel, us: 24 tokens 857 / 792, 64 1158 / 1104, 80 1324 / 1329, 96 1358 / 1361,
// 128 1581 / 1627, 160 1792 / 1952, 200 2079 / 2207; the rule changes over between 80 and 112.
bool hx_pf_attn_tc_wanted(int n_tok, int ctx, int NH, int NKV) {
    const int tpt = 128 / (NH / NKV), rt = (n_tok + tpt - 1) / tpt, kt = (ctx + AT_KT - 1) / AT_KT;
    const double waves = (rt * NKV + 147) / 148;
    const double tc = 8.0 + waves * (3.0 + 4.5 * (kt - 0.5 * (double)n_tok / AT_KT)), vec = 8.0 + 1.5e-3 * n_tok * (ctx - 0.5 * n_tok) * NH / 32.0;
    return tc < vec;
}

int hx_pf_attn_tc(const float* qkv, int ld, int n_tok, HxPfWhere wh, int NH, int NKV, const float* kc, const float* vc, int cap, float scale,
                  float* ctx, int ld_ctx, uint8_t* pieces, int ctx_len, int* err, cudaStream_t st) {
    HX_CHECK_ARG(!wh.pos_arr && pieces && NH % NKV == 0 && NH / NKV <= 128);
    const int GRP = NH / NKV, tpt = 128 / GRP, kt = (ctx_len + AT_KT - 1) / AT_KT;
    const size_t smem = 1024 + AT_HDR + (size_t)(6 + AT_RING) * AT_PIECE;
    static HxOncePerDevice once;
    const int rc = hx_max_smem(once, k_pf_attn_tc, 227 * 1024); if (rc) return rc;
    HX_CUDA(hx_launch_pdl(k_pf_kv_split, dim3(kt, NKV, 4), dim3(256), 0, st, kc, vc, wh, n_tok, cap, pieces));
    HX_CUDA(hx_launch_pdl(k_pf_attn_tc, dim3(NKV, (n_tok + tpt - 1) / tpt), dim3(AT_THREADS), smem, st, qkv, ld, wh, n_tok, GRP, pieces, kt, scale, ctx, ld_ctx, err));
    HX_COUNT_LAUNCH(2);
    HX_CUDA(cudaGetLastError());
    return HX_OK;
}
