// hx_prefill.cu -- batched prefill around the tcgen05 GEMM.
//
// Replaces forward_layer_llama / forward_full (helixc/runtime/gpt2_infer.c:1231-1333): where the reference runs
// f32 tiled_matmul_abt over a dequantized weight copy per layer, a chunk of prompt tokens here is one
// block-scaled NVFP4 GEMM per linear with the weights read in their packed form.  The activations enter the FP4
// tensor path as digits: after the optional RMSNorm each element is x = s_b * sum_d digit_d 13^(7-d) with eight base-13 digits
// of the integer x / S_b * 2^27 (S_b: the power of two at or below the largest element of the value's 32-column block b), every
// digit an E2M1 column; S_b over the vector's S is the column's block scale, the GEMM epilogue folds the eight accumulators
// of a token.  (The decode kernel uses sixteen exact base-4 digits: there the column count is free.)
// Norm, RoPE, KV append and attention are small f32 kernels over the chunk.
#include "hx_tc.cuh"
#include "hx_prefill.cuh"
#include "hx_digits.cuh"
#include "hx_kernels.cuh"
#include <math.h>

namespace {

__global__ void __launch_bounds__(256) k_pf_embed(const int* __restrict__ ids, HxPfWhere wh, const float* __restrict__ emb, const float* __restrict__ wpe, float* __restrict__ X, int DM) {
    hx_grid_dep_launch();
    const int t = blockIdx.x, pos = wh.pos_arr ? __ldcg(wh.pos_arr + t) : __ldcg(wh.posp) + t;
    const float4* src = reinterpret_cast<const float4*>(emb + (size_t)ids[wh.pos_arr ? t : pos] * DM);
    const float4* add = wpe ? reinterpret_cast<const float4*>(wpe + (size_t)pos * DM) : nullptr;
    float4* dst = reinterpret_cast<float4*>(X + (size_t)t * DM);
    for (int i = threadIdx.x; i < DM / 4; i += blockDim.x) {
        float4 v = src[i];
        if (add) { const float4 p = add[i]; v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w; }
        dst[i] = v;
    }
}

// grid (token, slice of 4096 columns), 512 threads: a thread takes eight consecutive elements and turns them into one 32-bit
// word per digit.  The statistics of a token with several slices are put together by a cluster (up to PFD_CL slices) through
// distributed shared memory; beyond that every CTA reads the whole vector.
// A warp holds a 256-column cell of the token; the digits are those of hx_digits.cuh.
// (Ten balanced base-9 digits against the vector's S: 25 % more columns for the tensor pipe, and the digits of a vector with one
// large element resolved 2^-29 of it everywhere; now 2^-27 of it in its own block and 2^-27 of the block's largest in the others.)
#define PFD_T 512
#define PFD_CL 8                    // CTAs of a token at most for a cluster
template <bool CL, bool LN>              // statistics by a cluster; LayerNorm instead of RMSNorm
__global__ void __launch_bounds__(PFD_T, 3) k_pf_digits(const float* __restrict__ src, int ld, int K, const float* __restrict__ g, const float* __restrict__ lb,
                                                     float eps, uint8_t* __restrict__ cells, int group, int groups, float* __restrict__ scale) {
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ float part[PFD_CL][2];    // (sum of squares, largest) of the token's slices
    hx_grid_dep_launch();
    if (CL) hxtc::cl_sync();             // every CTA of the cluster runs before a store into it
    hx_grid_dep_wait();
    const float* x = src + (size_t)t * ld;
    __shared__ float red[2 * PFD_T / 32];
    __shared__ uint8_t codes[HX_DIG_CODES];
    if (tid < HX_DIG_CODES) codes[tid] = dig_code(tid);
    const int k0 = (blockIdx.y * PFD_T + tid) * 8;       // this thread's item
    float v[8], ss = 0.0f, mx = 0.0f;
    {
        const bool in0 = k0 < K, in1 = k0 + 4 < K;       // K is a multiple of four
        const float4 z = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
        const float4 a = in0 ? __ldcg(reinterpret_cast<const float4*>(x + k0)) : z, b = in1 ? __ldcg(reinterpret_cast<const float4*>(x + k0 + 4)) : z;
        const float4 ga = (g && in0) ? __ldg(reinterpret_cast<const float4*>(g + k0)) : one, gb = (g && in1) ? __ldg(reinterpret_cast<const float4*>(g + k0 + 4)) : one;
        v[0] = a.x * ga.x; v[1] = a.y * ga.y; v[2] = a.z * ga.z; v[3] = a.w * ga.w;
        v[4] = b.x * gb.x; v[5] = b.y * gb.y; v[6] = b.z * gb.z; v[7] = b.w * gb.w;
        ss = ((a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w)) + ((b.x * b.x + b.y * b.y) + (b.z * b.z + b.w * b.w));
    }
    float inv = 1.0f, probe;             // probe: not a number when an element of the vector is not
    if (LN) {
        // LayerNorm (GPT-2): mean, then variance about it, then the largest result
        float mean = 0.0f;
        for (int ps = 0; ps < 2; ps++) {
            float s = 0.0f;
            for (int k = tid * 4; k < K; k += PFD_T * 4) {
                const float4 a = __ldcg(reinterpret_cast<const float4*>(x + k));
                if (ps == 0) s += (a.x + a.y) + (a.z + a.w);
                else s += ((a.x - mean) * (a.x - mean) + (a.y - mean) * (a.y - mean)) + ((a.z - mean) * (a.z - mean) + (a.w - mean) * (a.w - mean));
            }
            s = hx_warp_sum(s);
            __syncthreads();
            if (lane == 0) red[warp] = s;
            __syncthreads();
            s = 0.0f;
#pragma unroll
            for (int i = 0; i < PFD_T / 32; i++) s += red[i];
            if (ps == 0) mean = s / (float)K; else inv = rsqrtf(s / (float)K + eps);
        }
        for (int k = tid * 4; k < K; k += PFD_T * 4) {
            const float4 a = __ldcg(reinterpret_cast<const float4*>(x + k)), ga = __ldg(reinterpret_cast<const float4*>(g + k)), ba = __ldg(reinterpret_cast<const float4*>(lb + k));
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(ga.x * ((a.x - mean) * inv) + ba.x), fabsf(ga.y * ((a.y - mean) * inv) + ba.y)),
                                 fmaxf(fabsf(ga.z * ((a.z - mean) * inv) + ba.z), fabsf(ga.w * ((a.w - mean) * inv) + ba.w))));
        }
#pragma unroll
        for (int e = 0; e < 8; e++) v[e] = k0 + e < K ? __ldg(g + k0 + e) * ((__ldcg(x + k0 + e) - mean) * inv) + __ldg(lb + k0 + e) : 0.0f;
        probe = inv; inv = 1.0f;
        mx = hx_warp_max(mx);
        __syncthreads();
        if (lane == 0) red[PFD_T / 32 + warp] = mx;
        __syncthreads();
    } else {
    // sum of squares (of x) and largest |x * g| of the whole vector
    if (CL || gridDim.y == 1) {
#pragma unroll
        for (int e = 0; e < 8; e++) mx = fmaxf(mx, fabsf(v[e]));
    } else {
        ss = 0.0f;
        #pragma unroll 4
        for (int k = tid * 4; k < K; k += PFD_T * 4) {
            const float4 a = __ldcg(reinterpret_cast<const float4*>(x + k));
            const float4 ga = g ? __ldg(reinterpret_cast<const float4*>(g + k)) : make_float4(1.f, 1.f, 1.f, 1.f);
            ss = fmaf(a.x, a.x, ss); ss = fmaf(a.y, a.y, ss); ss = fmaf(a.z, a.z, ss); ss = fmaf(a.w, a.w, ss);
            mx = fmaxf(mx, fmaxf(fmaxf(fabsf(a.x * ga.x), fabsf(a.y * ga.y)), fmaxf(fabsf(a.z * ga.z), fabsf(a.w * ga.w))));
        }
    }
    ss = hx_warp_sum(ss); mx = hx_warp_max(mx);
    if (lane == 0) { red[warp] = ss; red[PFD_T / 32 + warp] = mx; }
    __syncthreads();
    static_assert(PFD_T / 32 == 16, "the warps' results are folded by sixteen lanes");
    float tss = red[lane & 15];
    mx = red[PFD_T / 32 + (lane & 15)];
#pragma unroll
    for (int d = 8; d >= 1; d >>= 1) { tss += __shfl_xor_sync(0xffffffffu, tss, d); mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d)); }
    if (CL) {
        if (tid < (int)gridDim.y) {
            const uint32_t to = hxtc::cl_map(hxtc::s_u32(&part[blockIdx.y][0]), (uint32_t)tid);
            hxtc::cl_st(to, tss); hxtc::cl_st(to + 4, mx);
        }
        hxtc::cl_sync();
        tss = 0.0f;
        for (int i = 0; i < (int)gridDim.y; i++) { tss += part[i][0]; mx = fmaxf(mx, part[i][1]); }
    }
    probe = tss;
    if (g) inv = rsqrtf(tss / (float)K + eps);
    }
    if (LN) {
        mx = red[PFD_T / 32 + (lane & 15)];
#pragma unroll
        for (int d = 8; d >= 1; d >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, d));
    }
    const float vmax = mx * inv * 1.0000005f, Sg = dig_scale(vmax);
    // digits cannot spell infinities or NaN: the scale does, so that the token's outputs show them
    if (tid == 0 && blockIdx.y == 0) scale[t] = (vmax < INFINITY && probe == probe) ? Sg * (2.0f / HX_TC_DIGIT_UNIT) : __int_as_float(0x7FC00000);
    if (k0 >= ((K + 255) & ~255)) return;
    const int r = dig_block_exp(Sg, dig_block_max(v) * inv * 1.0000005f);        // the warp's 256 columns are a cell
    uint32_t word[HX_TC_DIGITS];
    dig_words(v, (inv / Sg) * (float)(1 << r) * HX_TC_DIGIT_UNIT, codes, word);
    const int tg = t / group;
    dig_store(cells + ((size_t)(k0 >> 8) * groups + tg) * HX_TC_DCELL(group), group, t - tg * group, lane, word, r);
}

// The same for long chunks (no LayerNorm): one CTA of 256 threads per token, its values kept in shared memory between the statistics and
// the digits, a warp a cell at a time.  All tokens of a chunk are on the SMs at once where the kernel above, a CTA of 512
// threads per 4096 columns and a cluster's exchange at K = 12288, takes several waves of CTAs that wait most of their time.
#define PFL_T 256
__global__ void __launch_bounds__(PFL_T, 5) k_pf_digits_long(const float* __restrict__ src, int ld, int K, const float* __restrict__ g, float eps, uint8_t* __restrict__ cells,
                                                             int group, int groups, float* __restrict__ scale) {
    extern __shared__ __align__(16) float xs[];            // K rounded up to whole cells
    __shared__ float red[2 * PFL_T / 32];
    __shared__ uint8_t codes[HX_DIG_CODES];
    const int t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, kcells = (K + 255) >> 8;
    hx_grid_dep_launch();
    if (tid < HX_DIG_CODES) codes[tid] = dig_code(tid);
    hx_grid_dep_wait();
    const float* x = src + (size_t)t * ld;
    float ss = 0.0f, mx = 0.0f;
    #pragma unroll 4
    for (int k = tid * 4; k < kcells * 256; k += PFL_T * 4) {
        const bool in = k < K;                             // K is a multiple of four
        const float4 a = in ? __ldcg(reinterpret_cast<const float4*>(x + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float4 ga = (g && in) ? __ldg(reinterpret_cast<const float4*>(g + k)) : make_float4(1.f, 1.f, 1.f, 1.f);
        const float4 v = make_float4(a.x * ga.x, a.y * ga.y, a.z * ga.z, a.w * ga.w);
        *reinterpret_cast<float4*>(xs + k) = v;
        ss += (a.x * a.x + a.y * a.y) + (a.z * a.z + a.w * a.w);
        mx = fmaxf(mx, fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w))));
    }
    ss = hx_warp_sum(ss); mx = hx_warp_max(mx);
    if (lane == 0) { red[warp] = ss; red[PFL_T / 32 + warp] = mx; }
    __syncthreads();
    ss = 0.0f;
#pragma unroll
    for (int i = 0; i < PFL_T / 32; i++) { ss += red[i]; mx = fmaxf(mx, red[PFL_T / 32 + i]); }
    const float inv = g ? rsqrtf(ss / (float)K + eps) : 1.0f;
    const float vmax = mx * inv * 1.0000005f, Sg = dig_scale(vmax);
    // digits cannot spell infinities or NaN: the scale does, so that the token's outputs show them
    if (tid == 0) scale[t] = (vmax < INFINITY && ss == ss) ? Sg * (2.0f / HX_TC_DIGIT_UNIT) : __int_as_float(0x7FC00000);
    const int tg = t / group, tl = t - tg * group;
    #pragma unroll 1
    for (int c = warp; c < kcells; c += PFL_T / 32) {
        float v[8];
        const float4 a = *reinterpret_cast<const float4*>(xs + c * 256 + lane * 8), b = *reinterpret_cast<const float4*>(xs + c * 256 + lane * 8 + 4);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
        const int r = dig_block_exp(Sg, dig_block_max(v) * inv * 1.0000005f);
        uint32_t word[HX_TC_DIGITS];
        dig_words(v, (inv / Sg) * (float)(1 << r) * HX_TC_DIGIT_UNIT, codes, word);
        dig_store(cells + ((size_t)c * groups + tg) * HX_TC_DCELL(group), group, tl, lane, word, r);
    }
}

// q/k norm, rotate_half RoPE and KV append: a warp per (head section, token), EPL = DH / 32 consecutive elements per lane, so a
// row is one vector load per lane, the sum of squares one warp reduction and the rotation partner one exchange with lane ^ 16;
// grid (head sections / 8, n_tok / TPW).  Latency is what bounds it: loads of a row, gains and angles in flight together, no barrier,
// and for long chunks TPW tokens per warp, whose rows are on their way together.  (A CTA of DH threads per row with three barriers: 9.5
// us for 77 tokens of the 8B shape, 22 for 512; a token per warp 4.9 and 14.6.)
#define PF_QK_W 8
template <int EPL, int TPW>
__global__ void __launch_bounds__(PF_QK_W * 32) k_pf_qkpost(float* __restrict__ qkv, int ld, HxPfWhere wh, int n_tok, int NH, int NKV,
                                                    const float* __restrict__ qn_g, const float* __restrict__ kn_g, float eps,
                                                    const float* __restrict__ cosT, const float* __restrict__ sinT,
                                                    float* __restrict__ kc, float* __restrict__ vc, int cap) {
    constexpr int DH = 32 * EPL, half = DH / 2, VEC = EPL < 4 ? EPL : 4, NV = EPL / VEC;
    struct __align__(4 * VEC) Vec { float f[VEC]; };
    hx_grid_dep_launch();
    const int hs = blockIdx.x * PF_QK_W + (threadIdx.x >> 5), t0 = blockIdx.y * TPW, lane = threadIdx.x & 31;
    if (hs >= NH + 2 * NKV) return;
    const int sec = hs < NH ? 0 : (hs < NH + NKV ? 1 : 2), e0 = lane * EPL, er = e0 & (half - 1);
    const float* gg = sec == 0 ? qn_g : (sec == 1 ? kn_g : nullptr);
    auto load = [](const float* p, float (&v)[EPL], bool fresh) {
#pragma unroll
        for (int i = 0; i < NV; i++) {
            Vec x;
            if (EPL == 1) x.f[0] = fresh ? __ldcg(p) : __ldg(p);
            else if (EPL == 2) { const float2 y = fresh ? __ldcg(reinterpret_cast<const float2*>(p)) : __ldg(reinterpret_cast<const float2*>(p)); x.f[0] = y.x; x.f[VEC > 1 ? 1 : 0] = y.y; }
            else {
                const float4 y = fresh ? __ldcg(reinterpret_cast<const float4*>(p) + i) : __ldg(reinterpret_cast<const float4*>(p) + i);
                x.f[0] = y.x; x.f[VEC > 1 ? 1 : 0] = y.y; x.f[VEC > 2 ? 2 : 0] = y.z; x.f[VEC > 3 ? 3 : 0] = y.w;
            }
#pragma unroll
            for (int c = 0; c < VEC; c++) v[i * VEC + c] = x.f[c];
        }
    };
    float v[TPW][EPL], g[EPL], cs[TPW][EPL], sn[TPW][EPL];
    if (gg) load(gg + e0, g, false);
    hx_grid_dep_wait();
    const int first = wh.pos_arr ? 0 : __ldcg(wh.posp) + t0;
    const bool rot = cosT && sec < 2;
    float* row = qkv + (size_t)t0 * ld + (size_t)hs * DH + e0;
    int pos[TPW];
#pragma unroll
    for (int k = 0; k < TPW; k++) {
        if (TPW > 1 && t0 + k >= n_tok) break;
        pos[k] = wh.pos_arr ? __ldcg(wh.pos_arr + t0 + k) : first + k;
        load(row + (size_t)k * ld, v[k], true);
        if (rot) { load(cosT + (size_t)pos[k] * half + er, cs[k], false); load(sinT + (size_t)pos[k] * half + er, sn[k], false); }
    }
#pragma unroll
    for (int k = 0; k < TPW; k++) {
        if (TPW > 1 && t0 + k >= n_tok) break;
        const size_t seq_off = wh.seq_arr ? (size_t)__ldcg(wh.seq_arr + t0 + k) * wh.seq_stride : (wh.seqp ? (size_t)__ldcg(wh.seqp) * wh.seq_stride : 0);
        if (gg) {
            float ssq = 0.0f;
#pragma unroll
            for (int i = 0; i < EPL; i++) ssq = fmaf(v[k][i], v[k][i], ssq);
            const float inv = rsqrtf(hx_warp_sum(ssq) / (float)DH + eps);
#pragma unroll
            for (int i = 0; i < EPL; i++) v[k][i] = g[i] * (v[k][i] * inv);
        }
        if (rot) {
#pragma unroll
            for (int i = 0; i < EPL; i++) {
                const float other = __shfl_xor_sync(0xffffffffu, v[k][i], 16);
                v[k][i] = lane < 16 ? v[k][i] * cs[k][i] - other * sn[k][i] : v[k][i] * cs[k][i] + other * sn[k][i];
            }
        }
        float* dst = sec == 0 ? row + (size_t)k * ld : (sec == 1 ? kc : vc) + seq_off + ((size_t)(hs - NH - (sec == 2 ? NKV : 0)) * cap + pos[k]) * DH + e0;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            Vec x;
#pragma unroll
            for (int c = 0; c < VEC; c++) x.f[c] = v[k][i * VEC + c];
            reinterpret_cast<Vec*>(dst)[i] = x;
        }
    }
}

// ---- causal attention of a chunk over the cache ------------------------------------------------------------------
// grid (NKV, groups of TG tokens, NS), PF_AT threads: CTA (kv head, token group, s) covers the s-th run of whole key
// tiles of the group's context (NS runs at most, fewer for a short context; CTAs without a run leave at once).
// The K and V rows of a tile are contiguous in the cache, so one thread brings each tile into a ring of PF_ST
// shared-memory stages with two bulk copies (cp.async.bulk, completion on an mbarrier), PF_ST - 1 tiles ahead of the
// arithmetic: the loads of a CTA never wait for its softmax.  In a prefill chunk (one sequence, consecutive positions)
// the TG = 4 tokens of a group share every tile; in batched decode every token has a cache of its own (TG = 1).
// Per token: online softmax over the tiles (m seeded -1e8 like fused_decode_attn_kernel.hx:74-102).  Scores: a warp
// takes four keys at a time against every (token, head) query, the 4 x GRP dot products of a token are reduced across
// the lanes together (each exchange halves the values a lane carries).  Softmax step: a warp per (token, head).
// P*V: thread (dimension, run of keys inside the tile), a V value serving all tokens and heads; the runs are added
// up through shared memory at the end.  With more than one active run per (token group, kv head) each CTA leaves (sum, m, l) in
// `part`, and the last one to finish (a ticket per (token group, kv head)) merges them.  Waits are bounded: after a
// wait that ran out the CTA keeps to its barriers, writes nothing and raises *err.
#define PF_AT 512
#define PF_ST 3
#define PF_NS_MAX 16
#define PF_TILE_BYTES 32768          // K rows of a tile (and as many V rows)
#define PF_AT_WAIT (1u << 22)
__device__ __forceinline__ uint32_t pf_s32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool pf_mb_wait(uint64_t* b, uint32_t parity) {
    for (uint32_t i = 0; i < PF_AT_WAIT; i++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(pf_s32(b)), "r"(parity) : "memory");
        if (ok) return true;
    }
    return false;
}
template <int GRP, int TG>
__global__ void __launch_bounds__(PF_AT) k_pf_attn(const float* __restrict__ qkv, int ld, HxPfWhere wh, int n_tok, int NH, int DH,
                                                    const float* __restrict__ kc, const float* __restrict__ vc, int cap, float scale,
                                                    float* __restrict__ ctx, int ld_ctx, float* __restrict__ part, unsigned* __restrict__ tickets, int* err) {
    extern __shared__ __align__(128) float smf[];
    hx_grid_dep_launch();
    hx_grid_dep_wait();
    // The groups with the longest contexts start first: what is left for a second wave is short (77 tokens of the 8B shape, 160 CTAs: 23.7 -> 18.5 us).
    const int kvh = blockIdx.x, t0 = (TG > 1 ? gridDim.y - 1 - blockIdx.y : blockIdx.y) * TG, s = blockIdx.z, NS = gridDim.z, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = PF_AT / 32;
    constexpr int GP = GRP <= 1 ? 1 : (GRP <= 2 ? 2 : (GRP <= 4 ? 4 : 8));      // GRP rounded up to a power of two
    constexpr int NP = 4 * GP;                                                   // values reduced together (4 keys x GP heads)
    constexpr int LG = NP == 4 ? 2 : (NP == 8 ? 3 : (NP == 16 ? 4 : 5));
    const int KT = min(128, PF_TILE_BYTES / (DH * 4));                           // keys per tile (32 .. 128, a multiple of 32)
    const int ntk = min(TG, n_tok - t0);                                         // tokens of this group
    const int pos0 = wh.pos_arr ? __ldcg(wh.pos_arr + t0) : __ldcg(wh.posp) + t0;                // TG > 1 only with consecutive positions
    const int Tmax = pos0 + ntk;                                                 // context of the group's last token
    const int tiles = (Tmax + KT - 1) / KT, per = ((tiles + NS - 1) / NS) * KT;  // keys per run: whole tiles
    const int n_act = (Tmax + per - 1) / per;
    if (s >= n_act) return;
    const int j_lo = s * per, j_hi = min(Tmax, j_lo + per);
    const size_t seq_off = wh.seq_arr ? (size_t)__ldcg(wh.seq_arr + t0) * wh.seq_stride : (wh.seqp ? (size_t)__ldcg(wh.seqp) * wh.seq_stride : 0);
    // shared memory: ring [PF_ST][K tile | V tile], then q, p and the P*V partial outputs
    float* ringf = smf;
    const int stage_f = 2 * (PF_TILE_BYTES / 4);
    float* sq = smf + PF_ST * stage_f;         // [TG][GRP][DH]
    float* sp = sq + TG * GRP * DH;            // [TG][GRP][128]
    float* sacc = sp + TG * GRP * 128;              // [nsub][GRP][DH] partial outputs of the key runs inside a tile
    __shared__ float sm_m[TG][GRP], sm_l[TG][GRP], sm_r[TG][GRP];
    __shared__ unsigned sm_ticket;
    __shared__ int sm_abort;
    __shared__ __align__(8) uint64_t full[PF_ST];
    for (int i = tid; i < ntk * GRP * DH; i += PF_AT) {
        const int tk = i / (GRP * DH), r = i - tk * GRP * DH;
        sq[i] = __ldcg(qkv + (size_t)(t0 + tk) * ld + (size_t)kvh * GRP * DH + r);
    }
    if (tid < TG * GRP) { sm_m[tid / GRP][tid % GRP] = -100000000.0f; sm_l[tid / GRP][tid % GRP] = 0.0f; }
    if (tid == 0) {
        sm_abort = 0;
        for (int i = 0; i < PF_ST; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(pf_s32(&full[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const float* kbase = kc + seq_off + (size_t)kvh * cap * DH;
    const float* vbase = vc + seq_off + (size_t)kvh * cap * DH;
    const int ntile = (j_hi - j_lo + KT - 1) / KT;
    auto issue = [&](int it) {       // thread 0: tile `it` of this run into its stage
        const int j0 = j_lo + it * KT, nj = min(KT, j_hi - j0);
        const uint32_t bytes = (uint32_t)nj * DH * 4;
        float* st = ringf + (size_t)(it % PF_ST) * stage_f;
        uint64_t* bar = &full[it % PF_ST];
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(pf_s32(bar)), "r"(2 * bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(pf_s32(st)), "l"(kbase + (size_t)j0 * DH), "r"(bytes), "r"(pf_s32(bar)) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     :: "r"(pf_s32(st + PF_TILE_BYTES / 4)), "l"(vbase + (size_t)j0 * DH), "r"(bytes), "r"(pf_s32(bar)) : "memory");
    };
    if (tid == 0) for (int it = 0; it < PF_ST - 1 && it < ntile; it++) issue(it);
    const int nsub = PF_AT / DH, d = tid % DH, ksub = tid / DH;      // DH divides PF_AT (32, 64, 128, 256)
    const int krun = KT / nsub;                                      // keys of a tile per P*V thread: a multiple of 4
    float acc[TG][GRP];
#pragma unroll
    for (int tk = 0; tk < TG; tk++)
#pragma unroll
        for (int i = 0; i < GRP; i++) acc[tk][i] = 0.0f;
    // Batched decode at head_dim 128 (tiles of 64 keys): a leaner arrangement of the same arithmetic.  Scores: thread (key,
    // eighth of the row) with its slice of q in registers (groups of up to four heads) -- chunk c * 8 + eighth of the row, so that the eight lanes of a
    // key read eight different bank groups -- and three exchanges per head.  P*V: a warp per four keys, a lane per
    // float4 of the row; the sixteen warps' sums are added up through the (then idle) ring at the end.
    constexpr bool kLean = TG == 1;
    constexpr bool kQreg = GRP <= 4;       // larger groups read q from shared memory (eight lanes, one 128-byte row: a broadcast)
    const bool lean = kLean && DH == 128;
    float acc4[kLean ? GRP : 1][4];
#pragma unroll
    for (int i = 0; i < (kLean ? GRP : 1); i++) acc4[i][0] = acc4[i][1] = acc4[i][2] = acc4[i][3] = 0.0f;
    if (lean) {
        const int key = tid >> 3, pt = tid & 7;
        float4 qr[(kLean && kQreg) ? GRP : 1][4];
#pragma unroll
        for (int i = 0; i < ((kLean && kQreg) ? GRP : 1); i++)
#pragma unroll
            for (int c = 0; c < 4; c++) qr[i][c] = *reinterpret_cast<const float4*>(sq + i * 128 + (c * 8 + pt) * 4);
        for (int it = 0; it < ntile; it++) {
            const int j0 = j_lo + it * 64, nj = min(64, j_hi - j0);
            if (tid == 0 && it + PF_ST - 1 < ntile) issue(it + PF_ST - 1);
            if (!pf_mb_wait(&full[it % PF_ST], (uint32_t)(it / PF_ST) & 1u)) sm_abort = 1;
            const float* kt = ringf + (size_t)(it % PF_ST) * stage_f;
            const float* vt = kt + PF_TILE_BYTES / 4;
            {
                float4 k4[4];
#pragma unroll
                for (int c = 0; c < 4; c++) k4[c] = *reinterpret_cast<const float4*>(kt + key * 128 + (c * 8 + pt) * 4);
                float dot[kLean ? GRP : 1];
#pragma unroll
                for (int i = 0; i < (kLean ? GRP : 1); i++) {
                    float a = 0.0f;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float4 q4 = kQreg ? qr[kQreg ? i : 0][c] : *reinterpret_cast<const float4*>(sq + i * 128 + (c * 8 + pt) * 4);
                        a = fmaf(q4.x, k4[c].x, a); a = fmaf(q4.y, k4[c].y, a); a = fmaf(q4.z, k4[c].z, a); a = fmaf(q4.w, k4[c].w, a);
                    }
                    a += __shfl_xor_sync(0xffffffffu, a, 1); a += __shfl_xor_sync(0xffffffffu, a, 2); a += __shfl_xor_sync(0xffffffffu, a, 4);
                    dot[i] = a;
                }
#pragma unroll
                for (int i = 0; i < (kLean ? GRP : 1); i++)
                    if (pt == i && key < nj) sp[i * 128 + key] = dot[i] * scale;
            }
            __syncthreads();
            for (int i = warp; i < GRP; i += NW) {
                const float s0 = lane < nj ? sp[i * 128 + lane] : -INFINITY, s1 = lane + 32 < nj ? sp[i * 128 + lane + 32] : -INFINITY;
                const float tm = hx_warp_max(fmaxf(s0, s1));
                const float mo = sm_m[0][i], mn = fmaxf(mo, tm);
                const float p0 = lane < nj ? __expf(s0 - mn) : 0.0f, p1 = lane + 32 < nj ? __expf(s1 - mn) : 0.0f;
                sp[i * 128 + lane] = p0; sp[i * 128 + lane + 32] = p1;
                const float ls = hx_warp_sum(p0 + p1);
                if (lane == 0) { const float rr = __expf(mo - mn); sm_r[0][i] = rr; sm_l[0][i] = sm_l[0][i] * rr + ls; sm_m[0][i] = mn; }
            }
            __syncthreads();
            {
                float4 p4[kLean ? GRP : 1];
#pragma unroll
                for (int i = 0; i < (kLean ? GRP : 1); i++) {
                    const float rr = sm_r[0][i];
                    acc4[i][0] *= rr; acc4[i][1] *= rr; acc4[i][2] *= rr; acc4[i][3] *= rr;
                    p4[i] = *reinterpret_cast<const float4*>(sp + i * 128 + warp * 4);
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int j = warp * 4 + u;
                    const float4 v4 = j < nj ? *reinterpret_cast<const float4*>(vt + j * 128 + lane * 4) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int i = 0; i < (kLean ? GRP : 1); i++) {
                        const float pj = u == 0 ? p4[i].x : (u == 1 ? p4[i].y : (u == 2 ? p4[i].z : p4[i].w));
                        acc4[i][0] = fmaf(pj, v4.x, acc4[i][0]); acc4[i][1] = fmaf(pj, v4.y, acc4[i][1]);
                        acc4[i][2] = fmaf(pj, v4.z, acc4[i][2]); acc4[i][3] = fmaf(pj, v4.w, acc4[i][3]);
                    }
                }
            }
            __syncthreads();
        }
    } else
    for (int it = 0; it < ntile; it++) {
        const int j0 = j_lo + it * KT, njt = min(KT, j_hi - j0);
        // every thread is past tile it - 1 (the barrier that ended it), so its stage may be refilled
        if (tid == 0 && it + PF_ST - 1 < ntile) issue(it + PF_ST - 1);
        if (!pf_mb_wait(&full[it % PF_ST], (uint32_t)(it / PF_ST) & 1u)) sm_abort = 1;
        const float* kt = ringf + (size_t)(it % PF_ST) * stage_f;
        const float* vt = kt + PF_TILE_BYTES / 4;
        const int njm = min(njt, pos0 + ntk - j0);          // keys of the tile the group's last token may see (> 0)
        // ---- scores of all tokens: a warp takes four keys at a time against every (token, head) query
        for (int jb = warp; jb < njm; jb += 4 * NW) {
            float v[TG][NP];
#pragma unroll
            for (int tk = 0; tk < TG; tk++)
#pragma unroll
                for (int i = 0; i < NP; i++) v[tk][i] = 0.0f;
            for (int e = lane * 4; e < DH; e += 128) {
                float4 k4[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int j = jb + u * NW;
                    k4[u] = j < njm ? *reinterpret_cast<const float4*>(kt + (size_t)j * DH + e) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
#pragma unroll
                for (int tk = 0; tk < TG; tk++) {
                    if (tk >= ntk) break;
#pragma unroll
                    for (int i = 0; i < GRP; i++) {
                        const float4 q4 = *reinterpret_cast<const float4*>(sq + (tk * GRP + i) * DH + e);
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            float a = v[tk][u * GP + i];
                            a = fmaf(q4.x, k4[u].x, a); a = fmaf(q4.y, k4[u].y, a); a = fmaf(q4.z, k4[u].z, a); a = fmaf(q4.w, k4[u].w, a);
                            v[tk][u * GP + i] = a;
                        }
                    }
                }
            }
#pragma unroll
            for (int tk = 0; tk < TG; tk++) {
                if (tk >= ntk) break;
                // lanes with the exchange bit set keep the upper half of the values, the others the lower half
#pragma unroll
                for (int st = 0; st < 5; st++) {
                    const int o = 16 >> st;
                    if (st < LG) {
                        const int h = NP >> (st + 1);
                        const bool up = (lane & o) != 0;
#pragma unroll
                        for (int k = 0; k < h; k++) {
                            const float send = up ? v[tk][k] : v[tk][k + h], keep = up ? v[tk][k + h] : v[tk][k];
                            v[tk][k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                        }
                    } else v[tk][0] += __shfl_xor_sync(0xffffffffu, v[tk][0], o);
                }
                const int idx = lane >> (5 - LG), u = idx / GP, i = idx - u * GP, j = jb + u * NW;
                if ((lane & ((1 << (5 - LG)) - 1)) == 0 && i < GRP && j < njm) sp[(tk * GRP + i) * 128 + j] = v[tk][0] * scale;
            }
        }
        __syncthreads();
        // ---- softmax step of every (token, head) row: a warp per row; keys a token may not see count as absent
        for (int r = warp; r < ntk * GRP; r += NW) {
            const int tk = r / GRP, i = r - tk * GRP;
            const int nj = max(0, min(njt, pos0 + tk + 1 - j0));
            float tm = -INFINITY;
            for (int j = lane; j < nj; j += 32) tm = fmaxf(tm, sp[r * 128 + j]);
            tm = hx_warp_max(tm);
            const float mo = sm_m[tk][i], mn = fmaxf(mo, tm);
            float ls = 0.0f;
            for (int j = lane; j < KT; j += 32) {
                const float pr = j < nj ? __expf(sp[r * 128 + j] - mn) : 0.0f;
                sp[r * 128 + j] = pr; ls += pr;
            }
            ls = hx_warp_sum(ls);
            if (lane == 0) { const float rr = __expf(mo - mn); sm_r[tk][i] = rr; sm_l[tk][i] = sm_l[tk][i] * rr + ls; sm_m[tk][i] = mn; }
        }
        __syncthreads();
        // ---- P*V: a V value is fetched once for all tokens and heads
        {
#pragma unroll
            for (int tk = 0; tk < TG; tk++)
#pragma unroll
                for (int i = 0; i < GRP; i++) acc[tk][i] *= (tk < ntk ? sm_r[tk][i] : 1.0f);
            const int jlo = ksub * krun;
            for (int jj = 0; jj < krun; jj += 4) {
                const int j = jlo + jj;
                if (j >= njm) break;
                float vv[4];
#pragma unroll
                for (int u = 0; u < 4; u++) vv[u] = j + u < njm ? vt[(size_t)(j + u) * DH + d] : 0.0f;
#pragma unroll
                for (int tk = 0; tk < TG; tk++) {
                    if (tk >= ntk) break;
#pragma unroll
                    for (int i = 0; i < GRP; i++) {
                        const float4 p4 = *reinterpret_cast<const float4*>(sp + (tk * GRP + i) * 128 + j);
                        acc[tk][i] = fmaf(p4.x, vv[0], acc[tk][i]); acc[tk][i] = fmaf(p4.y, vv[1], acc[tk][i]);
                        acc[tk][i] = fmaf(p4.z, vv[2], acc[tk][i]); acc[tk][i] = fmaf(p4.w, vv[3], acc[tk][i]);
                    }
                }
            }
        }
        __syncthreads();
    }
    const bool bad = sm_abort != 0;       // (every thread passed a barrier after the last write of the flag)
    if (bad && tid == 0 && err) *err = 1;
    const int PW = GRP * (DH + 2);
    // per token: add the key runs inside the tiles up, then either the result or this run's (sum, m, l)
#pragma unroll
    for (int tk = 0; tk < TG; tk++) {
        if (tk >= ntk) break;
        const int t = t0 + tk;
        // (lean arrangement: one partial output per warp, in the ring, which no copy writes any more)
        const float* red = lean ? ringf : sacc;
        const int nred = lean ? NW : nsub;
        if (lean) {
#pragma unroll
            for (int i = 0; i < (kLean ? GRP : 1); i++)
                *reinterpret_cast<float4*>(ringf + ((size_t)warp * GRP + i) * DH + lane * 4) = make_float4(acc4[i][0], acc4[i][1], acc4[i][2], acc4[i][3]);
        } else {
#pragma unroll
            for (int i = 0; i < GRP; i++) sacc[((size_t)ksub * GRP + i) * DH + d] = acc[tk][i];
        }
        __syncthreads();
        float* mine = part + ((size_t)(t * gridDim.x + kvh) * NS + s) * PW;
        for (int o = tid; o < GRP * DH; o += PF_AT) {
            const int i = o / DH, dd = o - i * DH;
            float v = 0.0f;
            for (int u = 0; u < nred; u++) v += red[((size_t)u * GRP + i) * DH + dd];
            if (bad) continue;
            if (n_act == 1) ctx[(size_t)t * ld_ctx + (size_t)(kvh * GRP + i) * DH + dd] = v / sm_l[tk][i];
            else mine[o] = v;
        }
        if (n_act > 1 && tid < GRP && !bad) { mine[GRP * DH + tid] = sm_m[tk][tid]; mine[GRP * DH + GRP + tid] = sm_l[tk][tid]; }
        __syncthreads();
    }
    if (n_act == 1) return;
    // several runs: the last CTA of the (token group, kv head) merges the runs in order
    __threadfence();
    __syncthreads();
    if (tid == 0) sm_ticket = atomicAdd(tickets + blockIdx.y * gridDim.x + kvh, 1u);
    __syncthreads();
    if (sm_ticket != (unsigned)(n_act - 1)) return;
    __threadfence();
    for (int tk = 0; tk < ntk; tk++) {
        const int t = t0 + tk;
        const float* all = part + (size_t)(t * gridDim.x + kvh) * NS * PW;
        for (int o = tid; o < GRP * DH; o += PF_AT) {
            const int i = o / DH;
            float mx = -INFINITY;
            for (int r = 0; r < n_act; r++) mx = fmaxf(mx, __ldcg(all + (size_t)r * PW + GRP * DH + i));
            float num = 0.0f, den = 0.0f;
            for (int r = 0; r < n_act; r++) {
                const float w = __expf(__ldcg(all + (size_t)r * PW + GRP * DH + i) - mx);
                num = fmaf(w, __ldcg(all + (size_t)r * PW + o), num);
                den = fmaf(w, __ldcg(all + (size_t)r * PW + GRP * DH + GRP + i), den);
            }
            if (!bad) ctx[(size_t)t * ld_ctx + (size_t)kvh * GRP * DH + o] = num / den;
        }
    }
    if (tid == 0) tickets[blockIdx.y * gridDim.x + kvh] = 0u;
}

// Tensor-parallel chunk: the partial rows of a row-split linear (o_proj, down_proj) summed over the ranks and added to
// the residual stream.  Every rank stores its [n][DM] partial as 8-byte (value, epoch) pairs into every peer's
// exchange area (plain NVLink stores), then adds the ranks' values in rank order -- the same bits on every rank.  A
// matching epoch proves the value beside it (an aligned 8-byte store is single-copy atomic).  Waits are bounded.
struct HxPfPeers { unsigned long long* p[8]; };
__global__ void __launch_bounds__(256) k_pf_tp_reduce(const float* __restrict__ part, float* __restrict__ x, HxPfPeers peers, int rank, int world,
                                                      int count, size_t area_pairs, unsigned ep, unsigned wait_limit, int* err) {
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < (size_t)count; i += (size_t)gridDim.x * blockDim.x) {
        const float v = part[i];
        const unsigned long long w64 = ((unsigned long long)ep << 32) | (unsigned long long)__float_as_uint(v);
        for (int w = 0; w < world; w++)
            if (w != rank) asm volatile("st.relaxed.sys.global.u64 [%0], %1;" :: "l"(peers.p[w] + (size_t)rank * area_pairs + i), "l"(w64) : "memory");
        float sum = 0.0f;
        for (int w = 0; w < world; w++) {
            if (w == rank) { sum += v; continue; }
            const unsigned long long* src = peers.p[rank] + (size_t)w * area_pairs + i;
            unsigned long long got = 0; bool ok = false;
            for (unsigned t = 0; t < wait_limit; t++) {
                asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(got) : "l"(src) : "memory");
                if ((unsigned)(got >> 32) == ep) { ok = true; break; }
                if ((t & 1023u) == 1023u && *reinterpret_cast<volatile int*>(err) != 0) break;
            }
            if (!ok) { *err = 1; }
            sum += __uint_as_float((unsigned)got);
        }
        x[i] += sum;
    }
}

// Tensor-parallel batched decode: one CTA per sequence takes the first maximum of this rank's vocabulary slice, the ranks
// exchange (value, global index) as pairs, and every rank keeps the best of all (greater value, or equal value and smaller
// index -- the first maximum of the whole vocabulary); the sequence's position advances by one.
__global__ void __launch_bounds__(1024) k_pf_tp_argmax_rows(const float* __restrict__ logits, int n, int ld, int vocab_off, HxPfPeers peers, int rank, int world,
                                                            size_t area_pairs, unsigned ep, unsigned wait_limit, int* err, int* __restrict__ next, int* __restrict__ pos_arr) {
    const float* lg = logits + (size_t)blockIdx.x * ld;
    float bv = -INFINITY; int bi = INT_MAX;
    for (int i = threadIdx.x; i < n; i += 1024) { const float v = lg[i]; if (v > bv || (v == bv && i < bi)) { bv = v; bi = i; } }
    __shared__ float sv[1024]; __shared__ int si[1024];
    sv[threadIdx.x] = bv; si[threadIdx.x] = bi;
    __syncthreads();
    for (int s = 512; s >= 1; s >>= 1) {
        if (threadIdx.x < s) {
            const float ov = sv[threadIdx.x + s]; const int oi = si[threadIdx.x + s];
            if (ov > sv[threadIdx.x] || (ov == sv[threadIdx.x] && oi < si[threadIdx.x])) { sv[threadIdx.x] = ov; si[threadIdx.x] = oi; }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        float fv = sv[0]; int fi = si[0] == INT_MAX ? INT_MAX : si[0] + vocab_off;
        const size_t o = 2 * (size_t)blockIdx.x;
        const unsigned long long wv = ((unsigned long long)ep << 32) | (unsigned long long)__float_as_uint(fv);
        const unsigned long long wi = ((unsigned long long)ep << 32) | (unsigned long long)(unsigned)fi;
        for (int w = 0; w < world; w++) if (w != rank) {
            asm volatile("st.relaxed.sys.global.u64 [%0], %1;" :: "l"(peers.p[w] + (size_t)rank * area_pairs + o), "l"(wv) : "memory");
            asm volatile("st.relaxed.sys.global.u64 [%0], %1;" :: "l"(peers.p[w] + (size_t)rank * area_pairs + o + 1), "l"(wi) : "memory");
        }
        for (int w = 0; w < world; w++) if (w != rank) {
            unsigned long long gv = 0, gi = 0; bool ok = false;
            const unsigned long long* src = peers.p[rank] + (size_t)w * area_pairs + o;
            for (unsigned t = 0; t < wait_limit; t++) {
                asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(gv) : "l"(src) : "memory");
                asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(gi) : "l"(src + 1) : "memory");
                if ((unsigned)(gv >> 32) == ep && (unsigned)(gi >> 32) == ep) { ok = true; break; }
                if ((t & 1023u) == 1023u && *reinterpret_cast<volatile int*>(err) != 0) break;
            }
            if (!ok) { *err = 1; continue; }
            const float ov = __uint_as_float((unsigned)gv); const int oi = (int)(unsigned)gi;
            if (ov > fv || (ov == fv && oi < fi)) { fv = ov; fi = oi; }
        }
        next[blockIdx.x] = fi == INT_MAX ? 0 : fi;
        if (pos_arr) pos_arr[blockIdx.x] += 1;
    }
}

__global__ void k_pf_advance(int* posp, int n) { hx_grid_dep_launch(); hx_grid_dep_wait(); if (threadIdx.x == 0) *posp += n; }
// First maximum of logits[row][0..n) by a cluster of eight CTAs (blockIdx.y: the row): to next[row], and with `hist` to hist[pos + 1] and
// pos + 1 to *pos_out; a row's position in pos_arr advances by one.  Bound by latency: eight loads per thread in flight.  (One CTA of 1024
// threads per row: 21 us for 151936 logits.)
#define AM_CL 8
#define AM_T 512
__device__ __forceinline__ void am_better(float& v, int& i, float ov, int oi) { if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; } }
__global__ void __cluster_dims__(AM_CL, 1, 1) __launch_bounds__(AM_T) k_pf_argmax(const float* __restrict__ logits, int n, int ld, int* __restrict__ next, int* __restrict__ pos_arr,
                                                                                   int* __restrict__ hist, int* __restrict__ pos_out, int pos) {
    __shared__ float wv[AM_T / 32], cv[AM_CL];
    __shared__ int wi[AM_T / 32], ci[AM_CL];
    const int row = blockIdx.y, tid = threadIdx.x, lane = tid & 31, rank = (int)hxtc::cl_rank();
    const float* lg = logits + (size_t)row * ld;
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");      // waited for before the first remote store
    float bv = -INFINITY; int bi = INT_MAX;
    const int step = AM_CL * AM_T;
    int i = rank * AM_T + tid;
    for (; i + 7 * step < n; i += 8 * step) {
        float v[8];
#pragma unroll
        for (int k = 0; k < 8; k++) v[k] = __ldcg(lg + i + k * step);
#pragma unroll
        for (int k = 0; k < 8; k++) am_better(bv, bi, v[k], i + k * step);
    }
    for (; i < n; i += step) am_better(bv, bi, __ldcg(lg + i), i);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) am_better(bv, bi, __shfl_xor_sync(0xffffffffu, bv, d), __shfl_xor_sync(0xffffffffu, bi, d));
    if (lane == 0) { wv[tid >> 5] = bv; wi[tid >> 5] = bi; }
    __syncthreads();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (tid == 0) {
        for (int w = 1; w < AM_T / 32; w++) am_better(bv, bi, wv[w], wi[w]);
        hxtc::cl_st(hxtc::cl_map(hxtc::s_u32(&cv[rank]), 0u), bv);
        hxtc::cl_st(hxtc::cl_map(hxtc::s_u32(&ci[rank]), 0u), __int_as_float(bi));
    }
    hxtc::cl_sync();
    if (rank == 0 && tid == 0) {
        bv = cv[0]; bi = ci[0];
        for (int r = 1; r < AM_CL; r++) am_better(bv, bi, cv[r], ci[r]);
        const int nt = bi == INT_MAX ? 0 : bi;
        next[row] = nt;
        if (pos_arr) pos_arr[row] += 1;
        if (hist) hist[pos + 1] = nt;
        if (pos_out) *pos_out = pos + 1;
    }
}

// one CTA per token row: first maximum -> next[row], and how far the runner-up lies below it -> margin[row]
// (0 when two entries tie for the maximum).  The speculative decoder trusts a row only above a margin.
__global__ void __launch_bounds__(1024) k_pf_top2_rows(const float* __restrict__ logits, int n, int ld, int* __restrict__ next, float* __restrict__ margin) {
    const float* lg = logits + (size_t)blockIdx.x * ld;
    float bv = -INFINITY, b2 = -INFINITY; int bi = INT_MAX;
    for (int i = threadIdx.x; i < n; i += 1024) {
        const float v = lg[i];
        if (v > bv || (v == bv && i < bi)) { b2 = fmaxf(b2, bv); bv = v; bi = i; }
        else b2 = fmaxf(b2, v);
    }
    __shared__ float sv[1024], s2[1024]; __shared__ int si[1024];
    sv[threadIdx.x] = bv; s2[threadIdx.x] = b2; si[threadIdx.x] = bi;
    __syncthreads();
    for (int s = 512; s >= 1; s >>= 1) {
        if (threadIdx.x < s) {
            const float ov = sv[threadIdx.x + s], o2 = s2[threadIdx.x + s]; const int oi = si[threadIdx.x + s];
            const float mv = sv[threadIdx.x], m2 = s2[threadIdx.x];
            if (ov > mv || (ov == mv && oi < si[threadIdx.x])) { sv[threadIdx.x] = ov; si[threadIdx.x] = oi; s2[threadIdx.x] = fmaxf(fmaxf(m2, o2), mv); }
            else s2[threadIdx.x] = fmaxf(fmaxf(m2, o2), ov);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) { next[blockIdx.x] = si[0] == INT_MAX ? 0 : si[0]; margin[blockIdx.x] = sv[0] - s2[0]; }
}

}  // namespace

int hx_pf_embed(const int* ids, HxPfWhere wh, const float* emb, const float* wpe, float* X, int n_tok, int DM, cudaStream_t st) {
    k_pf_embed<<<n_tok, 256, 0, st>>>(ids, wh, emb, wpe, X, DM);
    HX_CUDA(cudaGetLastError());
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}

int hx_pf_digits(const float* src, int ld, int n_tok, int K, const float* g, const float* b, float eps, uint8_t* cells, float* scale, bool early, cudaStream_t st) {
    const int group = hx_gemm_dig_group(n_tok), groups = (n_tok + group - 1) / group;
    const dim3 grid(n_tok, (K + PFD_T * 8 - 1) / (PFD_T * 8));
    const bool cl = grid.y > 1 && grid.y <= PFD_CL && !b;
    // `early`: launched while the kernel before drains.  A prompt gains (12 layers of the 8B shape: 77 tokens 1690 -> 1640 us, 128
    // 2083 -> 1990, 512 5.35 -> 5.0 .. 5.5 ms).  A batch step gains where its kernels are launched one by one (hx_decode_batch: 5 sequences 924 -> 855,
    // 12 903 -> 855, 16 926 -> 885) and loses where it is replayed from a graph (hx_decode_batch_loop: 5 724 -> 747, 12 727 -> 746, 16 757 -> 776,
    // 48 1490 -> 1536, 64 1857 -> 1911): the line at HX_PF_EARLY_SEQ is a compromise between the two.
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = dim3(PFD_T); cfg.stream = st;
    cudaLaunchAttribute at[2];
    cfg.attrs = at;
    if (early) { at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1; }
    // The long form takes over where the CTAs of k_pf_digits fill the SMs more than twice (three per SM) and every SM has a token.  Alone, back to back, slices /
    // long: 4096 columns, 300 tokens 8.3 / 8.3 us, 1008 14.4 / 12.4; 12288, 150 10.4 / 10.3, 256 14.8 / 10.4, 300 17.8 / 13.1, 512 25.3 / 16.5; 25600, 150 18.8 / 18.5,
    // 512 59.5 / 45.1.  In a prompt it gives about 4 us a launch away: its CTAs hold the values in shared memory and cannot come up beside the GEMM
    // that is leaving, those of k_pf_digits can.  Twelve layers of the 8B shape, never / from more than one wave / from two: 150 tokens 2287 / 2345 / 2287, 200 2653 / 2711 /
    // 2652, 256 3058 / 3095 / 3052, 300 3532 / 3529 / 3521, 700 7269 / 7095 / 7113, 1024 10525 / 10322 / 10135.
    const size_t values = (size_t)((K + 255) / 256) * 1024;
    if (!b && n_tok >= 148 && (long long)n_tok * grid.y > 2 * 3 * 148 && values <= 192 * 1024) {
        static HxOncePerDevice once;
        const int rc = hx_max_smem(once, k_pf_digits_long, 192 * 1024); if (rc) return rc;
        cfg.gridDim = dim3(n_tok); cfg.blockDim = dim3(PFL_T); cfg.dynamicSmemBytes = values;
        HX_CUDA(cudaLaunchKernelEx(&cfg, k_pf_digits_long, src, ld, K, g, eps, cells, group, groups, scale));
    } else if (cl) {
        at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        at[cfg.numAttrs].val.clusterDim.x = 1; at[cfg.numAttrs].val.clusterDim.y = grid.y; at[cfg.numAttrs++].val.clusterDim.z = 1;
        HX_CUDA(cudaLaunchKernelEx(&cfg, k_pf_digits<true, false>, src, ld, K, g, b, eps, cells, group, groups, scale));
    } else if (b) HX_CUDA(cudaLaunchKernelEx(&cfg, k_pf_digits<false, true>, src, ld, K, g, b, eps, cells, group, groups, scale));
    else HX_CUDA(cudaLaunchKernelEx(&cfg, k_pf_digits<false, false>, src, ld, K, g, b, eps, cells, group, groups, scale));
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}

// The threads of an attention CTA split into whole rows of the head size (P*V), and the q/k kernel has a variant per size.
bool hx_pf_head_dim(int DH) { return DH == 32 || DH == 64 || DH == 128 || DH == 256; }

int hx_pf_qkpost(float* qkv, int ld, int n_tok, HxPfWhere wh, int NH, int NKV, int DH, const float* qn_g, const float* kn_g,
                  float eps, const float* cosT, const float* sinT, float* kc, float* vc, int cap, cudaStream_t st) {
    // Four tokens per warp where that still leaves every SM several CTAs: 512 tokens of the 8B shape 14.6 -> 11.4 us.
    const int cols = (NH + 2 * NKV + PF_QK_W - 1) / PF_QK_W;
    const bool four = (long long)cols * n_tok >= 4 * 3 * 148;
    const dim3 grid(cols, four ? (n_tok + 3) / 4 : n_tok);
#define PF_QKPOST(E) HX_CUDA(hx_launch_pdl(four ? k_pf_qkpost<E, 4> : k_pf_qkpost<E, 1>, grid, dim3(PF_QK_W * 32), 0, st, qkv, ld, wh, n_tok, NH, NKV, qn_g, kn_g, eps, cosT, sinT, kc, vc, cap))
    switch (DH) {
        case 32: PF_QKPOST(1); break;
        case 64: PF_QKPOST(2); break;
        case 128: PF_QKPOST(4); break;
        case 256: PF_QKPOST(8); break;
        default: return hx_fail(HX_ERR_ARG, "chunk path: head_dim %d", DH);
    }
#undef PF_QKPOST
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}

// Runs of key tiles per (token group, kv head): as many as one wave of CTAs holds (a CTA fills an SM's shared memory; with
// two CTAs per SM asked for, five sequences took 2.2 waves of short runs: 24.5 us per layer at 900 positions against 13),
// no more than the cache has tiles.
static int pf_attn_runs(int groups, int NKV, int DH, int cap) {
    const int KT = 128 < PF_TILE_BYTES / (DH * 4) ? 128 : PF_TILE_BYTES / (DH * 4);
    int ns = 148 / (NKV * groups);
    const int cap_tiles = (cap + KT - 1) / KT;
    if (ns > cap_tiles) ns = cap_tiles;
    if (ns > PF_NS_MAX) ns = PF_NS_MAX;
    return ns < 1 ? 1 : ns;
}
// Floats of scratch for chunks of up to n_tok tokens: runs x (token group, kv head) pairs stays within 148 where there are
// several runs, and a pair has at most four tokens.
size_t hx_pf_attn_scratch(int n_tok, int NH, int NKV, int DH) {
    size_t rows = (size_t)n_tok * NKV * PF_NS_MAX;
    if (rows > 4 * 148) rows = 4 * 148;
    return rows * (NH / NKV) * (DH + 2);
}

template <int GRP, int TG>
static int pf_attn_launch(dim3 grid, size_t smem, cudaStream_t st, const float* qkv, int ld, HxPfWhere wh, int n_tok, int NH, int DH, const float* kc,
                          const float* vc, int cap, float scale, float* ctx, int ld_ctx, float* part, unsigned* tickets, int* err) {
    static HxOncePerDevice once;
    const int rc = hx_max_smem(once, k_pf_attn<GRP, TG>, 226 * 1024); if (rc) return rc;      // the kernel has some static shared memory too
    HX_CUDA(hx_launch_pdl(k_pf_attn<GRP, TG>, grid, dim3(PF_AT), smem, st, qkv, ld, wh, n_tok, NH, DH, kc, vc, cap, scale, ctx, ld_ctx, part, tickets, err));
    return HX_OK;
}

int hx_pf_attn(const float* qkv, int ld, int n_tok, HxPfWhere wh, int NH, int NKV, int DH, const float* kc, const float* vc,
               int cap, float scale, float* ctx, int ld_ctx, float* part, unsigned* tickets, int* err, cudaStream_t st) {
    const int GRP = NH / NKV;
    if (DH > 256 || DH % 32) return hx_fail(HX_ERR_ARG, "batched prefill attention: head_dim %d is not a multiple of 32 up to 256", DH);
    if (!hx_pf_head_dim(DH)) return hx_fail(HX_ERR_ARG, "batched prefill attention: head_dim %d does not divide %d", DH, PF_AT);
    if (!part || !tickets) return hx_fail(HX_ERR_ARG, "batched prefill attention: no scratch for the key runs");
    // a prefill chunk (one sequence, consecutive positions): four tokens share the tiles of a CTA
    auto smem_of = [&](int tg) { return (size_t)PF_ST * 2 * PF_TILE_BYTES + ((size_t)tg * GRP * DH + (size_t)tg * GRP * 128 + (size_t)(PF_AT / DH) * GRP * DH) * 4; };
    const size_t smem_max = 226 * 1024;
    const int TG = (wh.pos_arr || smem_of(4) > smem_max) ? 1 : 4;
    const int groups = (n_tok + TG - 1) / TG;
    const size_t smem = smem_of(TG);
    if (smem > smem_max) return hx_fail(HX_ERR_ARG, "batched prefill attention: %zu bytes of shared memory", smem);
    const int ns = pf_attn_runs(groups, NKV, DH, cap);
    dim3 grid(NKV, groups, ns);
    int rc;
#define HX_PF_ATTN(G) case G: rc = TG == 1 ? pf_attn_launch<G, 1>(grid, smem, st, qkv, ld, wh, n_tok, NH, DH, kc, vc, cap, scale, ctx, ld_ctx, part, tickets, err) \
                                            : pf_attn_launch<G, 4>(grid, smem, st, qkv, ld, wh, n_tok, NH, DH, kc, vc, cap, scale, ctx, ld_ctx, part, tickets, err); break;
    switch (GRP) {
        HX_PF_ATTN(1) HX_PF_ATTN(2) HX_PF_ATTN(3) HX_PF_ATTN(4) HX_PF_ATTN(5) HX_PF_ATTN(6) HX_PF_ATTN(7) HX_PF_ATTN(8)
        default: return hx_fail(HX_ERR_ARG, "batched prefill attention: group of %d query heads per kv head not supported", GRP);
    }
#undef HX_PF_ATTN
    if (rc) return rc;
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}

void hx_pf_tp_reduce(const float* part, float* x, unsigned long long* const* peer_areas, int rank, int world, int count, size_t area_pairs,
                     unsigned ep, unsigned wait_limit, int* err, cudaStream_t st) {
    HxPfPeers pe = {};
    for (int w = 0; w < world && w < 8; w++) pe.p[w] = peer_areas[w];
    int g = (count + 255) / 256; if (g > 148 * 4) g = 148 * 4;
    k_pf_tp_reduce<<<g, 256, 0, st>>>(part, x, pe, rank, world, count, area_pairs, ep, wait_limit, err);
    HX_COUNT_LAUNCH(1);
}

void hx_pf_tp_argmax_rows(const float* logits, int n, int ld, int rows, int vocab_off, unsigned long long* const* peer_areas, int rank, int world,
                          size_t area_pairs, unsigned ep, unsigned wait_limit, int* err, int* next, int* pos_arr, cudaStream_t st) {
    HxPfPeers pe = {};
    for (int w = 0; w < world && w < 8; w++) pe.p[w] = peer_areas[w];
    k_pf_tp_argmax_rows<<<rows, 1024, 0, st>>>(logits, n, ld, vocab_off, pe, rank, world, area_pairs, ep, wait_limit, err, next, pos_arr);
    HX_COUNT_LAUNCH(1);
}

int hx_pf_advance(int* posp, int n, cudaStream_t st) {
    HX_CUDA(hx_launch_pdl(k_pf_advance, dim3(1), dim3(32), 0, st, posp, n));
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}

void hx_pf_argmax(const float* logits, int n, int* tok, int* hist, int* pos_out, int pos, cudaStream_t st) {
    k_pf_argmax<<<dim3(AM_CL, 1), AM_T, 0, st>>>(logits, n, 0, tok, nullptr, hist, pos_out, pos);
    HX_COUNT_LAUNCH(1);
}

void hx_pf_top2_rows(const float* logits, int n, int ld, int rows, int* next, float* margin, cudaStream_t st) {
    k_pf_top2_rows<<<rows, 1024, 0, st>>>(logits, n, ld, next, margin);
    HX_COUNT_LAUNCH(1);
}

void hx_pf_argmax_rows(const float* logits, int n, int ld, int rows, int* next, int* pos_arr, cudaStream_t st) {
    k_pf_argmax<<<dim3(AM_CL, rows), AM_T, 0, st>>>(logits, n, ld, next, pos_arr, nullptr, nullptr, 0);
    HX_COUNT_LAUNCH(1);
}
