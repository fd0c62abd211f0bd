// hx_gemm_dig.cu -- the GEMM of the chunk paths (batched prefill, batched decode, the verify forward): packed NVFP4 weights
// times f32 activations that enter the FP4 tensor cores as digit columns (hx_prefill.cu: k_pf_digits).  Replaces the f32
// tiled_matmul_abt projections of forward_layer_llama, helixc/runtime/gpt2_infer.c:1231-1287.
//
//   out[t][row] (+)= scale_t * ts(row) * sum_d 9^(9-d) * ( sum_k W[row,k] * SF[row,k/16] * digit_d[t,k] )
//
// A unit of work is a 128-row tile of W times a group of 24 tokens: 240 digit columns, tcgen05.mma kind::mxf4nvf4 with
// M = 128, N = 240, K = 64, 120 cycles each (the pipe's rate; the scale-factor copies of a weight cell hide behind it).
// What bounds a large chunk: the MMA's operands (98 bytes per cycle) and the weights that arrive (38) ask more than the 128 that
// shared memory moves, so the pipe is busy for about 155 cycles per MMA, and for a third of a launch (512 tokens, 8B shape) it
// waits for ramps, read-outs and the passage between blocks of K.  What bounds a small one (a group or two) is the weights
// from HBM and the fixed part of a launch.
//
// K is cut over the CTAs of a cluster, not over time: CTA q of C keeps the digit cells of its part of K (at most four
// 256-column cells, 120 KB) in shared memory and streams only weight cells (18 KB per four MMAs = 38 bytes per cycle and
// SM from L2, which delivers 65).  Two accumulators of 240 columns fill TMEM, so a unit's MMAs run while the unit before
// is read out: each thread folds a row's ten digit accumulators per token by Horner's rule and sends the sums through
// distributed shared memory to the CTA of the cluster that owns the token (24 / C tokens each); eight warps there add the
// C parts in K order and apply the epilogue.  So the partial sums never leave the SMs, no tickets are drawn, and the result
// does not depend on timing.  (Before: every K piece stored its sums to global memory and the last piece to finish, found
// by a ticket, read them back; the read-out warps did that work between two units and held the MMAs up.)
//
// K beyond four cells per CTA is done in blocks, one pass over the tiles each; the sums so far wait in global memory between
// the passes (the same thread writes and reads them).  Every wait is bounded; the roles meet only at mbarriers.
#include "hx_tc.cuh"
#include "hx_gemm_tc.cuh"
#include <mutex>

using namespace hxtc;

namespace {

constexpr int DG_STAGES = 4;                 // ring of weight cells
constexpr int DG_EPI = 12;                   // read-out warps: three per quarter of the TMEM lanes, eight tokens each
constexpr int DG_FIN = 8;                    // finishing warps: two threads per row of the tile, half of the CTA's tokens each
constexpr int DG_W_EPI = 3, DG_W_FIN = DG_W_EPI + DG_EPI;      // warp 0 loads weights, 1 issues MMAs, 2 loads digit cells
constexpr int DG_THREADS = (DG_W_FIN + DG_FIN) * 32;
constexpr int DG_TOK = HX_TC_MAX_TOK, DG_COLS = HX_TC_GROUP_COLS;
constexpr uint32_t DG_BCELL = DG_COLS * 128;      // digit cell of a group: 240 rows of 128 bytes
static_assert(DG_EPI * 8 == 4 * DG_TOK, "a read-out warp takes eight tokens of a quarter of the rows");
static_assert(2 * DG_COLS + 32 <= 512, "two accumulators and the scale factors fill TMEM");

struct DgSmem {
    uint64_t full[DG_STAGES], empty[DG_STAGES], bfull[HX_TC_RES_CELLS], bempty[HX_TC_RES_CELLS];
    uint64_t accum[2], acc_free[2], rx_full[2], rx_free[2];
    uint32_t tmem_base;
    volatile uint32_t zero;                  // see the hand-back of the finishing warps
    volatile int abort_flag;
};
constexpr uint32_t DG_HDR = 1024;            // header, then 512 bytes of unit scales
static_assert(sizeof(DgSmem) <= DG_HDR, "header");

// The units [u0, u1) of a cluster in order: group by group, and within a group one pass over its tiles per block of K.
// f(group, tile, K block, first tile of the pass, last tile of the pass) -> go on?
template <class F>
__device__ __forceinline__ void dg_walk(const HxGemmDig& g, int u0, int u1, F&& f) {
    while (u0 < u1) {
        const int grp = u0 / g.ntiles, t0 = u0 - grp * g.ntiles, t1 = min(g.ntiles, t0 + u1 - u0);
        for (int kb = 0; kb < g.nblk; kb++)
            for (int t = t0; t < t1; t++) if (!f(grp, t, kb, t == t0, t + 1 == t1)) return;
        u0 += t1 - t0;
    }
}

// The same walk, one step at a time.
struct DgStep {
    int u, u1, grp, tile, kb, t0, t1;
    __device__ __forceinline__ bool begin(const HxGemmDig& g) {      // at unit u: the pass over the group's tiles that starts here
        if (u >= u1) return false;
        grp = u / g.ntiles; t0 = tile = u - grp * g.ntiles; t1 = min(g.ntiles, t0 + u1 - u); kb = 0;
        return true;
    }
    __device__ __forceinline__ bool next(const HxGemmDig& g) {
        if (++tile < t1) return true;
        tile = t0;
        if (++kb < g.nblk) return true;
        u += t1 - t0;
        return begin(g);
    }
};

__device__ __forceinline__ float dg_gelu(float x) {      // gpu_gelu_stable_kernel.hx:15-28
    const float inner = 0.7978846f * (x + (0.044715f * (x * x * x))), two = 2.0f * inner;
    const float sgn = inner < 0.0f ? -1.0f : 1.0f;
    const float e = __expf(-(sgn * two));
    const float th = sgn * ((1.0f - e) / (1.0f + e));
    return 0.5f * x * (1.0f + th);
}

template <int C>
__global__ void __launch_bounds__(DG_THREADS, 1) k_gemm_dig(const __grid_constant__ HxGemmDig g) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    // swizzled operands need 1024-byte aligned cells (the swizzle is a function of the shared-memory address); the offset is
    // the same in every CTA of the cluster
    uint8_t* base = smem_raw + (((s_u32(smem_raw) + 1023u) & ~1023u) - s_u32(smem_raw));
    DgSmem& S = *reinterpret_cast<DgSmem*>(base);
    uint8_t* ones = base + DG_HDR;                                   // a chunk of unit scales
    uint8_t* ring = base + 2048;
    uint8_t* bres = ring + DG_STAGES * HX_T128_CELL;                 // digit cells of this CTA's part of K
    float* rx = reinterpret_cast<float*>(bres + HX_TC_RES_CELLS * DG_BCELL);      // [2][C source CTAs][tpc tokens][128 rows]
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    constexpr int tpc = DG_TOK / C;                                  // tokens that a CTA of the cluster finishes
    const int q = (int)cl_rank(), NP = g.nblk * C;
    const int ncl = gridDim.x / C, cl = blockIdx.x / C;
    const int units = g.ntiles * g.groups;
    const int u0 = (int)((long long)units * cl / ncl), u1 = (int)((long long)units * (cl + 1) / ncl);

    // The next kernel may start; this one has its barriers, tensor memory and first weight cells (which no kernel writes) ready
    // before it waits for the one before: the digit loader and the finishing warps do.
    hx_grid_dep_launch();
    if (tid < 128) reinterpret_cast<uint32_t*>(ones)[tid] = 0x38383838u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (tid == 0) {
        for (int i = 0; i < DG_STAGES; i++) { mb_init(&S.full[i], 1); mb_init(&S.empty[i], 1); }
        for (int i = 0; i < HX_TC_RES_CELLS; i++) { mb_init(&S.bfull[i], 1); mb_init(&S.bempty[i], 1); }
        for (int i = 0; i < 2; i++) { mb_init(&S.accum[i], 1); mb_init(&S.acc_free[i], DG_EPI); mb_init(&S.rx_full[i], DG_EPI * C); mb_init(&S.rx_free[i], DG_FIN * C); }
        S.abort_flag = 0; S.zero = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(s_u32(&S.tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    cl_sync();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    const uint32_t col_sfa = 2u * DG_COLS, col_sfb = 2u * DG_COLS + 16u;
    volatile int* ab_flag = &S.abort_flag;

    if (warp == 0) {
        // ------------------------------ weight loader ------------------------------
        if (lane == 0) {
            uint32_t slot = 0, round = 0;
            bool ok = true;
            dg_walk(g, u0, u1, [&](int, int t, int kb, bool, bool) {
                const int p = kb * C + q, c_lo = p * g.kcells / NP, c_hi = (p + 1) * g.kcells / NP;
                const uint8_t* src = g.a + ((size_t)t * g.kcells + c_lo) * HX_T128_CELL;
                for (int c = c_lo; c < c_hi; c++, src += HX_T128_CELL) {
                    if (round > 0 && !mb_wait(&S.empty[slot], (round - 1) & 1, ab_flag)) { ok = false; return false; }
                    mb_expect(&S.full[slot], HX_T128_CELL);
                    bulk_load(ring + slot * HX_T128_CELL, src, HX_T128_CELL, &S.full[slot]);
                    if (++slot == DG_STAGES) { slot = 0; round++; }
                }
                return true;
            });
            if (!ok)       // given up: the CTA must not end with a copy of its own in flight
                for (int i = 0; i < DG_STAGES; i++) {
                    const uint32_t uses = round + ((uint32_t)i < slot ? 1u : 0u);
                    if (uses > 0) mb_drain(&S.full[i], (uses - 1) & 1);
                }
        }
    } else if (warp == 2) {
        // ------------------------------ digit-cell loader ------------------------------
        hx_grid_dep_wait();
        if (lane == 0) {
            uint32_t uses[HX_TC_RES_CELLS] = {0, 0, 0, 0};
            bool ok = true;
            dg_walk(g, u0, u1, [&](int grp, int, int kb, bool fresh, bool) {
                if (!fresh) return true;
                const int p = kb * C + q, c_lo = p * g.kcells / NP, nc = (p + 1) * g.kcells / NP - c_lo;
#pragma unroll
                for (int i = 0; i < HX_TC_RES_CELLS; i++) {
                    if (i >= nc) break;
                    if (uses[i] > 0 && !mb_wait(&S.bempty[i], (uses[i] - 1) & 1, ab_flag)) { ok = false; return false; }
                    mb_expect(&S.bfull[i], DG_BCELL);
                    bulk_load(bres + i * DG_BCELL, g.b + ((size_t)(c_lo + i) * g.groups + grp) * DG_BCELL, DG_BCELL, &S.bfull[i]);
                    uses[i]++;
                }
                return true;
            });
            if (!ok)
#pragma unroll
                for (int i = 0; i < HX_TC_RES_CELLS; i++)
                    if (uses[i] > 0) mb_drain(&S.bfull[i], (uses[i] - 1) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        // instruction descriptor: E2M1 x E2M1, UE4M3 scales, K-major both, M = 128, N = 240, K = 64
        constexpr uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(DG_COLS >> 3) << 17) | (8u << 24);
        const uint64_t dA0 = smem_desc(s_u32(ring), 16, 1024, SW128), dS0 = smem_desc(s_u32(ring) + 16384, 16, 128);
        const uint64_t dB0 = smem_desc(s_u32(bres), 16, 1024, SW128);
        if (tc_elect()) for (int c = 0; c < 4; c++) tc_cp_sf(tmem + col_sfb + c * 4, smem_desc(s_u32(ones), 16, 128));
        __syncwarp();
        uint32_t slot = 0, par = 0, bpar = 0;
        int ou = 0;
        dg_walk(g, u0, u1, [&](int, int, int kb, bool fresh, bool done) {
            const int p = kb * C + q, nc = (p + 1) * g.kcells / NP - p * g.kcells / NP;
            const uint32_t acc = tmem + (uint32_t)(ou & 1) * DG_COLS;
            if (ou >= 2) {      // the accumulator's previous unit has been read out
                if (!warp_wait(&S.acc_free[ou & 1], (uint32_t)((ou >> 1) - 1) & 1u, ab_flag)) return false;
                tc_fence_after();
            }
            for (int ci = 0; ci < nc; ci++) {
                if (fresh) {
                    if (!warp_wait(&S.bfull[ci], (bpar >> ci) & 1u, ab_flag)) return false;
                    bpar ^= 1u << ci;
                }
                if (!warp_wait(&S.full[slot], par, ab_flag)) return false;
                tc_fence_after();
                // the descriptors of a cell's four steps differ by constants (the address field counts 16-byte units)
                const uint64_t dA = dA0 + (uint64_t)(slot * (HX_T128_CELL >> 4)), dS = dS0 + (uint64_t)(slot * (HX_T128_CELL >> 4));
                const uint64_t dB = dB0 + (uint64_t)((uint32_t)ci * (DG_BCELL >> 4));
                if (tc_elect()) {
#pragma unroll
                    for (int k = 0; k < 4; k++) tc_cp_sf(tmem + col_sfa + k * 4, dS + (uint64_t)(k * 32));
#pragma unroll
                    for (int k = 0; k < 4; k++)
                        tc_mma(acc, dA + (uint64_t)(k * 2), dB + (uint64_t)(k * 2), idesc, tmem + col_sfa + k * 4, tmem + col_sfb, (k > 0 || ci > 0) ? 1u : 0u);
                    tc_commit(&S.empty[slot]);
                    if (done) tc_commit(&S.bempty[ci]);
                    if (ci + 1 == nc) tc_commit(&S.accum[ou & 1]);
                }
                __syncwarp();
                if (++slot == DG_STAGES) { slot = 0; par ^= 1u; }
            }
            ou++;
            return true;
        });
    } else if (warp < DG_W_FIN) {
        // ------------------------------ read-out: TMEM -> fold -> the token's CTA ------------------------------
        const int ew = warp - DG_W_EPI, third = ew >> 2, sub = warp & 3;      // TMEM lanes 32 sub .. 32 sub + 31, tokens 8 third .. 8 third + 7
        const int row = sub * 32 + lane;
        uint32_t dst[8];                                                      // where token t's sum of this row goes
#pragma unroll
        for (int t = 0; t < 8; t++) {
            const int tok = third * 8 + t, d = tok / tpc;
            dst[t] = cl_map(s_u32(rx + ((size_t)q * tpc + (tok - d * tpc)) * 128 + row), (uint32_t)d);
        }
        const uint32_t full_bar = lane < C ? cl_map(s_u32(&S.rx_full[0]), (uint32_t)lane) : 0u;
        const uint32_t rx_stride = (uint32_t)(C * tpc * 128 * 4);
        int ou = 0;
        dg_walk(g, u0, u1, [&](int grp, int, int, bool, bool) {
            const int buf = ou & 1;
            const bool any = third * 8 < g.ntok - grp * DG_TOK;               // tokens of this warp exist
            if (!warp_wait(&S.accum[buf], (uint32_t)(ou >> 1) & 1u, ab_flag)) return false;
            tc_fence_after();
            float val[8];
#pragma unroll
            for (int t = 0; t < 8; t++) val[t] = 0.0f;
            if (any) {
                const uint32_t tcol = tmem + ((uint32_t)(sub * 32) << 16) + (uint32_t)(buf * DG_COLS + third * 8);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    uint32_t r[5][8];
#pragma unroll
                    for (int d = 0; d < 5; d++) tc_ld8(r[d], tcol + (uint32_t)((h * 5 + d) * DG_TOK));
                    tc_wait_ld();
#pragma unroll
                    for (int d = 0; d < 5; d++)
#pragma unroll
                        for (int t = 0; t < 8; t++) val[t] = fmaf(val[t], 9.0f, __uint_as_float(r[d][t]));
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive(&S.acc_free[buf]);
            if (ou >= 2 && !__all_sync(0xffffffffu, mb_wait_cl(&S.rx_free[buf], (uint32_t)((ou >> 1) - 1) & 1u, ab_flag))) return false;
            if (any) {
#pragma unroll
                for (int t = 0; t < 8; t++) cl_st(dst[t] + (uint32_t)buf * rx_stride, val[t]);
            }
            __syncwarp();
            if (lane < C) cl_arrive(full_bar + (uint32_t)buf * 8u);
            ou++;
            return true;
        });
    } else {
        // ------------------------------ finish: add the K parts, scale, store ------------------------------
        // What a unit needs from memory (residual values, sums of the K blocks so far) is fetched one unit ahead, and the
        // buffer is given back as soon as its sums are in registers: nothing here waits for a round trip to L2.  Plain
        // linears: thread (row, half of the tokens).  SwiGLU: thread (hidden element, quarter of the tokens) adds the gate row
        // and the up row.  K in blocks: the sums so far wait in `part` (the output itself when nothing else lies there); the
        // thread that wrote them reads them back.
        const int ft = tid - DG_W_FIN * 32;
        hx_grid_dep_wait();
        // The hand-back: the other CTAs store into the buffer once it arrives, so the warp's reads have to be over.  The arrival
        // goes to an address that is picked by a vote over the values read (both candidates are the same, which the compiler cannot
        // know: a zero from shared memory lies between them), so it cannot be issued before every lane's loads have returned.  (A release at cluster scope waits for the
        // thread's global stores as well: 1 us per unit, 445 us against 381 for a layer of the 8B shape at 512 tokens; by a warp
        // of its own behind a local barrier, 1 % of a prompt.)
        const uint32_t free_bar = cl_map(s_u32(&S.rx_free[0]), (uint32_t)(lane % C)), same_bar = free_bar + S.zero;
        auto hand_back = [&](float read, int buf) {
            const uint32_t bar = __any_sync(0xffffffffu, read == 1.0f) ? free_bar : same_bar;
            if (lane < C) cl_arrive_relaxed(bar + (uint32_t)buf * 8u);
        };
        DgStep it = {u0, u1, 0, 0, 0, 0, 0};
        bool more = it.begin(g);
        int cs_grp = -1;
        if (!g.swiglu) {
            constexpr int TB = (tpc + 1) / 2;
            const int r = ft & 127, j0 = (ft >> 7) * TB;
            float prev[TB], sofar[TB], cs[TB];
            auto tokens = [&](const DgStep& s) { return s.tile * 128 + r < g.rows ? min(min(TB, tpc - j0), g.ntok - (s.grp * DG_TOK + q * tpc + j0)) : 0; };
            auto offset = [&](const DgStep& s) { return (size_t)(s.grp * DG_TOK + q * tpc + j0) * g.ld_out + s.tile * 128 + r; };
            float* const part = g.resid ? g.acc : g.out;
            auto fetch = [&](const DgStep& s) {
                const int nt = tokens(s);
                const size_t off = offset(s);
#pragma unroll
                for (int j = 0; j < TB; j++) {
                    prev[j] = (g.resid && s.kb + 1 == g.nblk && j < nt) ? __ldcg(g.out + off + (size_t)j * g.ld_out) : 0.0f;
                    sofar[j] = (s.kb > 0 && j < nt) ? __ldcg(part + off + (size_t)j * g.ld_out) : 0.0f;
                }
            };
            if (more) fetch(it);
            for (int ou = 0; more; ou++) {
                const DgStep cur = it;
                const int buf = ou & 1, row = cur.tile * 128 + r, nt = tokens(cur);
                const bool lastb = cur.kb + 1 == g.nblk, firstb = cur.kb == 0;
                if (cur.grp != cs_grp) {
                    cs_grp = cur.grp;
#pragma unroll
                    for (int j = 0; j < TB; j++) { const int tk = cur.grp * DG_TOK + q * tpc + j0 + j; cs[j] = tk < g.ntok ? __ldcg(g.col_scale + tk) : 0.0f; }
                }
                if (!__all_sync(0xffffffffu, mb_wait_cl(&S.rx_full[buf], (uint32_t)(ou >> 1) & 1u, ab_flag))) break;
                const float* src = rx + ((size_t)buf * C * tpc + j0) * 128 + r;
                float v[TB];
#pragma unroll
                for (int j = 0; j < TB; j++) v[j] = 0.0f;
#pragma unroll
                for (int p = 0; p < C; p++)
#pragma unroll
                    for (int j = 0; j < TB; j++) v[j] += (j0 + j < tpc) ? src[(p * tpc + j) * 128] : 0.0f;
                float all = 0.0f;
#pragma unroll
                for (int j = 0; j < TB; j++) all += v[j];
                hand_back(all, buf);
                const float bias = (g.bias && lastb && row < g.rows) ? __ldg(g.bias + row) : 0.0f;
                const float tsr = g.pair64 ? (r < 64 ? g.ts[0] : g.ts[1]) : (row < g.bound0 ? g.ts[0] : (row < g.bound1 ? g.ts[1] : g.ts[2]));
                float* dst = (lastb ? g.out : part) + offset(cur);
#pragma unroll
                for (int j = 0; j < TB; j++) {
                    float y = v[j] * cs[j] * tsr;
                    if (!firstb) y += sofar[j];
                    if (lastb) { y += bias; if (g.gelu) y = dg_gelu(y); }
                    v[j] = (g.resid && lastb) ? prev[j] + y : y;
                }
                more = it.next(g);
                const bool same = cur.t1 - cur.t0 == 1;      // the next unit reads what this one is about to write
                if (more && !same) fetch(it);
#pragma unroll
                for (int j = 0; j < TB; j++) if (j < nt) __stcg(dst + (size_t)j * g.ld_out, v[j]);
                if (more && same) fetch(it);
            }
        } else {
            constexpr int TB = (tpc + 3) / 4;
            const int rr = ft & 63, j0 = (ft >> 6) * TB;
            const int ldp = g.ntiles * 128;
            float sg[TB], su[TB], cs[TB];
            auto fetch = [&](const DgStep& s) {
                const int tok0 = s.grp * DG_TOK + q * tpc + j0, nt = min(min(TB, tpc - j0), g.ntok - tok0);
                const float* part = g.acc + (size_t)tok0 * ldp + s.tile * 128 + rr;
#pragma unroll
                for (int j = 0; j < TB; j++) {
                    sg[j] = (s.kb > 0 && j < nt) ? __ldcg(part + (size_t)j * ldp) : 0.0f;
                    su[j] = (s.kb > 0 && j < nt) ? __ldcg(part + (size_t)j * ldp + 64) : 0.0f;
                }
            };
            if (more) fetch(it);
            for (int ou = 0; more; ou++) {
                const DgStep cur = it;
                const int buf = ou & 1, h = cur.tile * 64 + rr;
                const int tok0 = cur.grp * DG_TOK + q * tpc + j0, nt = min(min(TB, tpc - j0), g.ntok - tok0);
                const bool lastb = cur.kb + 1 == g.nblk, firstb = cur.kb == 0;
                if (cur.grp != cs_grp) {
                    cs_grp = cur.grp;
#pragma unroll
                    for (int j = 0; j < TB; j++) cs[j] = j < nt ? __ldcg(g.col_scale + tok0 + j) : 0.0f;
                }
                if (!__all_sync(0xffffffffu, mb_wait_cl(&S.rx_full[buf], (uint32_t)(ou >> 1) & 1u, ab_flag))) break;
                const float* src = rx + ((size_t)buf * C * tpc + j0) * 128 + rr;
                float vg[TB], vu[TB];
#pragma unroll
                for (int j = 0; j < TB; j++) vg[j] = vu[j] = 0.0f;
#pragma unroll
                for (int p = 0; p < C; p++)
#pragma unroll
                    for (int j = 0; j < TB; j++) if (j0 + j < tpc) { vg[j] += src[(p * tpc + j) * 128]; vu[j] += src[(p * tpc + j) * 128 + 64]; }
                float all = 0.0f;
#pragma unroll
                for (int j = 0; j < TB; j++) all += vg[j] + vu[j];
                hand_back(all, buf);
#pragma unroll
                for (int j = 0; j < TB; j++) {
                    vg[j] *= cs[j] * g.ts[0]; vu[j] *= cs[j] * g.ts[1];
                    if (!firstb) { vg[j] += sg[j]; vu[j] += su[j]; }
                }
                more = it.next(g);
                const bool same = cur.t1 - cur.t0 == 1;
                if (more && !same) fetch(it);
                if (!lastb) {
                    float* part = g.acc + (size_t)tok0 * ldp + cur.tile * 128 + rr;
#pragma unroll
                    for (int j = 0; j < TB; j++) if (j < nt) { __stcg(part + (size_t)j * ldp, vg[j]); __stcg(part + (size_t)j * ldp + 64, vu[j]); }
                } else {
#pragma unroll
                    for (int j = 0; j < TB; j++) if (j < nt) {
                        const float sgn = vg[j] < 0.0f ? -1.0f : 1.0f;
                        const float ex = __expf(-(sgn * vg[j]));
                        const float th = sgn * ((1.0f - ex) / (1.0f + ex));
                        if (h < g.rows) __stcg(g.out + (size_t)(tok0 + j) * g.ld_out + h, vg[j] * (0.5f * (1.0f + th)) * vu[j]);
                    }
                }
                if (more && same) fetch(it);
            }
        }
    }
    __syncthreads();
    if (S.abort_flag && tid == 0 && g.err) *g.err = 1;
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
    }
    cl_sync();      // nobody leaves while a CTA of the cluster may still write into its shared memory
}

size_t dg_smem() { return 1024 + 2048 + (size_t)DG_STAGES * HX_T128_CELL + (size_t)HX_TC_RES_CELLS * DG_BCELL + (size_t)2 * DG_TOK * 128 * 4; }

typedef void (*DgKernel)(HxGemmDig);
DgKernel dg_kernel(int C) { return C == 1 ? k_gemm_dig<1> : C == 2 ? k_gemm_dig<2> : k_gemm_dig<4>; }

void dg_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int ncl, int C, cudaStream_t st) {
    cfg = {};
    cfg.gridDim = dim3(ncl * C); cfg.blockDim = dim3(DG_THREADS); cfg.dynamicSmemBytes = dg_smem(); cfg.stream = st;
    at[0].id = cudaLaunchAttributeClusterDimension; at[0].val.clusterDim.x = C; at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
}

// Clusters of C CTAs that are resident together on the current device; asked once per device and size, together with the
// kernel's attribute.
int dg_clusters(int C, int* out) {
    static std::mutex mu;
    static int cached[64][5];
    int dev = 0;
    HX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return hx_fail(HX_ERR_ARG, "device index %d not supported", dev);
    std::lock_guard<std::mutex> lk(mu);
    if (!cached[dev][C]) {
        HX_CUDA(cudaFuncSetAttribute(dg_kernel(C), cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
        cudaLaunchConfig_t cfg; cudaLaunchAttribute at[1];
        dg_config(cfg, at, 64, C, nullptr);
        int n = 0;
        HX_CUDA(cudaOccupancyMaxActiveClusters(&n, dg_kernel(C), &cfg));
        if (n < 1) return hx_fail(HX_ERR_CUDA, "chunk GEMM: no cluster of %d CTAs fits the device", C);
        cached[dev][C] = n;
    }
    *out = cached[dev][C];
    return HX_OK;
}

int dg_blocks(int kcells, int C) { return (kcells + C * HX_TC_RES_CELLS - 1) / (C * HX_TC_RES_CELLS); }

}  // namespace

int hx_gemm_dig_prepare() {
    for (int C = 1; C <= 4; C *= 2) { int n; const int rc = dg_clusters(C, &n); if (rc) return rc; }
    return HX_OK;
}

int hx_gemm_dig_launch(HxGemmDig g, cudaStream_t st) {
    HX_CHECK_ARG(g.a && g.b && g.out && g.col_scale && g.ntiles > 0 && g.kcells > 0 && g.ntok > 0);
    g.groups = (g.ntok + DG_TOK - 1) / DG_TOK;
    // CTAs per cluster: two or four, whichever leaves fewer weight cells to the busiest CTA.  Large launches take pairs (all
    // SMs fit into pairs, 132 of 148 into fours); small ones cut K finer because their tiles do not divide evenly.  A
    // smaller cluster wins a tie: it finishes with fewer messages.  (Layer of the 8B shape, pairs / fours / eights: 58 / 50 /
    // 65 us at 24 tokens, 90 / 85 / 122 at 64, 381 / 387 / 678 at 512.)
    const int units = g.ntiles * g.groups;
    int C = 0, ncl = 0, nblk = 0; long best = 0;
    for (int c = g.kcells > 1 ? 2 : 1; c <= 4 && c <= g.kcells; c *= 2) {
        int n = 0;
        const int rc = dg_clusters(c, &n); if (rc) return rc;
        const int nb = dg_blocks(g.kcells, c), per = (units + n - 1) / n;
        if (nb * c > g.kcells) continue;
        const long cost = (long)per * nb * ((g.kcells + nb * c - 1) / (nb * c));
        if (!C || cost < best) { C = c; ncl = n < units ? n : units; nblk = nb; best = cost; }
    }
    g.nblk = nblk;
    HX_CHECK_ARG((!g.resid && !g.swiglu) || g.nblk == 1 || g.acc);
    cudaLaunchConfig_t cfg; cudaLaunchAttribute at[2];
    dg_config(cfg, at, ncl, C, st);
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    HX_CUDA(cudaLaunchKernelEx(&cfg, dg_kernel(C), g));
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}
