// hx_gemm_dig.cu -- the GEMM of the chunk paths (batched prefill, batched decode, the verify forward): packed NVFP4 weights
// times f32 activations that enter the FP4 tensor cores as digit columns (hx_prefill.cu: k_pf_digits).  Replaces the f32
// tiled_matmul_abt projections of forward_layer_llama, helixc/runtime/gpt2_infer.c:1231-1287.
//
//   out[t][row] (+)= scale_t * ts(row) * 13^7 * sum_d 13^-d ( sum_k W[row,k] * SF[row,k/16] * CS[t,block of k] * digit_d[t,k] )
//
// A unit of work is a 128-row tile of W times a group of G <= 26 tokens: 8 G digit columns, tcgen05.mma kind::mxf4nvf4 with
// M = 128, N = 8 G, K = 64, N / 2 cycles each at large N (the pipe's rate, which neither the scale copies nor loads, TMEM reads and
// polling warps beside it lower).  What bounds a large chunk (512 tokens, 8B shape): the pipe is busy for 46 (o) to 66 % (gate+up) of a launch.  A unit of sixteen
// MMAs takes 1664 cycles of it and 2270 in all, because a 18 KB weight cell is some 1900 cycles on its way round -- freed, asked for,
// brought from L2 (385 cycles of the SM's port each), used -- and the ring holds five; then ramp, drain and the passage
// between blocks of K.  What bounds a small one (a group or two): the weights from HBM and the fixed part of a launch.
//
// K is cut over the CTAs of a cluster, not over time: CTA q of C keeps the digit cells of its part of K (28 KB each at 26 tokens,
// as many as fit: four, or sixteen for six tokens) in shared memory and streams only weight cells (18 KB per four MMAs).  Two
// accumulators lie in TMEM, each with an issuing warp of its own, so a unit's MMAs run while the unit before is read out: a thread folds
// a row's eight digit accumulators of two tokens at a time (f32x2), the small ones first (v = D7; v = D6 + v / 13; ...: every step's
// rounding but the last is divided by the steps after it), into a staging block per CTA of the cluster; a sender warp copies the
// other CTAs' blocks to them (cp.async.bulk between shared memories, counted at the receiver's barrier); eight warps add the C
// parts of the tokens that the CTA owns, its own first and then the others in K order, and apply the epilogue.  The partial sums never leave the SMs, no
// tickets are drawn, and the result does not depend on timing.
//
// Digits, GEMM and epilogue of the four linears of a layer of the 8B shape, launch by launch, before / now (ten base-9 digits, 24 tokens a group, one issuing
// warp, sums sent by plain stores and a cluster-scope release that held the read-out up for 1500 cycles a unit): 5 tokens 80 / 74 us,
// 64 119 / 109, 77 137 / 113, 512 447 / 370, 1008 795 / 690.  Error against 64 bits (relative, 2-norm over
// the rows; K = 768 .. 12288; ten base-9 digits / now): 6e-8 .. 9e-8 / 5e-8 .. 8e-8 for N(0, 1), heavy-tailed vectors and those with an element 64 to a
// million times the others.  Rows whose weight on the large element is zero, which see the resolution of the elements beside it: 64 times
// 1.0e-7 .. 1.3e-7 / 7e-8 .. 9e-8, 1000 times 1.1e-6 .. 1.3e-6 / 2.6e-7 .. 9.6e-7, one in every 256 elements 64 times 1.3e-7 .. 1.5e-7 / 1.4e-7 ..
// 1.6e-7 (K = 256, one element 1000 times: 1.0e-6 / 1.5e-6).
//
// K beyond the resident cells is done in blocks, one pass over the tiles each; the sums so far wait in global memory between
// the passes (the same thread writes and reads them).  Every wait is bounded; the roles meet only at mbarriers.
#include "hx_tc.cuh"
#include "hx_gemm_tc.cuh"
#include <mutex>

using namespace hxtc;

namespace {

constexpr int DG_STAGES = 6;                 // ring of weight cells: at most, four at least
constexpr int DG_EPI = 8;                    // read-out warps: two per quarter of the TMEM lanes, half of the token pairs each
constexpr int DG_FIN = 8;                    // finishing warps: two threads per row of the tile, half of the CTA's tokens each
constexpr int DG_W_EPI = 3, DG_W_FIN = DG_W_EPI + DG_EPI;      // warp 0 loads weights, 1 issues MMAs, 2 loads digit cells
constexpr int DG_W_SEND = DG_W_FIN + DG_FIN;                   // sends sums to the other CTAs of the cluster
constexpr int DG_W_MMA2 = DG_W_SEND + 1;                       // (with warp 1)
constexpr int DG_THREADS = (DG_W_MMA2 + 1) * 32;
constexpr int DG_TOK = HX_TC_MAX_TOK, DG_RES = HX_TC_RES_CELLS;
constexpr int DG_EP = (DG_TOK / 2 + 1) / 2;      // token pairs of a read-out warp at most
constexpr float DG_13P7 = 62748516.0f;       // 13^7 - 1: fmaf(v, DG_13P7, v) is v * 13^7, rounded once
static_assert(HX_TC_DIGITS == 8, "a token is eight columns");

// Token pairs that a CTA of the cluster finishes, and their sums in one unit: [pair][128 rows][2 tokens].
__host__ __device__ constexpr int dg_pairs(int group, int C) { return (group / 2 + C - 1) / C; }
__host__ __device__ constexpr int dg_blk(int group, int C) { return dg_pairs(group, C) * 1024; }
// Digit cells that fit beside a ring of four, the staged sums (a block per CTA) and a received block per other CTA.
__host__ __device__ constexpr int dg_sum_bytes(int group, int C) { return (2 * C - 1) * dg_blk(group, C); }
// Token pairs per finishing thread for `shares` threads per row; a thread reads as many as a full group has, so the last block is
// followed by as many pairs as it may read too far.
__host__ __device__ constexpr int dg_share(int group, int C, int shares) { return (dg_pairs(group, C) + shares - 1) / shares; }
constexpr int dg_over(int group, int C) {
    const int p = dg_pairs(group, C), a = dg_share(group, C, 2) + dg_share(DG_TOK, C, 2) - p, b = 3 * dg_share(group, C, 4) + dg_share(DG_TOK, C, 4) - p;
    return (a > b ? a : b) * 1024;
}
constexpr int DG_HDR = 2048, DG_SMEM = 227 * 1024;
constexpr int dg_room(int group, int C) { return DG_SMEM - 1024 - DG_HDR - dg_sum_bytes(group, C) - dg_over(group, C); }
constexpr int dg_res_cells(int group, int C) {
    const int n = (dg_room(group, C) - 4 * HX_T128_CELL) / HX_TC_DCELL(group);
    return n < DG_RES ? n : DG_RES;
}
static_assert(16 * DG_TOK + 2 * 16 + 2 * 16 <= 512, "two accumulators, row scales and column scales of either issuing warp in TMEM");
static_assert(dg_res_cells(DG_TOK, 1) >= 4 && dg_res_cells(DG_TOK, 2) >= 4 && dg_res_cells(DG_TOK, 4) >= 4, "four cells of a full group");
// What the digit cells leave goes to the ring: loads in flight are what the MMAs wait for.
constexpr int dg_stages(int group, int C, int res) { const int n = (dg_room(group, C) - res * HX_TC_DCELL(group)) / HX_T128_CELL; return n < DG_STAGES ? n : DG_STAGES; }
static_assert(dg_stages(DG_TOK, 2, 4) >= 5, "five cells beside a full group of a pair");

struct DgSmem {
    // ring of weight cells: a pair of barriers per slot for each MMA warp.  (One for both would pass two uses on between two looks of a
    // warp, and a parity tells a use from the next one only.)
    uint64_t full[2][DG_STAGES], empty[2][DG_STAGES], bfull[DG_RES], bempty[DG_RES];
    uint64_t accum[2], acc_free[2], st_full, st_free, rx_full, rx_free, given_up[2];
    uint32_t tmem_base;
    volatile uint32_t zero;                  // see the hand-back of the finishing warps
    volatile int abort_flag;
};
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
    uint8_t* ring = base + DG_HDR;
    const uint32_t stages = (uint32_t)g.stages;
    uint8_t* bres = ring + stages * HX_T128_CELL;                 // digit cells of this CTA's part of K
    const int G = g.group, P = G / 2, ppc = dg_pairs(G, C), tpc = 2 * ppc;      // tokens and pairs of a group; those that a CTA of the cluster finishes
    const uint32_t dcell = HX_TC_DCELL(G);
    const int blk = dg_blk(G, C);
    uint8_t* stage = bres + (size_t)g.res * dcell;                                // [C destination CTAs] blocks
    uint8_t* rx = stage + C * blk;                                                // [C - 1 source CTAs] blocks
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int q = (int)cl_rank(), NP = g.nblk * C;
    const int ncl = gridDim.x / C, cl = blockIdx.x / C;
    const int units = g.ntiles * g.groups;
    const int u0 = (int)((long long)units * cl / ncl), u1 = (int)((long long)units * (cl + 1) / ncl);

    // The next kernel may start; this one has its barriers, tensor memory and first weight cells (which no kernel writes) ready
    // before it waits for the one before: the digit loader and the finishing warps do.
    hx_grid_dep_launch();
    if (tid == 0) {
        for (int i = 0; i < 2 * DG_STAGES; i++) { mb_init(&S.full[0][i], 1); mb_init(&S.empty[0][i], 1); }
        for (int i = 0; i < DG_RES; i++) { mb_init(&S.bfull[i], 1); mb_init(&S.bempty[i], 2); }
        for (int i = 0; i < 2; i++) { mb_init(&S.accum[i], 1); mb_init(&S.acc_free[i], DG_EPI); }
        mb_init(&S.rx_full, 1); mb_init(&S.rx_free, C > 1 ? DG_FIN * (C - 1) : 1);
        mb_init(&S.st_full, DG_EPI); mb_init(&S.st_free, DG_FIN + (C > 1 ? 1 : 0));
        mb_init(&S.given_up[0], 1); mb_init(&S.given_up[1], 1);
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
    const uint32_t ncols = 8u * (uint32_t)G, col_sfa = 2u * ncols, col_sfb = col_sfa + 32u;
    volatile int* ab_flag = &S.abort_flag;

    if (warp == 0) {
        // ------------------------------ weight loader ------------------------------
        if (lane == 0) {
            // Four bits per slot: parity of the next use by either warp's units, which warp's unit used it last, used before.  (Kept
            // short: at 430 cycles a cell, with the divisions of a unit among them, this thread held the MMAs up.)
            static_assert(DG_STAGES <= 8, "four bits per slot");
            const uint32_t bar0 = s_u32(&S.full[0][0]), ring0 = s_u32(ring);
            uint32_t slot = 0, state = 0, w = 0;
            bool ok = true;
            for (int u = u0; u < u1 && ok; ) {
                const int t0 = u % g.ntiles, nt = min(g.ntiles - t0, u1 - u);
                for (int kb = 0; kb < g.nblk && ok; kb++) {
                    const int p = kb * C + q, c_lo = p * g.kcells / NP, nc = (p + 1) * g.kcells / NP - c_lo;
                    const uint8_t* src = g.a + ((size_t)t0 * g.kcells + c_lo) * HX_T128_CELL;
                    const size_t step = (size_t)(g.kcells - nc) * HX_T128_CELL;
                    for (int t = 0; t < nt && ok; t++, src += step, w ^= 1u)
                        for (int c = 0; c < nc; c++, src += HX_T128_CELL) {
                            const uint32_t st = state >> (4u * slot), l = (st >> 2) & 1u;
                            if ((st & 8u) && !mb_wait(&S.empty[l][slot], ((st >> l) & 1u) ^ 1u, ab_flag)) { ok = false; break; }
                            const uint32_t bar = bar0 + (w * DG_STAGES + slot) * 8u;
                            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(HX_T128_CELL) : "memory");
                            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                         :: "r"(ring0 + slot * HX_T128_CELL), "l"(src), "r"(HX_T128_CELL), "r"(bar) : "memory");
                            state = (state & ~(4u << (4u * slot))) ^ ((1u << w) << (4u * slot));
                            state |= (8u | (w << 2)) << (4u * slot);
                            if (++slot == stages) slot = 0;
                        }
                }
                u += nt;
            }
            if (!ok)       // given up: the CTA must not end with a copy of its own in flight
                for (int i = 0; i < (int)stages; i++) {
                    const uint32_t st = state >> (4 * i), l = (st >> 2) & 1u;
                    if (st & 8u) mb_drain(&S.full[l][i], ((st >> l) & 1u) ^ 1u);
                }
        }
    } else if (warp == 2) {
        // ------------------------------ digit-cell loader ------------------------------
        hx_grid_dep_wait();
        if (lane == 0) {
            uint32_t used = 0, par = 0;          // a bit per resident cell: filled before; parity of its last fill
            bool ok = true;
            dg_walk(g, u0, u1, [&](int grp, int, int kb, bool fresh, bool) {
                if (!fresh) return true;
                const int p = kb * C + q, c_lo = p * g.kcells / NP, nc = (p + 1) * g.kcells / NP - c_lo;
                for (int i = 0; i < nc; i++) {
                    const uint32_t bit = 1u << i;
                    if ((used & bit) && !mb_wait(&S.bempty[i], (par & bit) ? 1u : 0u, ab_flag)) { ok = false; return false; }
                    mb_expect(&S.bfull[i], dcell);
                    bulk_load(bres + (size_t)i * dcell, g.b + ((size_t)(c_lo + i) * g.groups + grp) * dcell, dcell, &S.bfull[i]);
                    if (used & bit) par ^= bit;
                    used |= bit;
                }
                return true;
            });
            if (!ok)
                for (int i = 0; i < DG_RES; i++)
                    if (used >> i & 1u) mb_drain(&S.bfull[i], (par >> i) & 1u);
        }
    } else if (warp == 1 || warp == DG_W_MMA2) {
        // ------------------------------ MMA issuers ------------------------------
        // Two warps, one per accumulator: what lies between two units in a warp (waits, the walk, the issue of the first instructions:
        // about 1100 cycles) is more than the one or two MMAs that the pipe holds, so the other warp's unit fills it.  Each warp copies
        // the column scales of a cell before its MMAs, as it does the row scales, so neither depends on what the other has copied.  (Copied once
        // per pass over the tiles by the warp of its first unit, with a barrier that the other one waited at: 1 to 2 % slower, and that warp could take
        // the barrier of the pass before for this one's.)
        // instruction descriptor: E2M1 x E2M1, UE4M3 scales, K-major both, M = 128, N = 8 G, K = 64
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)G << 17) | (8u << 24);
        const int mw = warp == 1 ? 0 : 1;
        const uint64_t dA0 = smem_desc(s_u32(ring), 16, 1024, SW128), dS0 = smem_desc(s_u32(ring) + 16384, 16, 128);
        const uint64_t dB0 = smem_desc(s_u32(bres), 16, 1024, SW128);
        const uint64_t dC0 = smem_desc(s_u32(bres) + (uint32_t)G * 1024u, 16, 128);      // column scales of a digit cell: MMA steps 0 and 1, 2 and 3
        const uint32_t acc = tmem + (uint32_t)mw * ncols, sfa = tmem + col_sfa + (uint32_t)mw * 16u, sfb = tmem + col_sfb + (uint32_t)mw * 16u;
        const bool wide = ncols > 128u;
        const uint32_t dsf = (uint32_t)HX_TC_DSF(G) >> 4;
        uint32_t slot = 0, fpar = 0, bpar = 0;             // (fpar, bpar: a parity per slot and digit cell)
        int ou = 0;
        bool ok = true;
        for (int u = u0; u < u1 && ok; ) {
            const int t0 = u % g.ntiles, nt = min(g.ntiles - t0, u1 - u);
            for (int kb = 0; kb < g.nblk && ok; kb++) {
                const int p = kb * C + q, nc = (p + 1) * g.kcells / NP - p * g.kcells / NP;
                const int first = (ou ^ mw) & 1;                     // this warp's first unit of the pass
                for (int ci = 0; ci < nc && ok && first > 0; ci++) ok = warp_wait(&S.bfull[ci], (bpar >> ci) & 1u, ab_flag);
                if (first >= nt && ok && lane == 0)                  // none: the cells are not used here
                    for (int ci = 0; ci < nc; ci++) mb_arrive(&S.bempty[ci]);
                for (int t = 0; t < nt && ok; t++, ou++) {
                    if ((ou & 1) != mw) { slot = (slot + (uint32_t)nc) % stages; continue; }
                    const bool done = t + 2 >= nt;
                    if (ou >= 2 && !warp_wait(&S.acc_free[mw], (uint32_t)((ou >> 1) - 1) & 1u, ab_flag)) { ok = false; break; }     // its previous unit has been read out
                    for (int ci = 0; ci < nc; ci++) {
                        if (t == 0 && !warp_wait(&S.bfull[ci], (bpar >> ci) & 1u, ab_flag)) { ok = false; break; }
                        if (!warp_wait(&S.full[mw][slot], (fpar >> slot) & 1u, ab_flag)) { ok = false; break; }
                        fpar ^= 1u << slot;
                        tc_fence_after();
                        // the descriptors of a cell's four steps differ by constants (the address field counts 16-byte units)
                        const uint64_t dA = dA0 + (uint64_t)(slot * (HX_T128_CELL >> 4)), dS = dS0 + (uint64_t)(slot * (HX_T128_CELL >> 4));
                        const uint64_t dB = dB0 + (uint64_t)((uint32_t)ci * (dcell >> 4)), dC = dC0 + (uint64_t)((uint32_t)ci * (dcell >> 4));
                        if (tc_elect()) {
                            tc_cp_sf(sfb, dC);
                            tc_cp_sf(sfb + 8, dC + dsf);
                            if (wide) { tc_cp_sf(sfb + 4, dC + 32u); tc_cp_sf(sfb + 12, dC + dsf + 32u); }
#pragma unroll
                            for (int k = 0; k < 4; k++) tc_cp_sf(sfa + k * 4, dS + (uint64_t)(k * 32));
#pragma unroll
                            for (int k = 0; k < 4; k++)
                                tc_mma(acc, dA + (uint64_t)(k * 2), dB + (uint64_t)(k * 2), idesc, sfa + k * 4, sfb + (k >> 1) * 8, (k > 0 || ci > 0) ? 1u : 0u);
                            tc_commit(&S.empty[mw][slot]);
                            if (done) tc_commit(&S.bempty[ci]);
                            if (ci + 1 == nc) tc_commit(&S.accum[mw]);
                        }
                        __syncwarp();
                        if (++slot == stages) slot = 0;
                    }
                }
                bpar ^= (1u << nc) - 1u;
            }
            u += nt;
        }
        if (!ok) {       // given up: the tensor memory and the cells must outlive the MMAs that were issued
            if (tc_elect()) tc_commit(&S.given_up[mw]);
            __syncwarp();
            mb_drain(&S.given_up[mw], 0);
        }
    } else if (warp < DG_W_FIN) {
        // ------------------------------ read-out: TMEM -> fold -> the token's CTA ------------------------------
        const int part = (warp - DG_W_EPI) >> 2, sub = warp & 3;              // TMEM lanes 32 sub .. 32 sub + 31
        const int ep = (P + 1) / 2, p0 = part * ep, mine = min(ep, P - p0);   // this warp's token pairs of a group: p0 .. p0 + mine - 1
        uint8_t* const to = stage + (sub * 32 + lane) * 8;
        const f32x2 c13 = x2(1.0f / 13.0f, 1.0f / 13.0f);
        const uint32_t tcol = tmem + ((uint32_t)(sub * 32) << 16) + (uint32_t)(p0 * 16);
        int ou = 0;
        dg_walk(g, u0, u1, [&](int grp, int, int, bool, bool) {
            const int buf = ou & 1;
            const int np = min(mine, (g.ntok - grp * G + 1) / 2 - p0);        // pairs of this warp that exist
            if (!warp_wait(&S.accum[buf], (uint32_t)(ou >> 1) & 1u, ab_flag)) return false;
            tc_fence_after();
            const uint32_t col = tcol + (uint32_t)buf * ncols;
            f32x2 v[DG_EP];
#pragma unroll
            for (int h = 0; h < DG_EP; h += 3) {
                if (h > 0 && h >= np) break;
                uint32_t r[3][16];
#pragma unroll
                for (int t = 0; t < 3; t++) if (h + t < DG_EP) tc_ld16(r[t], col + (uint32_t)((h + t) * 16));      // (columns past the group's are TMEM all the same)
                tc_wait_ld();
                if (h + 3 >= DG_EP || h + 3 >= np) {      // all of it is in registers
                    tc_fence_before();
                    if (lane == 0) mb_arrive(&S.acc_free[buf]);
                }
#pragma unroll
                for (int t = 0; t < 3; t++) {
                    if (h + t >= DG_EP) break;
                    v[h + t] = x2(r[t][14], r[t][15]);
#pragma unroll
                    for (int d = 6; d >= 0; d--) v[h + t] = x2_fma(v[h + t], c13, x2(r[t][2 * d], r[t][2 * d + 1]));
                }
            }
            // The staging is free a trip to the other CTAs and back after the unit before was sent: the accumulator is not held up by that.
            if (ou >= 1 && !warp_wait(&S.st_free, (uint32_t)(ou - 1) & 1u, ab_flag)) return false;
#pragma unroll
            for (int t = 0; t < DG_EP; t++) if (t < np) *reinterpret_cast<f32x2*>(to + (p0 + t) * 1024) = v[t];
            if (C > 1) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mb_arrive(&S.st_full);
            ou++;
            return true;
        });
    } else if (warp == DG_W_SEND) {
        // ------------------------------ sums of the other CTAs' tokens on their way ------------------------------
        // A block per CTA by one bulk copy between shared memories, which counts its bytes at the receiver's barrier: nobody waits
        // for stores to arrive.  (st.async of single words counts a transaction per lane
        // and was unusable.)
        // Nothing at the source says when such a copy has read its block (bulk groups hold only copies that complete by group), so the
        // staging is given back when every other CTA has taken its sums of the unit: rx_free of unit u follows the reads of what the
        // copies wrote, these follow rx_full there, which counts the copies' bytes.  No circle: a CTA takes unit u as soon as its own
        // read-out and the copies of unit u are done, and both wait only for units before.
        if (C > 1) {
            const uint32_t to = lane < C ? cl_map(s_u32(rx) + (uint32_t)((q < lane ? q : q - 1) * blk), (uint32_t)lane) : 0u;
            const uint32_t bar = lane < C ? cl_map(s_u32(&S.rx_full), (uint32_t)lane) : 0u;
            int ou = 0, announced = 0;
            bool ok = true;
            dg_walk(g, u0, u1, [&](int, int, int, bool, bool) {
                ok = warp_wait(&S.st_full, (uint32_t)ou & 1u, ab_flag) &&
                     (ou == 0 || warp_wait(&S.rx_full, (uint32_t)(ou - 1) & 1u, ab_flag));                  // the unit before has arrived here: announce this one
                if (!ok) return false;
                if (lane == 0) mb_expect(&S.rx_full, (uint32_t)((C - 1) * blk));
                announced = ou + 1;
                if (lane < C && lane != q) cl_bulk(to, s_u32(stage + lane * blk), (uint32_t)blk, bar);      // (the unit before has been taken there)
                if (!(ok = warp_wait(&S.rx_free, (uint32_t)ou & 1u, ab_flag))) return false;
                if (lane == 0) mb_arrive(&S.st_free);
                ou++;
                return true;
            });
            // Given up: no CTA may end with copies to or from it in flight.  A CTA waits for those to it, the cluster leaves together.
            // What can still come is the unit announced last and, as the others cannot finish one without this CTA's part, one more.
            if (!ok && lane == 0) {
                const bool came = !announced || mb_drain(&S.rx_full, (uint32_t)(announced - 1) & 1u);
                if (came && announced < (u1 - u0) * g.nblk) {
                    mb_expect(&S.rx_full, (uint32_t)((C - 1) * blk));
                    mb_drain(&S.rx_full, (uint32_t)announced & 1u);
                }
            }
        }
    } else {
        // ------------------------------ finish: add the K parts, scale, store ------------------------------
        // What a unit needs from memory (residual values, sums of the K blocks so far) is fetched one unit ahead, and the
        // buffer is given back as soon as its sums are in registers: nothing here waits for a round trip to L2.  Plain
        // linears: thread (row, half of the tokens).  SwiGLU: thread (hidden element, quarter of the tokens) adds the gate row
        // and the up row.  K in blocks: the sums so far wait in `part` (the output itself when nothing else lies there); the
        // thread that wrote them reads them back.
        const int ft = tid - DG_W_FIN * 32;
        hx_grid_dep_wait();
        // The hand-back: the other CTAs write into the buffer once it arrives, so the warp's reads have to be over.  The arrival
        // goes to an address that is picked by a vote over the values read (both candidates are the same, which the compiler cannot
        // know: a zero from shared memory lies between them), so it cannot be issued before every lane's loads have returned.  (A
        // release at cluster scope waits for the thread's global stores as well, about a microsecond.)
        const uint32_t free_bar = cl_map(s_u32(&S.rx_free), (uint32_t)(lane % C)), same_bar = free_bar + S.zero;
        auto hand_back = [&](float read) {
            const uint32_t bar = __any_sync(0xffffffffu, read == 1.0f) ? free_bar : same_bar;
            if (lane < C && lane != q) cl_arrive_relaxed(bar);
        };
        // This CTA's own part of a unit's sums is taken first, so that the read-out can go on; the other parts are added to it in K
        // order.  Instructions are what a unit can run out of (its MMAs take 1664 cycles): tokens go in pairs, addresses are constants
        // or steps of a pointer, a thread reads NP pairs whether it has as many or not, and the common case loads and stores without
        // predicates.  (Token by token, with a comparison per token and part: 4000 cycles a unit.)
        const f32x2 c13p7 = x2(DG_13P7, DG_13P7);
        DgStep it = {u0, u1, 0, 0, 0, 0, 0};
        bool more = it.begin(g);
        int cs_grp = -1;
        if (!g.swiglu) {
            constexpr int NP = dg_share(DG_TOK, C, 2), TB = 2 * NP;
            const int sh = dg_share(G, C, 2), r = ft & 127, pr0 = (ft >> 7) * sh, j0 = 2 * pr0, nb = 2 * min(sh, min(ppc, P - q * ppc) - pr0);
            const uint8_t* const mine = stage + q * blk + pr0 * 1024 + r * 8;
            const uint8_t* const theirs = rx + pr0 * 1024 + r * 8;
            const size_t ld = (size_t)g.ld_out;
            float prev[TB], sofar[TB];
            f32x2 cs[NP];
            auto tokens = [&](const DgStep& s) { return s.tile * 128 + r < g.rows ? min(nb, g.ntok - (s.grp * G + q * tpc + j0)) : 0; };
            auto offset = [&](const DgStep& s) { return (size_t)(s.grp * G + q * tpc + j0) * ld + s.tile * 128 + r; };
            float* const part = g.resid ? g.acc : g.out;
            auto load = [&](float (&to)[TB], const float* p, int nt) {
                if (nt == TB) {
#pragma unroll
                    for (int j = 0; j < TB; j++, p += ld) to[j] = __ldcg(p);
                } else {
#pragma unroll
                    for (int j = 0; j < TB; j++, p += ld) to[j] = j < nt ? __ldcg(p) : 0.0f;
                }
            };
            auto fetch = [&](const DgStep& s) {
                if (g.resid && s.kb + 1 == g.nblk) load(prev, g.out + offset(s), tokens(s));
                if (s.kb > 0) load(sofar, part + offset(s), tokens(s));
            };
            if (more) fetch(it);
            for (int ou = 0; more; ou++) {
                const DgStep cur = it;
                const int row = cur.tile * 128 + r, nt = tokens(cur);
                const bool lastb = cur.kb + 1 == g.nblk, firstb = cur.kb == 0;
                if (cur.grp != cs_grp) {
                    cs_grp = cur.grp;
#pragma unroll
                    for (int j = 0; j < NP; j++) {
                        const int tk = cur.grp * G + q * tpc + j0 + 2 * j;
                        cs[j] = x2(tk < g.ntok ? __ldcg(g.col_scale + tk) : 0.0f, tk + 1 < g.ntok ? __ldcg(g.col_scale + tk + 1) : 0.0f);
                    }
                }
                f32x2 v[NP];
                if (!warp_wait(&S.st_full, (uint32_t)ou & 1u, ab_flag)) break;
#pragma unroll
                for (int j = 0; j < NP; j++) v[j] = *reinterpret_cast<const f32x2*>(mine + j * 1024);
                __syncwarp();
                if (lane == 0) mb_arrive(&S.st_free);
                if (C > 1 && !warp_wait(&S.rx_full, (uint32_t)ou & 1u, ab_flag)) break;
                if (C > 1) {
#pragma unroll
                    for (int p = 0; p < C - 1; p++) {
                        const uint8_t* src = theirs + p * blk;
#pragma unroll
                        for (int j = 0; j < NP; j++) v[j] = x2_add(v[j], *reinterpret_cast<const f32x2*>(src + j * 1024));
                    }
                    f32x2 got = v[0];
#pragma unroll
                    for (int j = 1; j < NP; j++) got = x2_add(got, v[j]);
                    hand_back(x2_lo(got));
                }
                const float tsr = g.pair64 ? (r < 64 ? g.ts[0] : g.ts[1]) : (row < g.bound0 ? g.ts[0] : (row < g.bound1 ? g.ts[1] : g.ts[2]));
                const f32x2 ts2 = x2(tsr, tsr);
                float y[TB];
#pragma unroll
                for (int j = 0; j < NP; j++) {
                    const f32x2 w = x2_mul(x2_fma(v[j], c13p7, v[j]), x2_mul(cs[j], ts2));
                    y[2 * j] = x2_lo(w); y[2 * j + 1] = x2_hi(w);
                }
                if (!firstb)
#pragma unroll
                    for (int j = 0; j < TB; j++) y[j] += sofar[j];
                if (lastb) {
                    if (g.bias) {
                        const float bias = row < g.rows ? __ldg(g.bias + row) : 0.0f;
#pragma unroll
                        for (int j = 0; j < TB; j++) y[j] += bias;
                    }
                    if (g.gelu)
#pragma unroll
                        for (int j = 0; j < TB; j++) y[j] = dg_gelu(y[j]);
                    if (g.resid)
#pragma unroll
                        for (int j = 0; j < TB; j++) y[j] += prev[j];
                }
                float* dst = (lastb ? g.out : part) + offset(cur);
                more = it.next(g);
                const bool same = cur.t1 - cur.t0 == 1;      // the next unit reads what this one is about to write
                if (more && !same) fetch(it);
                if (nt == TB) {
#pragma unroll
                    for (int j = 0; j < TB; j++, dst += ld) __stcg(dst, y[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < TB; j++, dst += ld) if (j < nt) __stcg(dst, y[j]);
                }
                if (more && same) fetch(it);
            }
        } else {
            constexpr int NP = dg_share(DG_TOK, C, 4), TB = 2 * NP;
            const int sh = dg_share(G, C, 4), rr = ft & 63, pr0 = (ft >> 6) * sh, j0 = 2 * pr0, nb = 2 * min(sh, min(ppc, P - q * ppc) - pr0);
            const uint8_t* const mine = stage + q * blk + pr0 * 1024 + rr * 8;
            const uint8_t* const theirs = rx + pr0 * 1024 + rr * 8;
            const size_t ldp = (size_t)g.ntiles * 128, ld = (size_t)g.ld_out;
            float sg[TB], su[TB];
            f32x2 cs[NP];
            auto tokens = [&](const DgStep& s) { return s.tile * 64 + rr < g.rows ? min(nb, g.ntok - (s.grp * G + q * tpc + j0)) : 0; };
            auto sums = [&](const DgStep& s) { return g.acc + (size_t)(s.grp * G + q * tpc + j0) * ldp + s.tile * 128 + rr; };
            auto fetch = [&](const DgStep& s) {
                if (s.kb == 0) return;
                const float* p = sums(s);
                const int nt = tokens(s);
                if (nt == TB) {
#pragma unroll
                    for (int j = 0; j < TB; j++, p += ldp) { sg[j] = __ldcg(p); su[j] = __ldcg(p + 64); }
                } else {
#pragma unroll
                    for (int j = 0; j < TB; j++, p += ldp) { sg[j] = j < nt ? __ldcg(p) : 0.0f; su[j] = j < nt ? __ldcg(p + 64) : 0.0f; }
                }
            };
            const f32x2 tsg = x2(g.ts[0], g.ts[0]), tsu = x2(g.ts[1], g.ts[1]);
            if (more) fetch(it);
            for (int ou = 0; more; ou++) {
                const DgStep cur = it;
                const int nt = tokens(cur);
                const bool lastb = cur.kb + 1 == g.nblk, firstb = cur.kb == 0;
                if (cur.grp != cs_grp) {
                    cs_grp = cur.grp;
#pragma unroll
                    for (int j = 0; j < NP; j++) {
                        const int tk = cur.grp * G + q * tpc + j0 + 2 * j;
                        cs[j] = x2(tk < g.ntok ? __ldcg(g.col_scale + tk) : 0.0f, tk + 1 < g.ntok ? __ldcg(g.col_scale + tk + 1) : 0.0f);
                    }
                }
                f32x2 vg[NP], vu[NP];
                if (!warp_wait(&S.st_full, (uint32_t)ou & 1u, ab_flag)) break;
#pragma unroll
                for (int j = 0; j < NP; j++) { vg[j] = *reinterpret_cast<const f32x2*>(mine + j * 1024); vu[j] = *reinterpret_cast<const f32x2*>(mine + j * 1024 + 512); }
                __syncwarp();
                if (lane == 0) mb_arrive(&S.st_free);
                if (C > 1 && !warp_wait(&S.rx_full, (uint32_t)ou & 1u, ab_flag)) break;
                if (C > 1) {
#pragma unroll
                    for (int p = 0; p < C - 1; p++) {
                        const uint8_t* src = theirs + p * blk;
#pragma unroll
                        for (int j = 0; j < NP; j++) {
                            vg[j] = x2_add(vg[j], *reinterpret_cast<const f32x2*>(src + j * 1024));
                            vu[j] = x2_add(vu[j], *reinterpret_cast<const f32x2*>(src + j * 1024 + 512));
                        }
                    }
                    f32x2 got = x2_add(vg[0], vu[0]);
#pragma unroll
                    for (int j = 1; j < NP; j++) got = x2_add(got, x2_add(vg[j], vu[j]));
                    hand_back(x2_lo(got));
                }
                float yg[TB], yu[TB];
#pragma unroll
                for (int j = 0; j < NP; j++) {
                    const f32x2 a = x2_mul(x2_fma(vg[j], c13p7, vg[j]), x2_mul(cs[j], tsg)), b = x2_mul(x2_fma(vu[j], c13p7, vu[j]), x2_mul(cs[j], tsu));
                    yg[2 * j] = x2_lo(a); yg[2 * j + 1] = x2_hi(a); yu[2 * j] = x2_lo(b); yu[2 * j + 1] = x2_hi(b);
                }
                if (!firstb)
#pragma unroll
                    for (int j = 0; j < TB; j++) { yg[j] += sg[j]; yu[j] += su[j]; }
                more = it.next(g);
                const bool same = cur.t1 - cur.t0 == 1;
                if (more && !same) fetch(it);
                if (!lastb) {
                    float* p = sums(cur);
                    if (nt == TB) {
#pragma unroll
                        for (int j = 0; j < TB; j++, p += ldp) { __stcg(p, yg[j]); __stcg(p + 64, yu[j]); }
                    } else {
#pragma unroll
                        for (int j = 0; j < TB; j++, p += ldp) if (j < nt) { __stcg(p, yg[j]); __stcg(p + 64, yu[j]); }
                    }
                } else {
                    float* p = g.out + (size_t)(cur.grp * G + q * tpc + j0) * ld + cur.tile * 64 + rr;
#pragma unroll
                    for (int j = 0; j < TB; j++) {
                        const float sgn = yg[j] < 0.0f ? -1.0f : 1.0f;
                        const float ex = __expf(-(sgn * yg[j]));
                        const float th = sgn * ((1.0f - ex) / (1.0f + ex));
                        yg[j] = yg[j] * (0.5f * (1.0f + th)) * yu[j];
                    }
#pragma unroll
                    for (int j = 0; j < TB; j++, p += ld) if (j < nt) __stcg(p, yg[j]);
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

typedef void (*DgKernel)(HxGemmDig);
DgKernel dg_kernel(int C) { return C == 1 ? k_gemm_dig<1> : C == 2 ? k_gemm_dig<2> : k_gemm_dig<4>; }

void dg_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, int ncl, int C, cudaStream_t st) {
    cfg = {};
    cfg.gridDim = dim3(ncl * C); cfg.blockDim = dim3(DG_THREADS); cfg.dynamicSmemBytes = DG_SMEM; cfg.stream = st;
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
        HX_CUDA(cudaFuncSetAttribute(dg_kernel(C), cudaFuncAttributeMaxDynamicSharedMemorySize, DG_SMEM));
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

int dg_blocks(int kcells, int C, int res) { return (kcells + C * res - 1) / (C * res); }

}  // namespace

int hx_gemm_dig_prepare() {
    for (int C = 1; C <= 4; C *= 2) { int n; const int rc = dg_clusters(C, &n); if (rc) return rc; }
    return HX_OK;
}

// How a launch is cut up.  CTAs per cluster: two or four, whichever leaves the busiest CTA less to do: its weight cells, 1.3 cells' time
// per unit (the gap between two units' MMAs) and eight per block of K (digit cells refilled, sums through memory).  Large launches
// take pairs (all SMs fit into pairs, 132 of 148 into fours); small ones cut K finer because their tiles do not divide evenly.  A
// smaller cluster wins a tie.  (Layer of the 8B shape, counting cells alone / with units and blocks: 24 tokens 58.9 / 58.1 us, 48 81.8 / 77.7, 64
// 95.2 / 93.7, 128 125.7 / 124.8, 512 345 / 344; fours for everything 365 at 512.)
struct DgPlan { int C, ncl, nblk, group, groups; };
static int dg_plan(int ntiles, int kcells, int ntok, DgPlan& p) {
    p = {};
    p.group = hx_gemm_dig_group(ntok);
    p.groups = (ntok + p.group - 1) / p.group;
    const int units = ntiles * p.groups;
    long best = 0;
    for (int c = kcells > 1 ? 2 : 1; c <= 4 && c <= kcells; c *= 2) {
        int n = 0;
        const int rc = dg_clusters(c, &n); if (rc) return rc;
        const int nb = dg_blocks(kcells, c, dg_res_cells(p.group, c)), per = (units + n - 1) / n;
        if (nb * c > kcells) continue;
        const long cost = (long)per * nb * (10 * ((kcells + nb * c - 1) / (nb * c)) + 13) + 80 * nb;
        if (!p.C || cost < best) { p.C = c; p.ncl = n < units ? n : units; p.nblk = nb; best = cost; }
    }
    return HX_OK;
}

int hx_gemm_dig_launch(HxGemmDig g, cudaStream_t st) {
    HX_CHECK_ARG(g.a && g.out && g.ntiles > 0 && g.kcells > 0 && g.ntok > 0 && g.b && g.col_scale);
    DgPlan p;
    const int rc = dg_plan(g.ntiles, g.kcells, g.ntok, p); if (rc) return rc;
    g.group = p.group; g.groups = p.groups; g.nblk = p.nblk; g.res = (g.kcells + p.nblk * p.C - 1) / (p.nblk * p.C);
    g.stages = dg_stages(p.group, p.C, g.res);
    HX_CHECK_ARG((!g.resid && !g.swiglu) || g.nblk == 1 || g.acc);
    cudaLaunchConfig_t cfg; cudaLaunchAttribute at[2];
    dg_config(cfg, at, p.ncl, p.C, st);
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    HX_CUDA(cudaLaunchKernelEx(&cfg, dg_kernel(p.C), g));
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}
