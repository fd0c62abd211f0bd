// hx_decode_df.cu -- the persistent decode-step kernel without grid barriers ("dataflow" engine).
//
// One cooperative CTA per SM runs the whole token as a list of phases (per layer qkv | attention | o_proj |
// gate+up | down, then lm_head + arg-max), the weights streaming through a shared-memory ring of T128 cells
// into tcgen05.mma kind::mxf4nvf4 exactly as in hx_persist_tc.cu (digit-sliced activations, TMEM
// accumulators, a producer thread that runs ahead of the consumers).  What differs is how the CTAs hand
// results to one another.  There is no grid-wide barrier: every vector that crosses CTAs (residual stream,
// q, the position's k and v, attention partials, the SwiGLU hidden vector, split-K partial sums, per-tile
// sums of squares) is stored as 8-byte (value, epoch) pairs with one 64-bit store per element, and the
// reader polls the data itself until the epoch of the producing phase shows up.  An 8-byte store is
// single-copy atomic, so a matching epoch proves the value beside it; no fence, flag or ticket travels
// separately, and a hand-over costs one store-to-load latency instead of release + barrier + load.
//
//  * A linear phase cuts its cells over the CTAs like hx_persist_tc.cu (tc_plan).  The CTA that holds
//    piece 0 of a tile is its merger: the other pieces store their partial rows as pairs, the merger polls
//    them, adds them in piece order (results do not depend on timing) and runs the epilogue.
//  * RMSNorm needs the sum of squares of the whole input: the residual epilogue that produces a tile of x
//    also publishes that tile's sum of squares, and every CTA of the consuming phase adds the per-tile
//    sums in tile order.  Polling them also keeps the CTAs in step: nobody enters a norm phase before all
//    tiles of the previous residual phase are final, which is what makes the reuse of the pair buffers
//    one layer later safe.  The digit scale is taken over the CTA's own K slice.
//  * Tensor parallel: the merger of a row-split linear stores its partial rows as pairs into every
//    rank's exchange buffer (plain NVLink stores, 8-byte atomic) and adds the ranks' rows in rank order,
//    so the all-reduce is one more hand-over of the same kind.
//
// Every wait is bounded (HxPersist::wait_limit polls).  A wait that runs out latches an abort flag; code
// between two phase boundaries never changes its barrier pattern because of it (waits return at once,
// the arithmetic runs on whatever is there) and the phase boundary decides with a barrier-wide OR, so all
// threads leave together through the common exit, which waits for the CTA's own bulk copies in flight
// and frees its tensor memory.  The host reports HX_ERR_TIMEOUT.
#define HX_TC_MAX_RING 12
#define RING_SLOTS ((uint32_t)P.tc_ring)
#ifndef NCW
#define NCW 8
#endif
#define NCT (NCW * 32)
#define NMW 2                       // MMA warps
#define PT (NCT + 32 + NMW * 32)    // + producer warp + MMA warps
// mbar_wait (hx_persist_common.cuh) reads its limit from the word after the abort flag it is given
#define WAIT_LIMIT (reinterpret_cast<volatile unsigned*>(abort_flag)[1])
#include "hx_persist.cuh"
#include "hx_persist_common.cuh"
#include "hx_gemm_tc.cuh"

#define TC_NDIG 16
#define TM_COLS 512
#define TM_D0 0                     // accumulators of TC_NDIG columns: two pieces in flight, one per MMA warp
#define TM_SFB 64                   // constant unit scales for the digit columns, + MMA warp * 4
#define TM_SFA 96                   // + slot * 16 + K step * 4
#define ATT_ROWS 160                // rows of an attention tile at most, and the stride of a head's probabilities
#define EPI_WARPS 4                 // warps 0..3 own TMEM lanes 0..127 = the rows of a tile
#define DRAIN_LIMIT (1u << 22)

typedef unsigned long long u64;

// per-phase time stamps of one CTA, debug builds only (-DHX_DEBUG_STAMPS)
#ifdef HX_DEBUG_STAMPS
#define DF_STAMP(i) do { if (P.dbg && cta == P.dbg_cta && tid == 0) { unsigned long long _t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(_t)); P.dbg[pi * 16 + (i)] = _t; } } while (0)
#define DF_MARK(ev) do { if (P.dbg_all && tid == 0) { unsigned long long _t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(_t)); P.dbg_all[((size_t)pi * gridDim.x + blockIdx.x) * 8 + (ev)] = _t; } } while (0)
#define DF_GT(v) asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(v))
#define DF_MMA_T0() unsigned long long _w0; DF_GT(_w0)
#define DF_MMA_T1() do { unsigned long long _w1; DF_GT(_w1); dbg_wait += _w1 - _w0; } while (0)
#define DF_MMA_OUT() do { if (P.dbg_all && mw == 0) { unsigned long long _t; DF_GT(_t); P.dbg_all[((size_t)pi * gridDim.x + blockIdx.x) * 8 + 7] = _t; P.dbg_all[((size_t)pi * gridDim.x + blockIdx.x) * 8 + 6] = dbg_wait; } } while (0)
#else
#define DF_STAMP(i) do { } while (0)
#define DF_MARK(ev) do { } while (0)
#define DF_MMA_T0() do { } while (0)
#define DF_MMA_T1() do { } while (0)
#define DF_MMA_OUT() do { } while (0)
#endif

namespace {

__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout = 0) {
    return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) | ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) |
           (1ull << 46) | ((uint64_t)layout << 61);
}
#define TC_SW128 2u
__device__ __forceinline__ void tc_cp_sf(uint32_t taddr, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" :: "r"(taddr), "l"(desc) : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t acc) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}"
                 :: "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(sfa), "r"(sfb) : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(smem_u32(bar)) : "memory");
}
// One lane of a converged warp; the branch it guards is known to be taken by a single thread.
__device__ __forceinline__ bool tc_elect() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
    return p != 0;
}
// A wait of the whole warp: every lane gets the same answer, so the warp leaves a loop together.
__device__ __forceinline__ bool warp_wait(uint64_t* b, uint32_t parity, volatile int* abort_flag) {
    if (__all_sync(0xffffffffu, mbar_try(b, parity))) return true;
    return __all_sync(0xffffffffu, mbar_wait(b, parity, abort_flag));
}
__device__ __forceinline__ void epi_sync() { asm volatile("bar.sync 2, %0;" :: "n"(EPI_WARPS * 32) : "memory"); }
// consumer barrier that also ORs a flag over the consumer threads: every thread gets the same answer
__device__ __forceinline__ bool consumer_sync_any(int flag) {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "r"(flag), "n"(NCT) : "memory");
    return r != 0;
}

struct SmemDf {
    uint64_t full[HX_TC_MAX_RING];
    uint64_t empty[HX_TC_MAX_RING];
    uint64_t acc_full[2], acc_empty[2], b_ready;
    float red[NCW * 2];
    float att_m[8], att_l[8], att_r[8];
    float bv[NCW]; int bi[NCW];
    float swi[128];
    HxPhase ph[2];
    AttPlan ap; int att_ns, ap_tile_rows, ap_ntiles;      // attention work split of this launch (depends on the position only)
    int rowk[ATT_ROWS], rowv[ATT_ROWS];                   // where the rows of the attention tile in flight lie
    unsigned ticket;
    uint32_t tmem_base;
    volatile int abort_flag; unsigned wait_limit;      // adjacent: bounded waits read the limit at (&abort_flag)[1]
};

// ---- (value, epoch) pairs ----
__device__ __forceinline__ void ll_st(u64* p, float v, unsigned ep) {
    const u64 w = ((u64)ep << 32) | (u64)__float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" :: "l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ void ll_st_sys(u64* p, float v, unsigned ep) {
    const u64 w = ((u64)ep << 32) | (u64)__float_as_uint(v);
    asm volatile("st.relaxed.sys.global.u64 [%0], %1;" :: "l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ u64 ll_ld(const u64* p) {
    u64 w; asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory"); return w;
}
__device__ __forceinline__ u64 ll_ld_sys(const u64* p) {
    u64 w; asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory"); return w;
}
__device__ __forceinline__ void ll_ld2(const u64* p, u64& a, u64& b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ float ll_val(u64 w) { return __uint_as_float((unsigned)w); }
__device__ __forceinline__ bool ll_ok(u64 w, unsigned ep) { return (unsigned)(w >> 32) == ep; }
__device__ __forceinline__ bool df_gave_up(SmemDf& S, const HxPersist& P) {
    return S.abort_flag != 0 || *reinterpret_cast<volatile int*>(P.err) != 0;
}
__device__ __forceinline__ void df_fail(SmemDf& S, const HxPersist& P) { S.abort_flag = 1; *P.err = 1; }

// One pair.  After an abort the wait returns at once with whatever is there.
template <bool SYS = false>
__device__ __forceinline__ float df_wait1(const u64* p, unsigned ep, SmemDf& S, const HxPersist& P) {
    const unsigned lim = S.abort_flag ? 1u : S.wait_limit;
    u64 w = 0;
    for (unsigned i = 0; i < lim; i++) {
        w = SYS ? ll_ld_sys(p) : ll_ld(p);
        if (ll_ok(w, ep)) return ll_val(w);
        if ((i & 63u) == 63u && df_gave_up(S, P)) break;
    }
    df_fail(S, P);
    return ll_val(w);
}
// Up to four pairs `stride` apart, all in flight together; returns their values added to `acc` in index order.
__device__ __forceinline__ float df_wait_add4(const u64* p, size_t stride, int n, unsigned ep, float acc, SmemDf& S, const HxPersist& P) {
    const unsigned lim = S.abort_flag ? 1u : S.wait_limit;
    u64 w[4] = {0, 0, 0, 0};
    bool ok = false;
    for (unsigned i = 0; i < lim && !ok; i++) {
        ok = true;
#pragma unroll
        for (int c = 0; c < 4; c++) if (c < n) w[c] = ll_ld(p + (size_t)c * stride);
#pragma unroll
        for (int c = 0; c < 4; c++) if (c < n) ok = ok && ll_ok(w[c], ep);
        if (!ok && (i & 63u) == 63u && df_gave_up(S, P)) break;
    }
    if (!ok) df_fail(S, P);
#pragma unroll
    for (int c = 0; c < 4; c++) if (c < n) acc += ll_val(w[c]);
    return acc;
}
// Two pairs at a 16-byte aligned address.
__device__ __forceinline__ void df_wait2(const u64* p, unsigned ep, float& a, float& b, SmemDf& S, const HxPersist& P) {
    const unsigned lim = S.abort_flag ? 1u : S.wait_limit;
    u64 x = 0, y = 0;
    for (unsigned i = 0; i < lim; i++) {
        ll_ld2(p, x, y);
        if (ll_ok(x, ep) && ll_ok(y, ep)) { a = ll_val(x); b = ll_val(y); return; }
        if ((i & 63u) == 63u && df_gave_up(S, P)) break;
    }
    df_fail(S, P);
    a = ll_val(x); b = ll_val(y);
}
// ---- attention work split: the number of splits follows the context length (about 16 positions each) ----
__device__ __noinline__ AttPlan att_plan_df(const HxPersist& P, int cta, int pos, int nring, int* ns_out, int* tile_rows, int* ntiles) {
#ifndef DF_SPLIT_ROWS_LOG2
#define DF_SPLIT_ROWS_LOG2 4          // about 16 cached positions per attention split while CTAs are left (measured best: 8..16)
#endif
    int ns = (pos + (1 << DF_SPLIT_ROWS_LOG2)) >> DF_SPLIT_ROWS_LOG2;
    ns = ns < 1 ? 1 : (ns > P.att_nsplit ? P.att_nsplit : ns);
    struct { int NKV, DH; } ph = {P.att_nkv, P.att_dh};
    AttPlan a;
    a.active = cta < ph.NKV * ns;
    a.kv = cta / ns; a.split = cta % ns;
    const int T = pos + 1, chunk = (T + ns - 1) / ns;
    a.t0 = a.split * chunk; a.t1 = min(T, a.t0 + chunk);
    if (!a.active || a.t0 >= a.t1) { a.t0 = a.t1 = 0; a.n_old = 0; a.has_new = 0; }
    else { a.has_new = (pos >= a.t0 && pos < a.t1); a.n_old = (a.t1 - a.t0) - a.has_new; }
    a.rows_per_slot = HX_RING_SLOT / (ph.DH * 4);
    a.nslots = (a.n_old + a.rows_per_slot - 1) / a.rows_per_slot;      // K slots == V slots
    const AttPlan2 a2 = att_plan2(a, nring);
    *ns_out = ns; *tile_rows = a2.tile_rows; *ntiles = a2.ntiles;
    return a;
}

// ------------------------------------------------------------------------------------------------
// Attention phase of one CTA: (kv head, split of the cached positions); the split of the work depends on the
// position only and is worked out once per launch (SmemDf::ap).  q (normed, rotated) and this position's k and v
// arrive as pairs from the qkv epilogue; older rows stream through the ring from the cache in tiles of up to four slots.
//  * scores: a warp takes eight rows at a time against all heads of the group, eight lanes per row and two rows per lane
//    (reading the queries from shared memory is most of the traffic); the heads' sums are reduced across the eight lanes
//    together (each exchange halves the values a lane carries);
//  * soft-max statistics (online, m seeded -1e8 like the reference, fused_decode_attn_kernel.hx:74-102): one warp
//    per head;
//  * P*V: a thread owns four output dimensions of ALL heads of the group over a contiguous run of the tile's rows, four
//    rows per step (a V row and a vector of four probabilities are read once); the runs are folded through shared memory.
// The split's partial output and (max, sum) leave as pairs; one CTA per head merges the splits (attention_merge_df, called
// from the phase loop: nested in this function its registers pushed values of the caller to local memory, and a reload a
// phase later comes from L2).
// What bounds it: shared memory and the arithmetic of the two products for groups of eight heads at long contexts, latency
// below.  The 64-layer shape at 4096 positions (228 rows x 8 heads a CTA): 29.8 us a phase with a thread per (row, head,
// eighth), 20.4 with all heads per row, 17.1 with two rows per lane.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void ring_adv(uint32_t& slot, uint32_t& par, uint32_t n, uint32_t nring) {
    slot += n;
    while (slot >= nring) { slot -= nring; par ^= 1u; }
}
// two pairs to a 16-byte aligned address (each of them is single-copy atomic)
__device__ __forceinline__ void ll_st2(u64* p, float a, float b, unsigned ep) {
    const u64 x = ((u64)ep << 32) | (u64)__float_as_uint(a), y = ((u64)ep << 32) | (u64)__float_as_uint(b);
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" :: "l"(p), "l"(x), "l"(y) : "memory");
}
// The splits of a head merged into the attention output, by one CTA per head: the CTA of (kv head, split s) takes
// the heads s, s + ns, ... of its group once its own partial is out.  out[d] = sum_s w_s acc_s[d] / sum_s w_s l_s with
// w_s = exp(m_s - M).  The threads form groups of DH / 2; group g polls the splits g, g + NG, ... -- their statistics and
// its two dimensions in the same breath, so a merge costs one round trip -- and the groups are combined in order, so the
// result does not depend on timing.  The o_proj phase then reads a plain vector.
__device__ __noinline__ void attention_merge_df(const HxPersist& P, const HxPhase& ph, SmemDf& S, float4* sm, int kv, int split, int ns, int grp, unsigned ep) {
    constexpr int SB = 5;
    const int DH = ph.DH, H2 = DH >> 1, NG = NCT / H2;
    const int tid = threadIdx.x, g = tid / H2, d2 = tid - g * H2;
    #pragma unroll 1
    for (int i = split; i < grp; i += ns) {
        const int h = kv * grp + i;
        const u64* pml = ph.pml_ll + 2 * (size_t)h * ns;
        const u64* pa = ph.pacc_ll + (size_t)h * ns * DH + 2 * d2;
        float M = -INFINITY, Ls = 0.0f, o0 = 0.0f, o1 = 0.0f;
        #pragma unroll 1
        for (int s0 = g; s0 < ns; s0 += SB * NG) {
            u64 w[SB][2], q[SB][2];
            const unsigned lim = S.abort_flag ? 1u : S.wait_limit;
            bool ok = false;
            #pragma unroll 1
            for (unsigned t = 0; t < lim && !ok; t++) {
                ok = true;
#pragma unroll
                for (int c = 0; c < SB; c++) if (s0 + c * NG < ns) { ll_ld2(pml + 2 * (s0 + c * NG), q[c][0], q[c][1]); ll_ld2(pa + (size_t)(s0 + c * NG) * DH, w[c][0], w[c][1]); }
#pragma unroll
                for (int c = 0; c < SB; c++) if (s0 + c * NG < ns) ok = ok && ll_ok(q[c][0], ep) && ll_ok(q[c][1], ep) && ll_ok(w[c][0], ep) && ll_ok(w[c][1], ep);
                if (!ok && (t & 63u) == 63u && df_gave_up(S, P)) break;
            }
            if (!ok) df_fail(S, P);
            float mx = M;
#pragma unroll
            for (int c = 0; c < SB; c++) if (s0 + c * NG < ns) mx = fmaxf(mx, ll_val(q[c][0]));
            const float r = __expf(M - mx);
            M = mx; Ls *= r; o0 *= r; o1 *= r;
#pragma unroll
            for (int c = 0; c < SB; c++) if (s0 + c * NG < ns) {
                const float e = __expf(ll_val(q[c][0]) - M);
                Ls = fmaf(e, ll_val(q[c][1]), Ls); o0 = fmaf(e, ll_val(w[c][0]), o0); o1 = fmaf(e, ll_val(w[c][1]), o1);
            }
        }
        sm[tid] = make_float4(M, Ls, o0, o1);
        consumer_sync();
        if (g == 0) {
            float mx = -INFINITY;
            #pragma unroll 1
            for (int k = 0; k < NG; k++) mx = fmaxf(mx, sm[k * H2 + d2].x);
            float L = 0.0f, a = 0.0f, b = 0.0f;
            #pragma unroll 1
            for (int k = 0; k < NG; k++) {
                const float4 v = sm[k * H2 + d2];
                const float e = __expf(v.x - mx);
                L = fmaf(e, v.y, L); a = fmaf(e, v.z, a); b = fmaf(e, v.w, b);
            }
            ll_st2(ph.out_ll + (size_t)h * DH + 2 * d2, a / L, b / L, ep);
        }
        if (i + ns < grp) consumer_sync();                         // the scratch is reused by the next head
    }
}

template <int GRP>
__device__ __noinline__ void attention_df(const HxPersist& P, const HxPhase& ph, SmemDf& S, uint8_t* ring, uint8_t* digb,
                                          uint32_t& cslot, uint32_t& cpar, int pi, int pos) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, cta = blockIdx.x;
    (void)cta; (void)pos;
    const int ns = S.att_ns;
    const AttPlan ap = S.ap;
    const int tr_rows = S.ap_tile_rows, ntiles = S.ap_ntiles;
    const unsigned ep = P.ep_base + (unsigned)pi + 1u, in_ep = P.ep_base + (unsigned)ph.in_dep + 1u;
    const int DH = ph.DH, HD = GRP * DH, CPT = DH >> 5, CH4 = DH >> 2, NSUB = NCT / CH4;
    constexpr int GP = GRP <= 1 ? 1 : (GRP <= 2 ? 2 : (GRP <= 4 ? 4 : 8)), LG = GP == 1 ? 0 : (GP == 2 ? 1 : (GP == 4 ? 2 : 3));
    const int rps = ap.rows_per_slot, KVD = ph.NKV * DH;
    const uint32_t nring = RING_SLOTS;
    float* sq = reinterpret_cast<float*>(digb);                 // [GRP][128] queries, zero from DH on
    float* knew = sq + 8 * 128;                                  // [DH] current k
    float* vnew = knew + 128;                                    // [DH] current v
    float* sp = vnew + 128;                                      // [GRP][ATT_ROWS] scores / probabilities; merge scratch
    float* accx = sp + 8 * ATT_ROWS;                             // [row run][GRP][DH] partial outputs
    const float* ringf = reinterpret_cast<const float*>(ring);
    const int c_sub = tid / CH4, c_c = tid - c_sub * CH4;
    if (!ap.active) return;
    if (ap.t1 <= ap.t0) {
        // empty split: neutral partial
        for (int i = tid; i < GRP; i += NCT) {
            const int hs = (ap.kv * GRP + i) * ns + ap.split;
            ll_st(ph.pml_ll + 2 * hs, -100000000.0f, ep); ll_st(ph.pml_ll + 2 * hs + 1, 0.0f, ep);
        }
        for (int i = tid; i < HD; i += NCT) {
            const int hs = (ap.kv * GRP + i / DH) * ns + ap.split;
            ll_st(ph.pacc_ll + (size_t)hs * DH + i % DH, 0.0f, ep);
        }
        return;
    }
    float4 acc[GRP];
#pragma unroll
    for (int i = 0; i < GRP; i++) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    {
        // q of the group, and k, v of this position when it falls into the split: one polling site
        const int nq = HD >> 1, nkv = ap.has_new ? DH >> 1 : 0;
        #pragma unroll 1
        for (int i = tid; i < nq + 2 * nkv; i += NCT) {
            const u64* src; float* dst;
            if (i < nq) { const int h = 2 * i / DH; src = ph.in_ll + (size_t)ap.kv * HD + 2 * i; dst = sq + h * 128 + 2 * i - h * DH; }
            else if (i < nq + nkv) { src = ph.kv_ll + (size_t)ap.kv * DH + 2 * (i - nq); dst = knew + 2 * (i - nq); }
            else { src = ph.kv_ll + (size_t)KVD + (size_t)ap.kv * DH + 2 * (i - nq - nkv); dst = vnew + 2 * (i - nq - nkv); }
            df_wait2(src, in_ep, dst[0], dst[1], S, P);
        }
    }
    #pragma unroll 1
    for (int i = tid; i < GRP * (128 - DH); i += NCT) sq[(i / (128 - DH)) * 128 + DH + i % (128 - DH)] = 0.0f;
    if (tid < 8) { S.att_m[tid] = -100000000.0f; S.att_l[tid] = 0.0f; }
    consumer_sync();
    DF_STAMP(7); DF_MARK(1);
    const int ntile = ntiles + ((ap.has_new && ap.n_old % tr_rows == 0) ? 1 : 0);
    #pragma unroll 1
    for (int s = 0; s < ntile; s++) {
        const bool ring_tile = s < ntiles;
        const int nr = ring_tile ? min(tr_rows, ap.n_old - s * tr_rows) : 0;
        const int nsl = (nr + rps - 1) / rps;                       // ring slots of this tile (K, then as many of V)
        const bool add_new = ap.has_new && (s == ntile - 1);       // the current position rides on the last tile
        const int ntot = nr + (add_new ? 1 : 0);
        uint32_t myslot = 0;
        // where the rows lie (floats from the ring's base); one thread per ring slot waits for its rows
        for (int r = tid; r < ntot; r += NCT) {
            const int j = (r >= rps) + (r >= 2 * rps) + (r >= 3 * rps);
            uint32_t ks = cslot + (uint32_t)j, vs = ks + (uint32_t)nsl;
            while (ks >= nring) ks -= nring;
            while (vs >= nring) vs -= nring;
            S.rowk[r] = r < nr ? (int)(ks * (HX_RING_SLOT / 4)) + (r - j * rps) * DH : (int)(knew - ringf);
            S.rowv[r] = r < nr ? (int)(vs * (HX_RING_SLOT / 4)) + (r - j * rps) * DH : (int)(vnew - ringf);
        }
        if (tid < 2 * nsl) {
            uint32_t sl = cslot, pr = cpar;
            ring_adv(sl, pr, (uint32_t)tid, nring);
            mbar_wait(&S.full[sl], pr, &S.abort_flag);
            myslot = sl;
        }
        ring_adv(cslot, cpar, (uint32_t)(2 * nsl), nring);
        consumer_sync();
        if (s == 0) { DF_STAMP(8); DF_MARK(2); }
        // scores
        {
            const int p = lane & 7;
            #pragma unroll 1
            for (int r0 = warp * 8; r0 < ntot; r0 += NCW * 8) {
                const int ra = r0 + (lane >> 3), rb = ra + 4;
                const float* ka = ringf + S.rowk[min(ra, ntot - 1)];
                const float* kb = ringf + S.rowk[min(rb, ntot - 1)];
                float4 k4[2][4];
#pragma unroll
                for (int c = 0; c < 4; c++) {                       // narrow heads: zeros
                    k4[0][c] = *reinterpret_cast<const float4*>((c < CPT ? ka : sq) + (p + 8 * c) * 4);
                    k4[1][c] = *reinterpret_cast<const float4*>((c < CPT ? kb : sq) + (p + 8 * c) * 4);
                }
                float v[2][GP];
#pragma unroll
                for (int i = 0; i < GP; i++) {
                    v[0][i] = v[1][i] = 0.0f;
                    if (i < GRP) {
                        float d0 = 0.0f, d1 = 0.0f, e0 = 0.0f, e1 = 0.0f;
#pragma unroll
                        for (int c = 0; c < 4; c++) {
                            const float4 q4 = *reinterpret_cast<const float4*>(sq + i * 128 + (p + 8 * c) * 4);
                            d0 = fmaf(q4.x, k4[0][c].x, d0); d1 = fmaf(q4.y, k4[0][c].y, d1); d0 = fmaf(q4.z, k4[0][c].z, d0); d1 = fmaf(q4.w, k4[0][c].w, d1);
                            e0 = fmaf(q4.x, k4[1][c].x, e0); e1 = fmaf(q4.y, k4[1][c].y, e1); e0 = fmaf(q4.z, k4[1][c].z, e0); e1 = fmaf(q4.w, k4[1][c].w, e1);
                        }
                        v[0][i] = d0 + d1; v[1][i] = e0 + e1;
                    }
                    asm volatile("" ::: "memory");                      // one head at a time: registers
                }
#pragma unroll
                for (int st = 0; st < 3; st++) {
                    const int o = 4 >> st;
                    if (st < LG) {
                        const int hh = GP >> (st + 1);
                        const bool up = (lane & o) != 0;
#pragma unroll
                        for (int u = 0; u < 2; u++)
#pragma unroll
                            for (int k = 0; k < hh; k++) {
                                const float send = up ? v[u][k] : v[u][k + hh], keep = up ? v[u][k + hh] : v[u][k];
                                v[u][k] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                            }
                    } else { v[0][0] += __shfl_xor_sync(0xffffffffu, v[0][0], o); v[1][0] += __shfl_xor_sync(0xffffffffu, v[1][0], o); }
                }
                const int i = p >> (3 - LG);
                if ((p & ((1 << (3 - LG)) - 1)) == 0 && i < GRP) {
                    if (ra < ntot) sp[i * ATT_ROWS + ra] = v[0][0] * ph.scale;
                    if (rb < ntot) sp[i * ATT_ROWS + rb] = v[1][0] * ph.scale;
                }
            }
        }
        consumer_sync();
        if (s == 0) DF_STAMP(9);
        if (tid < nsl) mbar_arrive(&S.empty[myslot]);
        // online softmax state per head
        if (warp < GRP) {
            const int i = warp;
            float* row = sp + i * ATT_ROWS;
            float x[ATT_ROWS / 32], tm = -INFINITY;
#pragma unroll
            for (int k = 0; k < ATT_ROWS / 32; k++) { x[k] = lane + 32 * k < ntot ? row[lane + 32 * k] : -INFINITY; tm = fmaxf(tm, x[k]); }
            tm = hx_warp_max(tm);
            const float mo = S.att_m[i], mn = fmaxf(mo, tm);
            float ls = 0.0f;
#pragma unroll
            for (int k = 0; k < ATT_ROWS / 32; k++) if (lane + 32 * k < ntot) { const float pr = __expf(x[k] - mn); row[lane + 32 * k] = pr; ls += pr; }
            ls = hx_warp_sum(ls);
            if (lane == 0) { const float rr = __expf(mo - mn); S.att_r[i] = rr; S.att_l[i] = S.att_l[i] * rr + ls; S.att_m[i] = mn; }
        }
        consumer_sync();
        if (s == 0) DF_STAMP(10);
        // P*V
        {
            if (s > 0) {
#pragma unroll
                for (int i = 0; i < GRP; i++) { const float rr = S.att_r[i]; acc[i].x *= rr; acc[i].y *= rr; acc[i].z *= rr; acc[i].w *= rr; }
            }
            const int run = ((ntot + NSUB - 1) / NSUB + 3) & ~3, ra = c_sub * run, rb = min(ntot, ra + run);
            #pragma unroll 1
            for (int r = ra; r < rb; r += 4) {
                float4 v4[4];
#pragma unroll
                for (int u = 0; u < 4; u++) v4[u] = r + u < rb ? *reinterpret_cast<const float4*>(ringf + S.rowv[r + u] + c_c * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                for (int i = 0; i < GRP; i++) {
                    const float4 p4 = *reinterpret_cast<const float4*>(sp + i * ATT_ROWS + r);
                    const float pw[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                    for (int u = 0; u < 4; u++) if (r + u < rb) {
                        acc[i].x = fmaf(pw[u], v4[u].x, acc[i].x); acc[i].y = fmaf(pw[u], v4[u].y, acc[i].y);
                        acc[i].z = fmaf(pw[u], v4[u].z, acc[i].z); acc[i].w = fmaf(pw[u], v4[u].w, acc[i].w);
                    }
                }
            }
        }
        if (s + 1 == ntile) {
#pragma unroll
            for (int i = 0; i < GRP; i++) *reinterpret_cast<float4*>(accx + (c_sub * GRP + i) * DH + c_c * 4) = acc[i];
        }
        consumer_sync();
        if (tid >= nsl && tid < 2 * nsl) mbar_arrive(&S.empty[myslot]);
    }
    DF_STAMP(11); DF_MARK(3);
    // fold the row runs and hand the split's partial over
    #pragma unroll 1
    for (int o = tid; o < GRP * CH4; o += NCT) {
        const int i = o / CH4, c = o - i * CH4;
        float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
        #pragma unroll 1
        for (int u = 0; u < NSUB; u++) {
            const float4 a = *reinterpret_cast<const float4*>(accx + (u * GRP + i) * DH + c * 4);
            O.x += a.x; O.y += a.y; O.z += a.z; O.w += a.w;
        }
        const int hs = (ap.kv * GRP + i) * ns + ap.split;
        u64* dst = ph.pacc_ll + (size_t)hs * DH + c * 4;
        ll_st2(dst, O.x, O.y, ep); ll_st2(dst + 2, O.z, O.w, ep);
        if (c == 0) ll_st2(ph.pml_ll + 2 * hs, S.att_m[i], S.att_l[i], ep);
    }
    DF_MARK(4);
}


template <bool TP>
__global__ void __launch_bounds__(PT, 1) k_decode_df(const __grid_constant__ HxPersist P) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    SmemDf& S = *reinterpret_cast<SmemDf*>(smem_raw);
    // swizzled operands need 1024-byte aligned cells (the swizzle is a function of the shared-memory address)
    uint8_t* sfb1 = smem_raw + ((sizeof(SmemDf) + 15) & ~(size_t)15);    // 512 bytes of 0x38 (scale 1.0)
    uint8_t* ring = smem_raw + (((smem_u32(smem_raw) + (uint32_t)sizeof(SmemDf) + 16u + 512u + 1023u) & ~1023u) - smem_u32(smem_raw));
    uint8_t* digb = ring + (size_t)P.tc_ring * HX_RING_SLOT;              // digit columns / attention scratch (1024-aligned)
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;      // warp-uniform for the compiler too
    const int cta = blockIdx.x, grid = gridDim.x;
    const int pos = *P.pos;
    const uint32_t nring = (uint32_t)P.tc_ring;

    if (tid == 0) {
        for (int i = 0; i < HX_TC_MAX_RING; i++) { mbar_init(&S.full[i], 1); mbar_init(&S.empty[i], 1); }
        mbar_init(&S.acc_full[0], NMW); mbar_init(&S.acc_full[1], NMW);
        mbar_init(&S.acc_empty[0], EPI_WARPS); mbar_init(&S.acc_empty[1], EPI_WARPS);
        mbar_init(&S.b_ready, 1);
        S.abort_flag = 0; S.wait_limit = P.wait_limit;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (tid < 128) reinterpret_cast<uint32_t*>(sfb1)[tid] = 0x38383838u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == NCW + 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" :: "r"(smem_u32(&S.tmem_base)), "n"(TM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = S.tmem_base;

    if (warp == NCW) {
        // =========================== producer ===========================
        if (lane == 0) {
            uint32_t slot = 0, par = 0, npush = 0;
            bool first_round = true;
            auto push = [&](const void* src, uint32_t bytes) -> bool {
                if (!first_round && !mbar_wait(&S.empty[slot], par, &S.abort_flag)) return false;
                mbar_expect_tx(&S.full[slot], bytes);
                bulk_g2s(ring + (size_t)slot * HX_RING_SLOT, src, bytes, &S.full[slot]);
                npush++;
                if (++slot == nring) { slot = 0; if (first_round) first_round = false; else par ^= 1u; }
                return true;
            };
            bool ok = true;
            int a_ns, a_trows, a_ntiles;
            const AttPlan ap = att_plan_df(P, cta, pos, (int)nring, &a_ns, &a_trows, &a_ntiles);
            HxPhase nxt = P.phases[0];
#pragma unroll 1
            for (int pi = 0; pi < P.nphases && ok; pi++) {
                const HxPhase ph = nxt;
                if (pi + 1 < P.nphases) {
                    nxt = P.phases[pi + 1];
                    // one CTA per phase pulls the small vectors of the next phase into L2 (a token's worth of weights
                    // has evicted them since their last use)
                    if (cta == (pi % grid)) {
                        const HxPhase& q = P.phases[pi + 1];
                        if (q.type == HX_PH_LINEAR_TC) {
                            if (q.norm == HX_NORM_RMS && q.g) l2_prefetch(q.g, (uint32_t)q.K * 4u);
                            if (q.epi == HX_EPI_QKV) {
                                if (q.qn_g) l2_prefetch(q.qn_g, (uint32_t)q.DH * 4u);
                                if (q.kn_g) l2_prefetch(q.kn_g, (uint32_t)q.DH * 4u);
                                if (q.cosT) { l2_prefetch(q.cosT + (size_t)pos * (q.DH >> 1), (uint32_t)q.DH * 2u); l2_prefetch(q.sinT + (size_t)pos * (q.DH >> 1), (uint32_t)q.DH * 2u); }
                            }
                        }
                    }
                }
                if (ph.type == HX_PH_LINEAR_TC) {
                    const int b0 = ph.plan[cta].b0, b1 = ph.plan[cta].b1;
                    const uint8_t* src = ph.w + (size_t)b0 * HX_T128_CELL;
#pragma unroll 1
                    for (int g = b0; g < b1 && ok; g++, src += HX_T128_CELL) ok = push(src, HX_T128_CELL);
                } else if (ph.type == HX_PH_ATTN) {
                    const size_t rowb = (size_t)ph.DH * 4;
                    // tiles of up to tr slots of K rows followed by as many of V rows (attention_df)
#pragma unroll 1
                    for (int t = 0; t < a_ntiles && ok; t++) {
                        const int r0 = ap.t0 + t * a_trows, nrt = min(a_trows, ap.t0 + ap.n_old - r0);
#pragma unroll 1
                        for (int kv2 = 0; kv2 < 2 && ok; kv2++) {
#pragma unroll 1
                            for (int r = 0; r < nrt && ok; r += ap.rows_per_slot) {
                                const size_t off = ((size_t)ap.kv * ph.cap + r0 + r) * ph.DH;
                                ok = push((kv2 ? ph.vc : ph.kc) + off, (uint32_t)(min(ap.rows_per_slot, nrt - r) * rowb));
                            }
                        }
                    }
                }
            }
            // the CTA must not end with a bulk copy of its own in flight: wait for the last copy into every slot
            const uint32_t first = npush > nring ? npush - nring : 0u;
            for (uint32_t j = first; j < npush; j++) {
                const uint32_t s = j % nring, pr = (j / nring) & 1u;
                for (uint32_t i = 0; i < DRAIN_LIMIT; i++) if (mbar_try(&S.full[s], pr)) break;
            }
        }
    } else if (warp > NCW) {
        // =========================== MMA issuers ===========================
        // Two warps: what one cell costs its issuer -- wait for the ring slot, copies, MMAs, commit -- is about 700 cycles of
        // latencies one after the other, against 350 on the tensor pipe, so with a single warp the cells that lay in the
        // ring already went by at 0.37 us each.  A warp takes the cells of the ring slots of its parity (so it sees every use
        // of a slot that it waits for) into its own accumulator; the read-out adds the two.
        // The whole warp runs the loop and one elected lane issues: with the control flow convergent, descriptors and
        // addresses stay in uniform registers.  A single-thread branch (lane == 0) makes the compiler move every operand
        // over for each instruction: 170 cycles per MMA (with its scale copy) against 87 at N = 16.
        {
            const uint32_t mw = (uint32_t)(warp - NCW - 1), sfb = tmem + TM_SFB + mw * 4;
            if (tc_elect()) tc_cp_sf(sfb, tc_desc(smem_u32(sfb1), 16, 128));
            const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(TC_NDIG >> 3) << 17) | (8u << 24);
            const uint64_t a_ring = tc_desc(smem_u32(ring), 16, 1024, TC_SW128);    // 8-row groups 1024 B apart, 128-byte swizzle
            const uint64_t sf_ring = tc_desc(smem_u32(ring) + 16384, 16, 128);
            const uint64_t b_base = tc_desc(smem_u32(digb), 16, 1024, TC_SW128);
            uint32_t slot = 0, par = 0, uc = 0, tcph = 0;
            bool ok = true;
            int a_ns, a_trows, a_ntiles;
            const AttPlan ap = att_plan_df(P, cta, pos, (int)nring, &a_ns, &a_trows, &a_ntiles);
#pragma unroll 1
            for (int pi = 0; pi < P.nphases && ok; pi++) {
                const HxPhase& ph = P.phases[pi];
                if (ph.type == HX_PH_LINEAR_TC) {
                    const HxCtaPlan tp = ph.plan[cta];
                    ok = warp_wait(&S.b_ready, tcph & 1, &S.abort_flag);        // digit columns of this phase are in place
                    tcph++;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    unsigned long long dbg_wait = 0; (void)dbg_wait;
                    int kc = tp.k0, dp = 0;              // K cell of the tile, its position among the digit cells
                    bool fresh = true, first = true;     // at the start of a piece; before this warp's first cell of it
                    uint32_t dcol = 0;
#pragma unroll 1
                    for (int g = tp.b0; g < tp.b1 && ok; g++) {
                        if (fresh) {
                            const uint32_t buf = uc & 1u;
                            if (uc >= 2) ok = warp_wait(&S.acc_empty[buf], ((uc >> 1) - 1) & 1, &S.abort_flag);
                            if (!ok) break;
                            dcol = tmem + TM_D0 + (buf * NMW + mw) * TC_NDIG;
                            first = true;
                        }
                        const bool last = kc + 1 == tp.C || g + 1 == tp.b1;      // last cell of this tile's piece
                        if ((slot & 1u) == mw) {
                            { DF_MMA_T0(); ok = warp_wait(&S.full[slot], par, &S.abort_flag); DF_MMA_T1(); }
                            if (!ok) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            // descriptors advance in 16-byte units: a K step is 32 B of a swizzled row, a scale chunk 512 B
                            const uint64_t a_slot = a_ring + (uint64_t)(slot * (HX_RING_SLOT >> 4));
                            const uint64_t sf_slot = sf_ring + (uint64_t)(slot * (HX_RING_SLOT >> 4));
                            const uint64_t b_cell = b_base + (uint64_t)(dp * 128);
                            const uint32_t tsf = tmem + TM_SFA + slot * 16;
                            if (tc_elect()) {
#pragma unroll
                                for (int e = 0; e < 4; e++) tc_cp_sf(tsf + e * 4, sf_slot + (uint64_t)(e * 32));
#pragma unroll
                                for (int e = 0; e < 4; e++)
                                    tc_mma(dcol, a_slot + (uint64_t)(e * 2), b_cell + (uint64_t)(e * 2), idesc, tsf + e * 4, sfb,
                                           (first && e == 0) ? 0u : 1u);
                                tc_commit(&S.empty[slot]);
                            }
                            __syncwarp();
                            first = false;
                        }
                        if (last) {
                            if (tc_elect()) tc_commit(&S.acc_full[uc & 1u]);     // arrives at once where this warp had no cell
                            __syncwarp();
                        }
                        fresh = last;
                        if (++slot == nring) { slot = 0; par ^= 1u; }
                        if (++dp == tp.C) dp = 0;
                        if (last) { uc++; kc = 0; } else kc++;
                    }
                    DF_MMA_OUT();
                } else if (ph.type == HX_PH_ATTN) {
                    ring_adv(slot, par, 2u * (uint32_t)ap.nslots, nring);         // ring slots the consumers use for K and V rows
                }
            }
        }
    } else {
        // =============================== consumers ===============================
        uint32_t cslot = 0, cpar = 0, uc = 0;                 // ring cursor of the consumers (attention rows), accumulator use count
        float best_v = -INFINITY; int best_i = INT_MAX;
        if (tid == 0) S.ap = att_plan_df(P, cta, pos, (int)nring, &S.att_ns, &S.ap_tile_rows, &S.ap_ntiles);

        constexpr int PH_CHUNKS = (int)(sizeof(HxPhase) / 16);
        if (tid < PH_CHUNKS) reinterpret_cast<uint4*>(&S.ph[0])[tid] = __ldg(reinterpret_cast<const uint4*>(P.phases) + tid);
        if (P.inject_stall && tid == 0) (void)df_wait1(reinterpret_cast<const u64*>(P.err) + 1, 0xFFFFFFFFu, S, P);   // nothing ever writes this epoch
        if (consumer_sync_any(S.abort_flag)) goto aborted;
#pragma unroll 1
        for (int pi = 0; pi < P.nphases; pi++) {
            const HxPhase& ph = S.ph[pi & 1];
            const unsigned ep = P.ep_base + (unsigned)pi + 1u;
            DF_STAMP(0); DF_MARK(0);
            // the next descriptor travels to shared memory while this phase runs (its slot was last read a phase ago)
            if (pi + 1 < P.nphases && tid < PH_CHUNKS)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(smem_u32(reinterpret_cast<uint4*>(&S.ph[(pi + 1) & 1]) + tid)),
                             "l"(reinterpret_cast<const uint4*>(P.phases + pi + 1) + tid) : "memory");
            if (ph.type == HX_PH_LINEAR_TC) {
                // ---------- prologue: x -> (norm) -> sixteen base-4 digit columns in operand layout ----------
                // Pass 1 stages the CTA's K slice of the input (times the norm gain) in the first half of each digit
                // cell and finds its largest magnitude; pass 2 turns the staged values into digit words.  The code runs
                // once per phase from a cold instruction cache, so it is kept small: one polling site, one digit site.
                const int K = ph.K;
                const HxCtaPlan tp = ph.plan[cta];
                const unsigned in_ep = P.ep_base + (unsigned)ph.in_dep + 1u;
                const bool rms = ph.norm == HX_NORM_RMS;
                // layer 0: the embedding row of the token is the input of qkv and the residual of o_proj
                const float* xrow = ph.tok ? ph.x + (size_t)(ph.tok[P.tok_by_pos ? pos : 0]) * (size_t)ph.res_ld : ph.x;
                const int nitems = tp.run * 32;
                float ss = 0.0f, mx = 0.0f;
                {
                    // Sum of squares of the whole input: per-tile sums published by the producing epilogue, added in tile
                    // order (every CTA gets the same bits); layer 0 reads the embedding row itself.
                    if (rms && !ph.in_stat) {
                        #pragma unroll 1
                        for (int k = tid * 4; k < K; k += NCT * 4) {
                            const float4 a = __ldcg(reinterpret_cast<const float4*>(xrow + k));
                            ss += a.x * a.x + a.y * a.y + a.z * a.z + a.w * a.w;
                        }
                    }
                    // A unit is two consecutive elements (one 16-byte load), so a warp's load is 512 contiguous bytes.  UI
                    // units per thread and round are in flight together, with the norm gains fetched before the wait and,
                    // in the first round of warp 0, the per-tile sums of squares polled in the same breath.  A poll asks only
                    // for what has not come yet: the tiles arrive over a microsecond or two, and 148 CTAs asking for the whole
                    // vector again and again (4.8 MB a round at K = 4096) would keep L2 busy for longer than a round trip.
                    constexpr int UI = 8;
                    const int nunits = nitems * 4;
                    #pragma unroll 1
                    for (int u0 = tid; u0 < nunits; u0 += UI * NCT) {
                        int kk[UI]; float2 gg[UI]; u64 w[UI][2];
#pragma unroll
                        for (int j = 0; j < UI; j++) {
                            const int u = u0 + j * NCT;
                            int kc = tp.k0 + (u >> 7); if (kc >= tp.C) kc -= tp.C;
                            const int k = kc * 256 + (u & 127) * 2;
                            kk[j] = (u < nunits && k < K) ? k : -1;
                            gg[j] = (rms && kk[j] >= 0) ? *reinterpret_cast<const float2*>(ph.g + k) : make_float2(1.0f, 1.0f);
                            w[j][0] = w[j][1] = 0;
                        }
                        const bool stat_round = rms && ph.in_stat != nullptr && warp == 0 && u0 == tid;
                        const bool st_a = stat_round && lane < ph.n_in_stat, st_b = stat_round && lane + 32 < ph.n_in_stat;
                        u64 sa = 0, sb = 0;
                        if (ph.in_ll) {
                            const unsigned lim = S.abort_flag ? 1u : S.wait_limit;
                            bool ok = false;
                            #pragma unroll 1
                            for (unsigned t = 0; t < lim && !ok; t++) {
#pragma unroll
                                for (int j = 0; j < UI; j++)
                                    if (kk[j] >= 0 && !(ll_ok(w[j][0], in_ep) && ll_ok(w[j][1], in_ep))) ll_ld2(ph.in_ll + kk[j], w[j][0], w[j][1]);
                                if (st_a && !ll_ok(sa, in_ep)) sa = ll_ld(ph.in_stat + lane);
                                if (st_b && !ll_ok(sb, in_ep)) sb = ll_ld(ph.in_stat + lane + 32);
                                ok = (!st_a || ll_ok(sa, in_ep)) && (!st_b || ll_ok(sb, in_ep));
#pragma unroll
                                for (int j = 0; j < UI; j++) if (kk[j] >= 0) ok = ok && ll_ok(w[j][0], in_ep) && ll_ok(w[j][1], in_ep);
                                if (!ok && (t & 63u) == 63u && df_gave_up(S, P)) break;
                            }
                            if (!ok) df_fail(S, P);
                        } else {
#pragma unroll
                            for (int j = 0; j < UI; j++) if (kk[j] >= 0) {
                                const float2 a = __ldcg(reinterpret_cast<const float2*>(xrow + kk[j]));
                                w[j][0] = __float_as_uint(a.x); w[j][1] = __float_as_uint(a.y);
                            }
                        }
                        if (st_a) ss += ll_val(sa);
                        if (st_b) ss += ll_val(sb);
#pragma unroll
                        for (int j = 0; j < UI; j++) {
                            const int u = u0 + j * NCT;
                            if (u >= nunits) continue;
                            const float v0 = kk[j] >= 0 ? ll_val(w[j][0]) * gg[j].x : 0.0f, v1 = kk[j] >= 0 ? ll_val(w[j][1]) * gg[j].y : 0.0f;
                            mx = fmaxf(mx, fmaxf(fabsf(v0), fabsf(v1)));
                            *reinterpret_cast<float2*>(digb + (size_t)(u >> 7) * 2048 + (u & 127) * 8) = make_float2(v0, v1);
                        }
                    }
                }
                DF_MARK(1);
                ss = hx_warp_sum(ss); mx = hx_warp_max(mx);
                if (lane == 0) { S.red[warp] = ss; S.red[NCW + warp] = mx; }
                consumer_sync();
                float inv = 1.0f, Sg = 1.0f;
                {
                    float tss = 0.0f, tmx = 0.0f;
#pragma unroll
                    for (int i = 0; i < NCW; i++) { tss += S.red[i]; tmx = fmaxf(tmx, S.red[NCW + i]); }
                    if (rms) inv = rsqrtf(tss / (float)K + ph.eps);
                    const float vmax = tmx * inv * 1.0000005f;            // margin for the rounding of x*g*inv
                    if (vmax > 0.0f && vmax < INFINITY) Sg = __uint_as_float(__float_as_uint(vmax) & 0x7F800000u);   // vmax/Sg in [1,2)
                }
                DF_STAMP(14);
                const float mul = (inv / Sg) * 2147483648.0f;             // |x_n| / Sg * 2^31 < 2^32
                #pragma unroll 1
                for (int it = tid; it < nitems; it += NCT) {
                    const float4* xs = reinterpret_cast<const float4*>(digb + (size_t)(it >> 5) * 2048 + (it & 31) * 32);
                    const float4 va = xs[0], vb = xs[1];
                    __syncwarp();                                          // a warp turns a whole cell over: read, then written
                    const float v[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, vb.w};
                    uint32_t M[8]; uint32_t sg = 0u;
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        M[e] = __float2uint_rn(fabsf(v[e]) * mul);
                        sg |= (__float_as_uint(v[e]) >> (28 - 4 * e)) & (8u << (4 * e));
                    }
                    // digit n of element e is bits 31-2n, 30-2n of M[e]; it lands on bits 4e+1, 4e of the word of row n
                    const int j = (it >> 2) & 7, w = it & 3;               // 16-byte chunk and word of this item in its cell
                    uint8_t* dst = digb + (size_t)(it >> 5) * 2048 + w * 4;
                    uint32_t rowv[16];
                    hx_digit_rows(M, sg, rowv);
#pragma unroll
                    for (int n = 0; n < TC_NDIG; n++) *reinterpret_cast<uint32_t*>(dst + n * 128 + ((j ^ (n & 7)) << 4)) = rowv[n];
                }
                DF_STAMP(15);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                consumer_sync();
                if (tid == 0) mbar_arrive(&S.b_ready);
                DF_STAMP(1); DF_MARK(2);

                // ---------- pieces of tiles: accumulator -> digits recombined -> merge -> epilogue ----------
                uint32_t pslot = cslot;                    // ring slot of the first cell of a piece
                int pleft = tp.b1 - tp.b0, pk = tp.k0;     // cells left, first K cell of the piece
                ring_adv(cslot, cpar, (uint32_t)(tp.b1 - tp.b0), nring);
                const int t_first = tp.t_first, t_last = tp.t_last;
                if (warp < EPI_WARPS) {
                    const float out_scale = Sg;       // x_n = Sg * sum_j 4^-j * (digit_j / 2), and digit/2 is the E2M1 value
                    const int rl = warp * 32 + lane;
                    const unsigned res_ep = P.ep_base + (unsigned)ph.res_dep + 1u;
#pragma unroll 1
                    for (int tile = t_first; tile <= t_last; tile++) {
                        const uint32_t buf = uc & 1u;
                        // the MMA warps that had a cell of this piece (both from three cells on: two neighbours are of one
                        // parity only where an odd ring wraps)
                        const int pn = min(tp.C - pk, pleft);
                        const uint32_t pnext = pslot + 1 == nring ? 0u : pslot + 1;
                        const bool had0 = pn > 2 || !(pslot & 1u) || (pn == 2 && !(pnext & 1u)), had1 = pn > 2 || (pslot & 1u) || (pn == 2 && (pnext & 1u));
                        pslot = (pslot + (uint32_t)pn) % nring; pleft -= pn; pk = 0;
                        // the CTA holding a tile's first cell merges it (see HxCtaPlan)
                        const bool merger = tile > t_first || tp.first_merger;
                        const int others = tile == t_last ? tp.last_others : 0;
                        // operands of the epilogue that are final already travel while the MMAs of this piece run
                        float yres = 0.0f;
                        if (merger && ph.epi == HX_EPI_RESID && tile * 128 + rl < ph.N)
                            yres = ph.res_ll ? df_wait1(ph.res_ll + tile * 128 + rl, res_ep, S, P) : __ldcg(xrow + tile * 128 + rl);
                        float pre_g = 1.0f, pre_cs = 1.0f, pre_sn = 0.0f;
                        if (merger && ph.epi == HX_EPI_QKV) {
                            const int row = tile * 128 + rl, e = row % ph.DH, half = ph.DH >> 1;
                            const int sec = row < ph.NH * ph.DH ? 0 : (row < (ph.NH + ph.NKV) * ph.DH ? 1 : 2);
                            const float* gg = sec == 0 ? ph.qn_g : (sec == 1 ? ph.kn_g : nullptr);
                            if (gg) pre_g = gg[e];
                            if (ph.cosT) { pre_cs = ph.cosT[(size_t)pos * half + (e < half ? e : e - half)]; pre_sn = ph.sinT[(size_t)pos * half + (e < half ? e : e - half)]; }
                        }
                        mbar_wait(&S.acc_full[buf], (uc >> 1) & 1, &S.abort_flag);
                        uc++;
                        if (tile == t_last) DF_MARK(3);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        float v = 0.0f;
#pragma unroll
                        for (int h = 0; h < NMW; h++) {
                            if (h == 0 ? !had0 : !had1) continue;
                            uint32_t r[16];
                            const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + TM_D0 + (buf * NMW + h) * TC_NDIG;
                            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                                           "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                                         : "r"(ta));
                            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                            float a = 0.0f;
#pragma unroll
                            for (int j = TC_NDIG - 1; j >= 0; j--) a = fmaf(a, 0.25f, __uint_as_float(r[j]));
                            v += a;
                        }
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&S.acc_empty[buf]);
                        v *= out_scale;
                        if (!merger) {            // pieces 1.. hand their rows to the merger
                            ll_st(ph.part_ll + ((size_t)tile * ph.pieces + (size_t)tp.first_piece) * 128 + rl, v, ep);
                            continue;
                        }
                        #pragma unroll 1
                        for (int q = 0; q < others; q += 4)
                            v = df_wait_add4(ph.part_ll + ((size_t)tile * ph.pieces + (size_t)q) * 128 + rl, 128, min(4, others - q), ep, v, S, P);
                        if (tile == t_last) DF_MARK(4);
                        if (ph.epi == HX_EPI_QKV) {
                            // A tile holds 128 / DH whole heads (DH is 32, 64 or 128).  Per-head RMSNorm and rotate_half
                            // RoPE on q and k; q leaves as pairs, k and v as pairs and into the cache row of this position.
                            const int DH = ph.DH, half = DH >> 1, QD = ph.NH * DH, KVD = ph.NKV * DH;
                            const int row = tile * 128 + rl;
                            const bool valid = row < ph.N;
                            const int sec = row < QD ? 0 : (row < QD + KVD ? 1 : 2);
                            const int e = row % DH;
                            v = valid ? v * ph.ts[sec] : 0.0f;
                            const float* gg = sec == 0 ? ph.qn_g : (sec == 1 ? ph.kn_g : nullptr);
                            float ssq = hx_warp_sum(v * v);
                            if (DH > 32) {
                                if (lane == 0) S.swi[warp] = ssq;
                                epi_sync();
                                const int w0 = (rl / DH) * (DH >> 5);
                                ssq = 0.0f;
                                for (int j = 0; j < (DH >> 5); j++) ssq += S.swi[w0 + j];
                                epi_sync();
                            }
                            if (gg) v = pre_g * (v * rsqrtf(ssq / (float)DH + ph.eps));
                            if (ph.cosT) {                       // every thread meets the barriers, v rows keep their value
                                S.swi[rl] = v;
                                epi_sync();
                                const float other = S.swi[e < half ? rl + half : rl - half];
                                if (sec < 2) v = e < half ? v * pre_cs - other * pre_sn : v * pre_cs + other * pre_sn;
                                epi_sync();
                            }
                            if (valid) {
                                if (sec == 0) ll_st(ph.out_ll + row, v, ep);
                                else {
                                    const int hrow = row - QD - (sec == 2 ? KVD : 0);
                                    float* dst = sec == 1 ? ph.kc : ph.vc;
                                    dst[((size_t)(hrow / DH) * ph.cap + pos) * DH + e] = v;
                                    ll_st(ph.kv_ll + (sec == 2 ? KVD : 0) + hrow, v, ep);
                                }
                            }
                        } else if (ph.epi == HX_EPI_SWIGLU) {
                            // rows 0..63 of a tile are gate rows, 64..127 the matching up rows
                            S.swi[rl] = v * (rl < 64 ? ph.ts[0] : ph.ts[1]);
                            epi_sync();
                            const int hi = tile * 64 + rl;
                            if (rl < 64 && hi < ph.N) ll_st(ph.out_ll + hi, pz_silu_mul(S.swi[rl], S.swi[rl + 64]), ep);
                            epi_sync();
                        } else {
                            const int row = tile * 128 + rl;
                            const bool valid = row < ph.N;
                            v *= (row < ph.bound0) ? ph.ts[0] : (row < ph.bound1 ? ph.ts[1] : ph.ts[2]);
                            if (ph.epi == HX_EPI_RESID) {
                                if (TP && ph.tp_partial) {
                                    // row-split linear: this rank's partial row goes to every rank's exchange buffer, then the
                                    // ranks' rows are added in rank order -- the same bits on every rank
                                    const size_t o = ((size_t)(ph.tp_partial - 1) * P.tp_world) * P.tp_dm + row;
                                    if (valid) for (int w = 0; w < P.tp_world; w++)
                                        if (w != P.tp_rank) ll_st_sys(P.tp_x[w] + o + (size_t)P.tp_rank * P.tp_dm, v, ep);
                                    float sum = 0.0f;
                                    if (valid) for (int w = 0; w < P.tp_world; w++)
                                        sum += (w == P.tp_rank) ? v : df_wait1<true>(P.tp_x[P.tp_rank] + o + (size_t)w * P.tp_dm, ep, S, P);
                                    v = sum;
                                }
                                v = valid ? yres + v : 0.0f;
                                if (valid) ll_st(ph.out_ll + row, v, ep);
                                // this tile's share of the next norm's sum of squares
                                const float ssq = hx_warp_sum(v * v);
                                if (lane == 0) S.swi[warp] = ssq;
                                epi_sync();
                                if (rl == 0) ll_st(ph.out_stat + tile, (S.swi[0] + S.swi[1]) + (S.swi[2] + S.swi[3]), ep);
                                epi_sync();
                            } else if (valid) {
                                ph.y[row] = v;
                                if (ph.epi == HX_EPI_ARGMAX && pz_better(v, row, best_v, best_i)) { best_v = v; best_i = row; }
                            }
                        }
                    }
                } else uc += (uint32_t)(t_last - t_first + 1);
                if (ph.epi == HX_EPI_ARGMAX) {
                    // per-CTA best (held by warps 0-3), then the last CTA to arrive folds all of them
#pragma unroll
                    for (int d = 16; d >= 1; d >>= 1) {
                        const float ov = __shfl_xor_sync(0xffffffffu, best_v, d);
                        const int oi = __shfl_xor_sync(0xffffffffu, best_i, d);
                        if (pz_better(ov, oi, best_v, best_i)) { best_v = ov; best_i = oi; }
                    }
                    if (lane == 0) { S.bv[warp] = best_v; S.bi[warp] = best_i; }
                    consumer_sync();
                    if (tid == 0) {
                        float bv = S.bv[0]; int bi = S.bi[0];
                        for (int i = 1; i < 4; i++) if (pz_better(S.bv[i], S.bi[i], bv, bi)) { bv = S.bv[i]; bi = S.bi[i]; }
                        P.am_val[cta] = bv; P.am_idx[cta] = bi;
                        S.ticket = S.abort_flag ? 0u : ticket_acq_rel(P.am_cnt);       // an aborting CTA never finishes the token
                    }
                    consumer_sync();
                    if (S.ticket == (unsigned)grid - 1 && warp == 0) {
                        float bv = -INFINITY; int bi = INT_MAX;
                        for (int i = lane; i < grid; i += 32) {
                            const float ov = __ldcg(P.am_val + i); const int oi = __ldcg(P.am_idx + i);
                            if (pz_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
                        }
#pragma unroll
                        for (int d = 16; d >= 1; d >>= 1) {
                            const float ov = __shfl_xor_sync(0xffffffffu, bv, d);
                            const int oi = __shfl_xor_sync(0xffffffffu, bi, d);
                            if (pz_better(ov, oi, bv, bi)) { bv = ov; bi = oi; }
                        }
                        if (TP && lane == 0 && P.tp_world > 1) {
                            // vocabulary split over the ranks: exchange (value, global index) and take the best of all
                            const size_t ao = (size_t)2 * P.tp_world * P.tp_dm;
                            const int gi = bi == INT_MAX ? INT_MAX : bi + P.tp_vocab_off;
                            for (int w = 0; w < P.tp_world; w++) if (w != P.tp_rank) {
                                ll_st_sys(P.tp_x[w] + ao + 2 * P.tp_rank, bv, ep);
                                ll_st_sys(P.tp_x[w] + ao + 2 * P.tp_rank + 1, __int_as_float(gi), ep);
                            }
                            float fv = bv; int fi = gi;
                            for (int w = 0; w < P.tp_world; w++) if (w != P.tp_rank) {
                                const float ov = df_wait1<true>(P.tp_x[P.tp_rank] + ao + 2 * w, ep, S, P);
                                const int oi = __float_as_int(df_wait1<true>(P.tp_x[P.tp_rank] + ao + 2 * w + 1, ep, S, P));
                                if (pz_better(ov, oi, fv, fi)) { fv = ov; fi = oi; }
                            }
                            bv = fv; bi = fi;
                        }
                        if (lane == 0) {
                            const int nt = (bi == INT_MAX) ? 0 : bi;
                            *P.next_tok = nt;
                            *P.pos_inc = pos + 1;
                            if (P.hist) P.hist[pos + 1] = nt;
                            *P.am_cnt = 0u;
                        }
                    }
                }
            } else if (ph.type == HX_PH_ATTN) {
                switch (ph.NH / ph.NKV) {
                    case 1: attention_df<1>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    case 2: attention_df<2>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    case 3: attention_df<3>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    case 4: attention_df<4>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    case 5: attention_df<5>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    case 6: attention_df<6>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    case 7: attention_df<7>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                    default: attention_df<8>(P, ph, S, ring, digb, cslot, cpar, pi, pos); break;
                }
                // (scratch: the probabilities, free since the last barrier of the tiles)
                if (S.ap.active) attention_merge_df(P, ph, S, reinterpret_cast<float4*>(digb + (8 * 128 + 128 + 128) * 4), S.ap.kv, S.ap.split, S.att_ns, ph.NH / ph.NKV, ep);
            }
            DF_STAMP(2); DF_MARK(5);
            // ---------- phase boundary: the digit columns and the attention scratch are free again ----------
            asm volatile("cp.async.wait_all;" ::: "memory");
            if (consumer_sync_any(S.abort_flag)) goto aborted;
            DF_STAMP(3);
        }
        if (P.advance_pos && tid == 0) {
            // no lm_head in this launch: the last CTA to finish advances the position
            if (ticket_acq_rel(P.done_cnt) == (unsigned)grid - 1) { *P.pos_inc = pos + 1; *P.done_cnt = 0u; }
        }
        goto done;
aborted:
        if (tid == 0) { S.abort_flag = 1; *P.err = 1; }
done:   ;
    }
    // every role meets here; the MMA warp then releases the tensor memory
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == NCW + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "n"(TM_COLS) : "memory");
}

size_t df_smem_fixed(int bdig_bytes) {
    return ((sizeof(SmemDf) + 15) & ~(size_t)15) + 512 + 1024 + (size_t)bdig_bytes;      // + ring slots
}

}  // namespace

// Shared-memory scratch of the attention phase for a group of `grp` query heads per kv head (queries, the position's k
// and v, probabilities, partial outputs of the row subsets); the digit columns share the space.
int hx_decode_df_att_bytes(int grp) { return (8 * 128 + 128 + 128 + 8 * ATT_ROWS + NCT * 4 * grp) * 4; }

// Ring depth that fits beside the digit columns (0 = does not fit).
int hx_decode_df_ring(int bdig_bytes) {
    const size_t fixed = df_smem_fixed(bdig_bytes);
    if (fixed + 3 * (size_t)HX_RING_SLOT > 227 * 1024) return 0;
    size_t n = (227 * 1024 - fixed) / HX_RING_SLOT;
    return (int)(n > HX_TC_MAX_RING ? HX_TC_MAX_RING : n);
}

int hx_decode_df_prepare() {
    HX_CUDA(cudaFuncSetAttribute(k_decode_df<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    HX_CUDA(cudaFuncSetAttribute(k_decode_df<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
    return HX_OK;
}

int hx_decode_df_launch(const HxPersist& p, int grid, cudaStream_t st) {
    if (p.tc_ring < 3 || p.tc_ring > HX_TC_MAX_RING) return hx_fail(HX_ERR_ARG, "dataflow decode: ring depth %d", p.tc_ring);
    const size_t smem = df_smem_fixed(p.bdig_bytes) + (size_t)p.tc_ring * HX_RING_SLOT;
    if (smem > 227 * 1024) return hx_fail(HX_ERR_ARG, "dataflow decode needs %zu bytes of shared memory", smem);
    void* args[] = {(void*)&p};
    void* fn = p.tp_world > 1 ? (void*)k_decode_df<true> : (void*)k_decode_df<false>;
    HX_CUDA(cudaLaunchCooperativeKernel(fn, dim3(grid), dim3(PT), args, smem, st));
    HX_COUNT_LAUNCH(1);
    return HX_OK;
}
