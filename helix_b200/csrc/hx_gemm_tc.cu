// hx_gemm_tc.cu -- block-scaled NVFP4 GEMM on the 5th-generation tensor cores (tcgen05, TMEM), raw form.
//
//   D[row, n] = sum_k  A[row,k] * SFA[row,k/16]  *  B[n,k] * SFB[n,k/16]         (f32 accumulate in TMEM)
//
// A = weights, E2M1 codes with one UE4M3 scale per 16 elements along K: exactly the information of
// the committed NVFP4 layout (helixc/runtime/gpt2_pack.c:350-373), so the weights feed the tensor
// cores without any per-weight instruction.  B = any E2M1 columns with their own UE4M3 block scales.
//
// A CTA per SM walks through 128-row tiles of A.  Warp 0 streams A and B cells into a shared-memory ring with
// cp.async.bulk; warp 1 copies the scale factors to TMEM (tcgen05.cp) and issues
// tcgen05.mma.kind::mxf4nvf4.block_scale (M=128, N=ncols, K=64 per instruction); warps 2-13 read the
// accumulator with tcgen05.ld and store it.
//
// "T128" layout of A: per (128-row tile, group of 256 columns = four MMA K steps) one 18432-byte cell:
// 128 rows x 128 bytes of codes in the canonical K-major 128-byte-swizzle operand layout (row r at
// r*128, its 16-byte chunk j stored at position j ^ (r & 7)), then four 512-byte scale chunks, one per
// K step (byte (row%32)*16 + (row/32)*4 + block).  B cells: N rows x 128 swizzled bytes + four scale
// chunks indexed by n.  The cells are the shared-memory image, so plain bulk copies load them; the
// 128-byte swizzle lets the tensor core fetch operands at full shared-memory width (the unswizzled
// layout measured 8x slower per instruction).  Every wait is bounded.
#include "hx_tc.cuh"
#include "hx_gemm_tc.cuh"

using namespace hxtc;

namespace {

struct TcSmem {
    uint64_t full[HX_TC_STAGES], empty[HX_TC_STAGES], accum, acc_free;
    uint32_t tmem_base;
    volatile int abort_flag;
};
#define TC_EPI_Q 3              // epilogue warps per quarter of the TMEM lanes: each takes every third group of eight columns
#define TC_THREADS ((2 + 4 * TC_EPI_Q) * 32)
#define TC_HDR 1024u

__global__ void __launch_bounds__(TC_THREADS, 1) k_gemm_tc(const __grid_constant__ HxGemmTC g) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    TcSmem& S = *reinterpret_cast<TcSmem*>(smem_raw);
    // swizzled operands need 1024-byte aligned cells (the swizzle is a function of the shared-memory address)
    uint8_t* ring = smem_raw + (((s_u32(smem_raw) + TC_HDR + 1023u) & ~1023u) - s_u32(smem_raw));
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int Sk = g.stage_ksteps, NB = g.ncols;
    const uint32_t b_cell_bytes = (uint32_t)NB * 128u + 2048u;                    // one 256-column cell of B
    const uint32_t a_cell = HX_T128_CELL / 4, b_cell = b_cell_bytes / 4;          // bytes per K step
    const uint32_t stage_bytes = (uint32_t)Sk * (a_cell + b_cell);

    if (tid == 0) {
        for (int i = 0; i < HX_TC_STAGES; i++) { mb_init(&S.full[i], 1); mb_init(&S.empty[i], 1); }
        mb_init(&S.accum, 1); mb_init(&S.acc_free, 4 * TC_EPI_Q);
        S.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {    // one warp owns the TMEM allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" :: "r"(s_u32(&S.tmem_base)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = S.tmem_base;
    // TMEM columns: [0, 256) accumulator, then per ring slot Sk*4 columns of SFA and of SFB
    const uint32_t col_sfa = 256u, col_sfb = 256u + HX_TC_STAGES * HX_TC_MAX_SK * 4;

    if (warp == 0) {
        // ------------------------------ loader ------------------------------
        if (lane == 0) {
            uint32_t git = 0;
            bool ok = true;
            for (int mt = blockIdx.x; mt < g.ntiles && ok; mt += gridDim.x) {
                for (int ks0 = 0; ks0 < g.ksteps; ks0 += Sk, git++) {
                    const uint32_t slot = git % HX_TC_STAGES, round = git / HX_TC_STAGES;
                    if (round > 0 && !mb_wait(&S.empty[slot], (round - 1) & 1, &S.abort_flag)) { ok = false; break; }
                    const int nk = min(Sk, g.ksteps - ks0);
                    uint8_t* sa = ring + (size_t)slot * stage_bytes;
                    mb_expect(&S.full[slot], (uint32_t)nk * (a_cell + b_cell));
                    bulk_load(sa, g.a + ((size_t)mt * g.ksteps + ks0) * a_cell, (uint32_t)nk * a_cell, &S.full[slot]);
                    bulk_load(sa + (size_t)Sk * a_cell, g.b + (size_t)ks0 * b_cell, (uint32_t)nk * b_cell, &S.full[slot]);
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer ------------------------------
        // instruction descriptor: E2M1 x E2M1, UE4M3 scales, K-major both, N = NB, M = 128, K = 64
        const uint32_t idesc = (1u << 7) | (1u << 10) | ((uint32_t)(NB >> 3) << 17) | (8u << 24);
        uint32_t git = 0;
        bool ok = true;
        int unit_iter = 0;
        for (int mt = blockIdx.x; mt < g.ntiles && ok; mt += gridDim.x, unit_iter++) {
            if (unit_iter > 0) {      // the epilogue has read the previous unit's accumulator out
                if (!warp_wait(&S.acc_free, (uint32_t)(unit_iter - 1) & 1u, &S.abort_flag)) break;
                tc_fence_after();
            }
            for (int ks0 = 0; ks0 < g.ksteps; ks0 += Sk, git++) {
                const uint32_t slot = git % HX_TC_STAGES, round = git / HX_TC_STAGES;
                if (!warp_wait(&S.full[slot], round & 1, &S.abort_flag)) { ok = false; break; }
                tc_fence_after();
                const int nk = min(Sk, g.ksteps - ks0);
                const uint32_t sa = s_u32(ring + (size_t)slot * stage_bytes);
                const uint32_t sb = sa + (uint32_t)Sk * a_cell;
                if (tc_elect()) {
                    for (int k = 0; k < nk; k++) {
                        const uint32_t ta = tmem + col_sfa + (slot * HX_TC_MAX_SK + k) * 4;
                        const uint32_t tb = tmem + col_sfb + (slot * HX_TC_MAX_SK + k) * 4;
                        const uint32_t acell = sa + (uint32_t)(k >> 2) * HX_T128_CELL, bcell = sb + (uint32_t)(k >> 2) * b_cell_bytes;
                        const uint32_t e = (uint32_t)(k & 3);
                        tc_cp_sf(ta, smem_desc(acell + 16384 + e * 512, 16, 128));
                        tc_cp_sf(tb, smem_desc(bcell + (uint32_t)NB * 128u + e * 512, 16, 128));
                        tc_mma(tmem, smem_desc(acell + e * 32, 16, 1024, SW128), smem_desc(bcell + e * 32, 16, 1024, SW128), idesc,
                               ta, tb, (ks0 > 0 || k > 0) ? 1u : 0u);
                    }
                    tc_commit(&S.empty[slot]);          // the slot is free once these MMAs have read it
                }
                __syncwarp();
            }
            if (ok && tc_elect()) tc_commit(&S.accum);         // accumulator complete
            __syncwarp();
        }
    } else {
        // ------------------------------ epilogue: TMEM -> registers -> global ------------------------------
        const int ew = warp - 2, sub = warp & 3, third = ew >> 2;      // TMEM lanes 32*sub .. 32*sub+31
        int unit_iter = 0;
        for (int mt = blockIdx.x; mt < g.ntiles; mt += gridDim.x, unit_iter++) {
            if (!warp_wait(&S.accum, (uint32_t)unit_iter & 1u, &S.abort_flag)) break;
            tc_fence_after();
            const int row = mt * 128 + sub * 32 + lane;
            const uint32_t tlane = tmem + ((uint32_t)(sub * 32) << 16);
            for (int c0 = third * 8; c0 < NB; c0 += 8 * TC_EPI_Q) {
                uint32_t r[8];
                tc_ld8(r, tlane + (uint32_t)c0);
                tc_wait_ld();
                if (row < g.rows) {
#pragma unroll
                    for (int j = 0; j < 8; j++) g.y[(size_t)row * NB + c0 + j] = __uint_as_float(r[j]);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mb_arrive(&S.acc_free);
        }
    }
    __syncthreads();
    if (S.abort_flag && tid == 0 && g.err) *g.err = 1;
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
    }
}

}  // namespace

#define TC_FRONT (TC_HDR + 1024u)      // header and the slack of the 1024-byte alignment of the ring
size_t hx_gemm_tc_smem(int ncols, int stage_ksteps) {
    return TC_FRONT + (size_t)HX_TC_STAGES * (stage_ksteps / 4) * (HX_T128_CELL + (size_t)ncols * 128 + 2048);
}
int hx_gemm_tc_launch(const HxGemmTC& g, cudaStream_t st) {
    HX_CHECK_ARG(g.a && g.b && g.y && g.ntiles > 0 && g.ksteps > 0);
    HX_CHECK_ARG(g.stage_ksteps >= 4 && g.stage_ksteps <= HX_TC_MAX_SK && g.stage_ksteps % 4 == 0 && g.ksteps % 4 == 0);
    HX_CHECK_ARG(g.ncols >= 8 && g.ncols <= 256 && g.ncols % 8 == 0);
    const size_t smem = hx_gemm_tc_smem(g.ncols, g.stage_ksteps);
    if (smem > 227 * 1024) return hx_fail(HX_ERR_ARG, "tensor-core GEMM stage too large (%zu bytes of shared memory)", smem);
    static HxOncePerDevice once;
    const int rc = hx_max_smem(once, k_gemm_tc, 227 * 1024); if (rc) return rc;
    k_gemm_tc<<<g.ntiles < 148 ? g.ntiles : 148, TC_THREADS, smem, st>>>(g);
    HX_COUNT_LAUNCH(1);
    HX_CUDA(cudaGetLastError());
    return HX_OK;
}

// C-ABI entry for tests and tools: all pointers are device pointers.
HX_API int hx_gemm_nvfp4_tc(const uint8_t* a_t128, int rows, int K, const uint8_t* b_cells, int ncols, float* y,
                            int stage_ksteps, void* stream) {
    HX_CHECK_ARG(rows > 0 && K > 0 && K % 256 == 0);
    HxGemmTC g = {};
    g.a = a_t128; g.b = b_cells; g.y = y; g.rows = rows; g.ntiles = (rows + 127) / 128; g.ksteps = K / 64;
    g.ncols = ncols; g.stage_ksteps = stage_ksteps > 0 ? stage_ksteps : 4;
    int* derr = nullptr;
    HX_CUDA(cudaMalloc(&derr, 4));
    HX_CUDA(cudaMemsetAsync(derr, 0, 4, (cudaStream_t)stream));
    g.err = derr;
    int rc = hx_gemm_tc_launch(g, (cudaStream_t)stream);
    int e = 0;
    if (!rc) {
        cudaError_t ce = cudaStreamSynchronize((cudaStream_t)stream);
        if (ce != cudaSuccess) rc = hx_fail(HX_ERR_CUDA, "tensor-core GEMM: %s", cudaGetErrorString(ce));
        else { cudaMemcpy(&e, derr, 4, cudaMemcpyDeviceToHost); if (e) rc = hx_fail(HX_ERR_TIMEOUT, "tensor-core GEMM: a bounded wait ran out"); }
    }
    cudaFree(derr);
    return rc;
}

// Timing helper: `reps` back-to-back launches between two CUDA events (device pointers as above).
HX_API int hx_gemm_nvfp4_tc_bench(const uint8_t* a_t128, int rows, int K, const uint8_t* b_cells, int ncols, float* y,
                                  int stage_ksteps, int reps, float* ms_per_launch) {
    HX_CHECK_ARG(rows > 0 && K > 0 && K % 256 == 0 && reps > 0 && ms_per_launch);
    HxGemmTC g = {};
    g.a = a_t128; g.b = b_cells; g.y = y; g.rows = rows; g.ntiles = (rows + 127) / 128; g.ksteps = K / 64;
    g.ncols = ncols; g.stage_ksteps = stage_ksteps > 0 ? stage_ksteps : 4;
    int* derr = nullptr;
    HX_CUDA(cudaMalloc(&derr, 4));
    HX_CUDA(cudaMemset(derr, 0, 4));
    g.err = derr;
    cudaEvent_t e0, e1;
    HX_CUDA(cudaEventCreate(&e0)); HX_CUDA(cudaEventCreate(&e1));
    int rc = hx_gemm_tc_launch(g, nullptr);
    if (!rc) {
        cudaEventRecord(e0, nullptr);
        for (int i = 0; i < reps && !rc; i++) rc = hx_gemm_tc_launch(g, nullptr);
        cudaEventRecord(e1, nullptr);
        cudaError_t ce = cudaEventSynchronize(e1);
        if (ce != cudaSuccess) rc = hx_fail(HX_ERR_CUDA, "tensor-core GEMM: %s", cudaGetErrorString(ce));
        else { float t = 0; cudaEventElapsedTime(&t, e0, e1); *ms_per_launch = t / reps; }
    }
    int e = 0; cudaMemcpy(&e, derr, 4, cudaMemcpyDeviceToHost);
    if (!rc && e) rc = hx_fail(HX_ERR_TIMEOUT, "tensor-core GEMM: a bounded wait ran out");
    cudaEventDestroy(e0); cudaEventDestroy(e1); cudaFree(derr);
    return rc;
}
