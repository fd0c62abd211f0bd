// hx_common.cuh -- shared declarations of libhelix_b200: error plumbing, the NVFP4 codecs
// (host + device) and small device helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <math.h>
#include "../../include/helix_b200.h"

#define HX_API extern "C" __attribute__((visibility("default")))

// ---- error plumbing -----------------------------------------------------------------------------
void hx_set_error(const char* fmt, ...);
int  hx_fail(int code, const char* fmt, ...);

#define HX_CUDA(call)                                                                         \
    do {                                                                                      \
        cudaError_t _e = (call);                                                              \
        if (_e != cudaSuccess) {                                                              \
            (void)cudaGetLastError();   /* reported here, not by the next call's launch check */ \
            return hx_fail(HX_ERR_CUDA, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_e), \
                           __FILE__, __LINE__);                                               \
        }                                                                                     \
    } while (0)

#define HX_CHECK_ARG(cond)                                                                    \
    do {                                                                                      \
        if (!(cond)) return hx_fail(HX_ERR_ARG, "bad argument: %s (%s:%d)", #cond, __FILE__, __LINE__); \
    } while (0)

// A function attribute belongs to the device that is current when it is set, so "done once" is tracked per device (the first 64; on
// others it is set every time).  A caller that comes while another thread is setting waits for it; what failed is tried again.
#include <atomic>
#include <mutex>
struct HxOncePerDevice {
    std::atomic<unsigned long long> done{0};
    std::mutex mu;
    template <class Set> int operator()(Set&& set) {
        int dev = 0;
        HX_CUDA(cudaGetDevice(&dev));
        const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0;
        if (done.load(std::memory_order_acquire) & bit) return HX_OK;
        std::lock_guard<std::mutex> lock(mu);
        if (done.load(std::memory_order_relaxed) & bit) return HX_OK;
        const int rc = set();
        if (!rc) done.fetch_or(bit, std::memory_order_release);
        return rc;
    }
};
#ifdef __CUDACC__
template <class Kernel> static int hx_max_smem(HxOncePerDevice& once, Kernel kernel, int bytes) {
    return once([&]() -> int { HX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes)); return HX_OK; });
}
#endif

// Count of kernels this library launched (reported by the benchmark as gpu_launches).
extern unsigned long long g_hx_launches;
#define HX_COUNT_LAUNCH(n) (g_hx_launches += (n))

// ---- codecs -------------------------------------------------------------------------------------
// E2M1 magnitudes {0,.5,1,1.5,2,3,4,6}: as_float(mag3 << 22) is mag * 2^-126 (the e=0 codes land on
// f32 subnormals), so one exact multiply by 2^126 decodes all eight without a table.
__host__ __device__ __forceinline__ float hx_e2m1_mag(int c3) {
#ifdef __CUDA_ARCH__
    return __uint_as_float((unsigned)(c3 & 7) << 22) * 8.507059173023462e37f;   // 2^126
#else
    const float MAG[8] = {0.0f, 0.5f, 1.0f, 1.5f, 2.0f, 3.0f, 4.0f, 6.0f};
    return MAG[c3 & 7];
#endif
}
__host__ __device__ __forceinline__ float hx_e2m1_dec(int code) {
    float m = hx_e2m1_mag(code);
    return (code & 8) ? -m : m;
}

// Threshold encoder; a tie takes the smaller magnitude, magnitude 0 never carries a sign, NaN maps
// to code 7 (every comparison false).  Reference: e2m1_encode, gpt2_pack.c:306-318.
__host__ __device__ __forceinline__ int hx_e2m1_enc(float v) {
    float a = v < 0.0f ? -v : v;
    if (a <= 0.25f) return 0;
    int mag = 1 + (int)!(a <= 0.75f) + (int)!(a <= 1.25f) + (int)!(a <= 1.75f) + (int)!(a <= 2.5f) +
              (int)!(a <= 3.5f) + (int)!(a <= 5.0f);
    return mag | (v < 0.0f ? 8 : 0);
}

// E4M3 decode for non-NaN codes: (1+m/8)*2^(e-7), subnormals (m/8)*2^-6.  Built from the bit
// pattern: as_float((c & 0x7F) << 20) is the value times 2^-120 (e=0 lands on f32 subnormals).
// Reference: e4m3_decode, gpt2_pack.c:333-338.
__host__ __device__ __forceinline__ float hx_e4m3_dec(int c) {
    if ((c & 0x7F) == 0x7F) {
#ifdef __CUDA_ARCH__
        return __uint_as_float(0x7FC00000u);
#else
        return nanf("");
#endif
    }
    uint32_t bits = (uint32_t)(c & 0x7F) << 20;
    float mag;
#ifdef __CUDA_ARCH__
    mag = __uint_as_float(bits) * 1.329227995784916e36f;   // 2^120, exact
#else
    float f; memcpy(&f, &bits, 4); mag = f * 1.329227995784916e36f;
#endif
    return (c & 0x80) ? -mag : mag;
}

// E4M3 encode of v with the reference's semantics: the nearest of the 254 non-NaN codes by
// |decode(c) - v| evaluated in f32, the first (lowest) code on a tie, code 0 when no distance is
// below 1e30.  For 0 <= v <= 512 (everything the quantizer can produce: the ratio never exceeds
// 448 by more than rounding) the winner is found in closed form: values are monotonic in the code
// and the distances to the two neighbours are exact (Sterbenz), so the rule is "round to nearest, a
// tie goes to the lower code".  Outside that range f32 rounding of the distances themselves creates
// ties between far-apart codes, so the search is run as written.
// Reference: e4m3_encode, gpt2_pack.c:339-343.
__host__ __device__ __forceinline__ int hx_e4m3_enc_search(float v) {
    int best = 0; float bd = 1.0e30f;
    for (int c = 0; c < 256; c++) {
        if ((c & 0x7F) == 0x7F) continue;
        float d = hx_e4m3_dec(c) - v; if (d < 0) d = -d;
        if (d < bd) { bd = d; best = c; }
    }
    return best;
}
__host__ __device__ __forceinline__ int hx_e4m3_enc(float v) {
    if (!(v >= 0.0f && v <= 512.0f)) return hx_e4m3_enc_search(v);   // negative, huge or NaN: rare
    if (v >= 448.0f) return 0x7E;
    if (v < 0.015625f) {                           // below 2^-6: subnormal codes, step 2^-9
        const float t = v * 512.0f;                // exact
        const int k = (int)t;
        return k + ((t - (float)k) > 0.5f ? 1 : 0);   // 8 rolls into code 0x08 = 2^-6
    }
    uint32_t bits;
#ifdef __CUDA_ARCH__
    bits = __float_as_uint(v);
#else
    memcpy(&bits, &v, 4);
#endif
    const int e = (int)(bits >> 23) - 127 + 7;     // 1..15
    const uint32_t man = bits & 0x7FFFFFu;
    int c = (e << 3) | (int)(man >> 20);
    if ((man & 0xFFFFFu) > 0x80000u) c += 1;       // above the midpoint; carries into the exponent
    return c > 0x7E ? 0x7E : c;
}

// ---- device helpers -----------------------------------------------------------------------------
#ifdef __CUDACC__
// ---- two f32 in one instruction, each rounded as by itself ----
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 x2(float a, float b) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(a), "f"(b)); return d; }
__device__ __forceinline__ f32x2 x2(uint32_t a, uint32_t b) { f32x2 d; asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(a), "r"(b)); return d; }
__device__ __forceinline__ float x2_lo(f32x2 a) { return __uint_as_float((uint32_t)a); }
__device__ __forceinline__ float x2_hi(f32x2 a) { return __uint_as_float((uint32_t)(a >> 32)); }
__device__ __forceinline__ f32x2 x2_fma(f32x2 a, f32x2 b, f32x2 c) { f32x2 d; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c)); return d; }
__device__ __forceinline__ f32x2 x2_mul(f32x2 a, f32x2 b) { f32x2 d; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }
__device__ __forceinline__ f32x2 x2_add(f32x2 a, f32x2 b) { f32x2 d; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b)); return d; }

__device__ __forceinline__ float hx_warp_sum(float v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    return v;
}
__device__ __forceinline__ float hx_warp_max(float v) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
    return v;
}
#define HX_TC_WAIT_NS 2000000000u        // limit of a device-side wait that is bounded by time

// Programmatic dependent launch: wait for the kernels this one depends on / let dependents start.
__device__ __forceinline__ void hx_grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void hx_grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with programmatic stream serialization: the kernel may start while the one before it in the stream drains, and
// calls hx_grid_dep_wait() before it touches anything that an earlier kernel writes or reads.  Every kernel launched this
// way waits in at least one CTA before it ends -- otherwise it could complete ahead of its predecessor, and the wait of its
// successor would not cover that one.
template <class... KArgs, class... Args>
static inline cudaError_t hx_launch_pdl(void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization; at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k, KArgs(args)...);
}
#endif
