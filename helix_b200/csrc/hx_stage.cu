// hx_stage.cu -- moving large pageable host buffers to and from the device.
//
// A cudaMemcpy from pageable memory stages through the driver on one thread (about 12 GB/s where the link does 50), and a
// call that allocates and frees its device buffers pays for mapping them each time.  Here up to eight threads copy slices of
// one megabyte between the caller's memory and page-locked slots, two per thread, while the link moves the slot before;
// slots, streams and a device workspace stay with the device for the next call.  They are bounded (16 MB page-locked, made per
// thread when a call first needs it; 256 MB of device memory; a larger workspace is freed when the call ends), handed to one
// call at a time, and the workspace is given back when device memory is short elsewhere in the library (hx_dev_malloc).  The
// threads live for one call: a call that needs one slice starts none.
#include "hx_stage.cuh"
#include <condition_variable>
#include <mutex>
#include <thread>
#include <vector>

namespace {
constexpr int ST_WORKERS = 8;
constexpr size_t ST_SLICE = 1u << 20;
constexpr size_t ST_KEEP = (size_t)256 << 20;
}

struct HxStageArea {
    std::mutex mu; std::condition_variable cv;
    bool busy = false;                                    // a call has the area (mu is held for moments only)
    int dev = -1;
    uint8_t* pinned[ST_WORKERS] = {};                     // two slots each
    cudaStream_t st = nullptr, wst[ST_WORKERS] = {};
    cudaEvent_t ev[ST_WORKERS][2] = {}, done[ST_WORKERS] = {}, mark = nullptr;
    void* work = nullptr; size_t work_bytes = 0;
    int prepare() {
        HX_CUDA(cudaGetDevice(&dev));
        if (!st) HX_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        if (!mark) HX_CUDA(cudaEventCreateWithFlags(&mark, cudaEventDisableTiming));
        return HX_OK;
    }
    int prepare_worker(int w) {
        if (!pinned[w]) HX_CUDA(cudaHostAlloc((void**)&pinned[w], 2 * ST_SLICE, cudaHostAllocDefault));
        if (!wst[w]) HX_CUDA(cudaStreamCreateWithFlags(&wst[w], cudaStreamNonBlocking));
        if (!done[w]) HX_CUDA(cudaEventCreateWithFlags(&done[w], cudaEventDisableTiming));
        for (int i = 0; i < 2; i++) if (!ev[w][i]) HX_CUDA(cudaEventCreateWithFlags(&ev[w][i], cudaEventDisableTiming));
        return HX_OK;
    }
};

static HxStageArea* areas() { static HxStageArea* a = new HxStageArea[64]; return a; }      // never destroyed: the driver outlives no destructor order

HxStage::HxStage() : a_(nullptr), rc_(HX_OK) {
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) { rc_ = hx_fail(HX_ERR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e)); return; }
    if (dev < 0 || dev >= 64) { rc_ = hx_fail(HX_ERR_ARG, "device index %d not supported", dev); return; }
    a_ = areas() + dev;
    {
        std::unique_lock<std::mutex> lk(a_->mu);
        a_->cv.wait(lk, [&] { return !a_->busy; });
        a_->busy = true;
    }
    rc_ = a_->prepare();
}

HxStage::~HxStage() {
    if (!a_) return;
    if (open_) {      // a call that failed: its copies must not meet the next call's in the slots or in the workspace
        for (cudaStream_t s : a_->wst) if (s) cudaStreamSynchronize(s);
        if (a_->st) cudaStreamSynchronize(a_->st);
    }
    if (big_ && a_->work) { cudaStreamSynchronize(a_->st); cudaFree(a_->work); a_->work = nullptr; a_->work_bytes = 0; }
    { std::lock_guard<std::mutex> lk(a_->mu); a_->busy = false; }
    a_->cv.notify_one();
}

cudaStream_t HxStage::stream() const { return a_->st; }

int HxStage::workspace(void** dptr, size_t bytes) {
    if (bytes > a_->work_bytes) {
        HX_CUDA(cudaStreamSynchronize(a_->st));
        if (a_->work) { cudaFree(a_->work); a_->work = nullptr; a_->work_bytes = 0; }
        const cudaError_t e = hx_dev_malloc(&a_->work, bytes);
        if (e != cudaSuccess) { a_->work = nullptr; return hx_fail(HX_ERR_CUDA, "cudaMalloc(%zu bytes): %s", bytes, cudaGetErrorString(e)); }
        a_->work_bytes = bytes;
    }
    big_ = a_->work_bytes > ST_KEEP;
    *dptr = a_->work;
    return HX_OK;
}

int HxStage::run(const HxCopy* c, int n, bool up) {
    HxStageArea& A = *a_;
    struct Slice { uint8_t *dev, *host; size_t bytes; };
    auto slices_of = [](const HxCopy& x) { return (x.bytes + ST_SLICE - 1) / ST_SLICE; };
    size_t nsl = 0;
    for (int i = 0; i < n; i++) nsl += slices_of(c[i]);
    if (!nsl) return HX_OK;
    auto slice = [&](size_t k) {
        int i = 0;
        while (k >= slices_of(c[i])) k -= slices_of(c[i++]);
        const size_t o = k * ST_SLICE, left = c[i].bytes - o;
        return Slice{(uint8_t*)c[i].dev + o, (uint8_t*)c[i].host + o, left < ST_SLICE ? left : ST_SLICE};
    };
    open_ = true;
    std::atomic<size_t> next{0};
    std::atomic<int> err{0};
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(A.dev);
        uint8_t* slot[2] = {A.pinned[w], A.pinned[w] + ST_SLICE};
        Slice held[2]; bool full[2] = {false, false};
        auto finish = [&](int s) {                        // the slot's copy over the link is done; a download goes on to the caller's memory
            if (!full[s]) return;
            full[s] = false;
            if (e == cudaSuccess) e = cudaEventSynchronize(A.ev[w][s]);
            if (e == cudaSuccess && !up) memcpy(held[s].host, slot[s], held[s].bytes);
        };
        for (int s = 0; e == cudaSuccess && !err.load(std::memory_order_relaxed); s ^= 1) {
            const size_t i = next.fetch_add(1);
            if (i >= nsl) break;
            finish(s);
            if (e != cudaSuccess) break;
            held[s] = slice(i);
            if (up) {
                memcpy(slot[s], held[s].host, held[s].bytes);
                e = cudaMemcpyAsync(held[s].dev, slot[s], held[s].bytes, cudaMemcpyHostToDevice, A.wst[w]);
            } else e = cudaMemcpyAsync(slot[s], held[s].dev, held[s].bytes, cudaMemcpyDeviceToHost, A.wst[w]);
            if (e == cudaSuccess) { e = cudaEventRecord(A.ev[w][s], A.wst[w]); full[s] = e == cudaSuccess; }
        }
        if (up) { if (e == cudaSuccess) e = cudaEventRecord(A.done[w], A.wst[w]); }
        else { finish(0); finish(1); }
        if (e != cudaSuccess) { int z = 0; err.compare_exchange_strong(z, (int)e); }
    };
    size_t nw = std::thread::hardware_concurrency() / 2;
    if (nw > ST_WORKERS) nw = ST_WORKERS;
    if (nw > (nsl + 1) / 2) nw = (nsl + 1) / 2;      // two slices are worth a thread
    if (nw < 1) nw = 1;
    for (size_t w = 0; w < nw; w++) {
        const int rc = A.prepare_worker((int)w);
        if (rc && w == 0) return rc;
        if (rc) nw = w;                              // page-locked memory is short: the others take its slices
    }
    // downloads follow what stream() has been given so far, uploads what it still reads from the workspace
    HX_CUDA(cudaEventRecord(A.mark, A.st));
    for (size_t w = 0; w < nw; w++) HX_CUDA(cudaStreamWaitEvent(A.wst[w], A.mark, 0));
    std::vector<std::thread> th;
    size_t started = 1;
    try { for (; started < nw; started++) th.emplace_back(work, (int)started); } catch (...) { }      // fewer threads: the others take their slices
    work(0);
    for (auto& t : th) t.join();
    if (err.load()) return hx_fail(HX_ERR_CUDA, "host copy: %s", cudaGetErrorString((cudaError_t)err.load()));
    if (up) for (size_t w = 0; w < started; w++) HX_CUDA(cudaStreamWaitEvent(A.st, A.done[w], 0));
    else open_ = false;                                   // (downloads have been waited for, and they follow all that came before)
    return HX_OK;
}

int HxStage::upload(const HxCopy* c, int n) { return run(c, n, true); }
int HxStage::download(const HxCopy* c, int n) { return run(c, n, false); }

cudaError_t hx_dev_malloc(void** p, size_t bytes) {
    cudaError_t e = cudaMalloc(p, bytes);
    int dev = 0;
    if (e != cudaSuccess) (void)cudaGetLastError();       // no error stays behind: the caller reports it
    if (e == cudaErrorMemoryAllocation && cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        HxStageArea& A = areas()[dev];
        std::lock_guard<std::mutex> lk(A.mu);             // (a call that has the area keeps its workspace)
        if (!A.busy && A.work) { cudaFree(A.work); A.work = nullptr; A.work_bytes = 0; e = cudaMalloc(p, bytes); }
        if (e != cudaSuccess) (void)cudaGetLastError();
    }
    return e;
}
