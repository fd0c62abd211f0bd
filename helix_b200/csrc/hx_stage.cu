// hx_stage.cu -- moving large pageable host buffers to and from the device.
//
// A cudaMemcpy from pageable memory stages through the driver on one thread (about 12 GB/s where the link does 50), and a
// call that allocates and frees its device buffers pays for mapping them each time.  Here up to eight threads copy slices of
// one megabyte between the caller's memory and page-locked slots, two per thread, while the link moves the slot before;
// slots, streams and a device workspace stay with the device for the next call.  They are bounded (16 MB page-locked, 256 MB
// of device memory; a larger workspace is freed when the call ends), handed to one call at a time, and the workspace is
// given back when device memory is short elsewhere in the library (hx_dev_malloc).  The threads live for one call: a call that needs one slice starts none.
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
    bool ready = false;
    uint8_t* pinned = nullptr;                            // [worker][2] slots
    cudaStream_t st = nullptr, wst[ST_WORKERS] = {};
    cudaEvent_t ev[ST_WORKERS][2] = {}, done[ST_WORKERS] = {}, mark = nullptr;
    void* work = nullptr; size_t work_bytes = 0;
    int prepare() {
        if (ready) return HX_OK;
        HX_CUDA(cudaGetDevice(&dev));
        if (!pinned) HX_CUDA(cudaHostAlloc((void**)&pinned, ST_WORKERS * 2 * ST_SLICE, cudaHostAllocDefault));
        if (!st) HX_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        if (!mark) HX_CUDA(cudaEventCreateWithFlags(&mark, cudaEventDisableTiming));
        for (int w = 0; w < ST_WORKERS; w++) {
            if (!wst[w]) HX_CUDA(cudaStreamCreateWithFlags(&wst[w], cudaStreamNonBlocking));
            if (!done[w]) HX_CUDA(cudaEventCreateWithFlags(&done[w], cudaEventDisableTiming));
            for (int i = 0; i < 2; i++) if (!ev[w][i]) HX_CUDA(cudaEventCreateWithFlags(&ev[w][i], cudaEventDisableTiming));
        }
        ready = true;
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
    std::vector<Slice> sl;
    for (int i = 0; i < n; i++)
        for (size_t o = 0; o < c[i].bytes; o += ST_SLICE)
            sl.push_back({(uint8_t*)c[i].dev + o, (uint8_t*)c[i].host + o, c[i].bytes - o < ST_SLICE ? c[i].bytes - o : ST_SLICE});
    if (sl.empty()) return HX_OK;
    std::atomic<size_t> next{0};
    std::atomic<int> err{0};
    auto work = [&](int w) {
        cudaError_t e = cudaSetDevice(A.dev);
        uint8_t* slot[2] = {A.pinned + (size_t)(2 * w) * ST_SLICE, A.pinned + (size_t)(2 * w + 1) * ST_SLICE};
        Slice held[2]; bool full[2] = {false, false};
        auto finish = [&](int s) {                        // the slot's copy over the link is done; a download goes on to the caller's memory
            if (!full[s]) return;
            full[s] = false;
            if (e == cudaSuccess) e = cudaEventSynchronize(A.ev[w][s]);
            if (e == cudaSuccess && !up) memcpy(held[s].host, slot[s], held[s].bytes);
        };
        for (int s = 0; e == cudaSuccess && !err.load(std::memory_order_relaxed); s ^= 1) {
            const size_t i = next.fetch_add(1);
            if (i >= sl.size()) break;
            finish(s);
            if (e != cudaSuccess) break;
            held[s] = sl[i];
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
    if (nw > (sl.size() + 1) / 2) nw = (sl.size() + 1) / 2;      // two slices are worth a thread
    if (nw < 1) nw = 1;
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
