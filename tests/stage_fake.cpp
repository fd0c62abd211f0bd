// hx_stage.cu on the host, over a CUDA runtime of its own: device memory is host memory, and a copy given to a stream is done no
// earlier than something waits for that stream (or for a later event of it).  Exit code 0: every check held.
#include "../helix_b200/csrc/hx_stage.cu"
#include <deque>
#include <map>
#include <stdarg.h>
#include <stdio.h>
#include <stdlib.h>

unsigned long long g_hx_launches = 0;
int hx_fail(int code, const char*, ...) { return code; }

namespace {
struct Op { void* dst; const void* src; size_t n; cudaEvent_t mark, after; };
struct Stream { std::deque<Op> q; };
struct Event { int recorded = 0, reached = 0; Stream* on = nullptr; };
std::recursive_mutex mu;
std::vector<Stream*> streams;
size_t pinned_bytes = 0, live = 0, room = ~(size_t)0;
std::map<void*, size_t> blocks;

void run_until(Stream* s, Event* e) {      // everything of s, or up to the record of e that has been asked for
    while (!s->q.empty()) {
        Op o = s->q.front(); s->q.pop_front();
        if (o.after) { Event* a = (Event*)o.after; if (a->on && a->reached < a->recorded) run_until(a->on, a); }
        if (o.n) memcpy(o.dst, o.src, o.n);
        if (o.mark) { Event* m = (Event*)o.mark; m->reached++; if (m == e && e->reached == e->recorded) return; }
    }
}
size_t in_flight() { size_t n = 0; for (Stream* s : streams) for (auto& o : s->q) n += o.n != 0; return n; }
}

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = malloc(n); std::lock_guard<std::recursive_mutex> l(mu); pinned_bytes += n; return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (live + n > room) return cudaErrorMemoryAllocation;
    *p = malloc(n); blocks[*p] = n; live += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) { std::lock_guard<std::recursive_mutex> l(mu); if (p) { live -= blocks[p]; blocks.erase(p); free(p); } return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { std::lock_guard<std::recursive_mutex> l(mu); streams.push_back(new Stream()); *s = (cudaStream_t)streams.back(); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t) new Event(); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) { std::lock_guard<std::recursive_mutex> l(mu); ((Stream*)st)->q.push_back({d, s, n, nullptr, nullptr}); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) { std::lock_guard<std::recursive_mutex> l(mu); ((Event*)e)->recorded++; ((Event*)e)->on = (Stream*)st; ((Stream*)st)->q.push_back({nullptr, nullptr, 0, e, nullptr}); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) { std::lock_guard<std::recursive_mutex> l(mu); ((Stream*)st)->q.push_back({nullptr, nullptr, 0, nullptr, e}); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { std::lock_guard<std::recursive_mutex> l(mu); Event* v = (Event*)e; if (v->on && v->reached < v->recorded) run_until(v->on, v); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { std::lock_guard<std::recursive_mutex> l(mu); if (s) run_until((Stream*)s, nullptr); return cudaSuccess; }
}

#define CHECK(x) do { if (!(x)) { printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main() {
    // a small call page-locks what one thread needs
    std::vector<uint8_t> a(1000, 1), b(1000, 0);
    {
        HxStage s; void* d = nullptr;
        CHECK(!s.status() && !s.workspace(&d, 1000));
        HxCopy c = {d, a.data(), 1000}, e = {d, b.data(), 1000};
        CHECK(!s.upload(&c, 1) && !s.download(&e, 1));
        CHECK(b == a && pinned_bytes <= (size_t)2 << 20);
    }
    // several copies, slices of a megabyte that do not divide them
    const size_t n0 = (5u << 20) + 17, n1 = 3;
    std::vector<uint8_t> x(n0), y(n1), u(n0), v(n1);
    for (size_t i = 0; i < n0; i++) x[i] = (uint8_t)(i * 7 + i / 1000);
    for (size_t i = 0; i < n1; i++) y[i] = (uint8_t)(i + 1);
    {
        HxStage s; void* d = nullptr;
        CHECK(!s.workspace(&d, n0 + 256));
        HxCopy in[2] = {{d, x.data(), n0}, {(uint8_t*)d + n0, y.data(), n1}}, out[2] = {{(uint8_t*)d + n0, v.data(), n1}, {d, u.data(), n0}};
        CHECK(!s.upload(in, 2) && !s.download(out, 2));
        CHECK(u == x && v == y && in_flight() == 0);
    }
    // a call that ends between its upload and its download leaves nothing in flight
    {
        HxStage s; void* d = nullptr;
        CHECK(!s.workspace(&d, n0));
        HxCopy in = {d, x.data(), n0};
        CHECK(!s.upload(&in, 1));
    }
    CHECK(in_flight() == 0);
    // the idle workspace is given back to an allocation that needs it, the workspace of a call is not
    room = live + 100;
    void* p = nullptr;
    { HxStage s; CHECK(hx_dev_malloc(&p, 4 << 20) == cudaErrorMemoryAllocation); }
    CHECK(hx_dev_malloc(&p, 4 << 20) == cudaSuccess);
    printf("ok\n");
    return 0;
}
