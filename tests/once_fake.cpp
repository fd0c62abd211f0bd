// HxOncePerDevice (hx_common.cuh) on the host, over a runtime that knows two devices.  Exit code 0: every check held.
#include "../helix_b200/csrc/hx_common.cuh"
#include <chrono>
#include <stdio.h>
#include <thread>
#include <vector>

unsigned long long g_hx_launches = 0;
int hx_fail(int code, const char*, ...) { return code; }
static thread_local int device = 0;
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

int main() {
    HxOncePerDevice once;
    std::atomic<int> calls{0}, set[2] = {{0}, {0}}, early{0};
    // the first attempt fails; what it was to set is tried again, once per device, and nobody goes on before it is set
    auto work = [&](int dev) {
        device = dev;
        for (int i = 0; i < 2; i++) {
            const int rc = once([&]() -> int {
                if (calls++ == 0) return HX_ERR_CUDA;
                std::this_thread::sleep_for(std::chrono::milliseconds(30));
                set[dev]++;
                return HX_OK;
            });
            if (rc == HX_OK && !set[dev]) early++;
        }
    };
    std::vector<std::thread> t;
    for (int i = 0; i < 8; i++) t.emplace_back(work, i & 1);
    for (auto& x : t) x.join();
    if (early || set[0] != 1 || set[1] != 1 || calls != 3) { printf("early %d, set %d and %d, calls %d\n", (int)early, (int)set[0], (int)set[1], (int)calls); return 1; }
    puts("ok");
    return 0;
}
