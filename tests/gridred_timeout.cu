// A grid_reduce whose second block never arrives: the first block's waits run
// out (test_gpu_barrier_timeout.py compiles this with a short limit).  Prints
// how many calls reported it, the calls, their clocks and the limit.
#include <cstdio>

#include "gridred.cuh"

namespace crimson {
void set_last_error(const std::string&) {}
void note_launch() {}
int sm_count() { return 1; }
}  // namespace crimson
using namespace crimson;

__global__ void k(ulonglong2* pk, int calls, long long* out) {
    __shared__ double red[32], tot[1];
    __shared__ unsigned char fpend[32];
    if (blockIdx.x == 1) return;
    if (threadIdx.x < 32) red[threadIdx.x] = 1.0;
    bool fail = false;
    int reported = 0;
    const long long t0 = clock64();
    for (int i = 1; i <= calls; ++i) {
        fail = grid_reduce(pk, 1, red, 0, 0u, fpend, (unsigned long long)i, i & 1, tot, fail);
        reported += fail ? 1 : 0;
    }
    if (threadIdx.x == 0) {
        out[0] = reported;
        out[1] = clock64() - t0;
    }
}

int main() {
    const int calls = 60;
    ulonglong2* pk = nullptr;
    long long *out = nullptr, h[2] = {0, 0};
    if (cudaMalloc(&pk, 2 * 2 * sizeof(ulonglong2)) || cudaMalloc(&out, sizeof(h))) return 2;
    if (cudaMemset(pk, 0, 2 * 2 * sizeof(ulonglong2)) || cudaMemset(out, 0, sizeof(h))) return 2;
    k<<<2, 256>>>(pk, calls, out);
    if (cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost)) return 3;   // the context is usable
    std::printf("%lld %d %lld %lld\n", h[0], calls, h[1], (long long)kGrWaitClocks);
    return 0;
}
