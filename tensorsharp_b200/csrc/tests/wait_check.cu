// Stand-alone check of the bounded waits of tcgen05.cuh: a phase that nobody ends is given up at its limit, by one limit for several of them
// where a kernel waits for its copies in flight, and a phase that ends late is waited for.
//
//     wait_check        exit code 0 when every case passes, 77 without a GPU; one line per case on stdout
#include <cuda_runtime.h>

#include <cstdio>

#include "../tcgen05.cuh"

constexpr uint64_t MS = 1000000;

struct Seen { int ok; uint64_t ns; };

__device__ void note(Seen* out, int i, bool ok, uint64_t t0) {
    if (threadIdx.x == 0) out[i] = {ok, tc::global_timer_ns() - t0};
}

// one block of two warps: the first waits, the second ends a phase after 3 ms
__global__ void waits(Seen* out) {
    __shared__ uint64_t bar[8];
    if (threadIdx.x == 0) {
        for (int i = 0; i < 8; ++i) tc::mbar_init(&bar[i], 1);
        tc::fence_barrier_init();
    }
    __syncthreads();
    uint64_t t0 = tc::global_timer_ns();
    if (threadIdx.x >= 32) {
        while (tc::global_timer_ns() - t0 < 3 * MS) __nanosleep(1000);
        if (threadIdx.x == 32) tc::mbar_arrive(&bar[7]);
        return;
    }
    const bool late = tc::hold<true>(&bar[7], 0);
    note(out, 0, late, t0);
    t0 = tc::global_timer_ns();
    note(out, 1, tc::hold(&bar[7], 0), t0);                        // a phase that has ended
    t0 = tc::global_timer_ns();
    note(out, 2, tc::hold<false>(&bar[0], 0), t0);
    t0 = tc::global_timer_ns();
    note(out, 3, tc::hold<true>(&bar[0], 0), t0);
    t0 = tc::global_timer_ns();
    bool given_up = false, any = false;
    for (int i = 0; i < 7; ++i) any |= tc::settle(&bar[i], 0, given_up);
    note(out, 4, any, t0);
    t0 = tc::global_timer_ns();
    note(out, 5, tc::settle(&bar[7], 0, given_up), t0);            // what is there already is seen all the same
}

int main() {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n == 0) {
        std::printf("SKIP no GPU\n");
        return 77;
    }
    Seen* d = nullptr;
    Seen h[6] = {};
    if (cudaMalloc(&d, sizeof(h)) != cudaSuccess) return 2;
    waits<<<1, 64>>>(d);
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpy(h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) {
        std::printf("FAIL %s\n", cudaGetErrorString(cudaGetLastError()));
        return 1;
    }
    // the least and the most that a case may take: a wait's limit is about a second, two at most
    const struct { const char* what; int ok; uint64_t least, most; } want[6] = {
        {"a phase that ends after 3 ms", 1, 2 * MS, 200 * MS}, {"a phase that has ended", 1, 0, 1 * MS},
        {"nobody arrives", 0, 200 * MS, 2200 * MS}, {"nobody arrives, idle", 0, 200 * MS, 2200 * MS},
        {"seven that nobody ends, one limit", 0, 200 * MS, 2300 * MS}, {"there already, limit past", 1, 0, 1 * MS}};
    bool all = true;
    for (int i = 0; i < 6; ++i) {
        const bool good = h[i].ok == want[i].ok && h[i].ns >= want[i].least && h[i].ns <= want[i].most;
        std::printf("%s %s: %d after %.3f ms\n", good ? "ok  " : "FAIL", want[i].what, h[i].ok, h[i].ns / 1e6);
        all &= good;
    }
    std::printf(all ? "OK\n" : "FAILED\n");
    return all ? 0 : 1;
}
