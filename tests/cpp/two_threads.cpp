// Products of different sizes from two host threads, a stream each: prints how many launches were refused.
#include <atomic>
#include <cstdio>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "twm_dense.h"

static std::atomic<int> refused{0}, launches{0};

struct Shape { int m, n, k; };
static void run(int dtype, std::vector<Shape> shapes) {
    void *a, *w, *c;
    cudaStream_t s;
    if (cudaSetDevice(0) || cudaStreamCreate(&s) || cudaMalloc(&a, 1 << 20) || cudaMalloc(&w, 16 << 20) || cudaMalloc(&c, 16 << 20) ||
        cudaMemset(a, 0, 1 << 20) || cudaMemset(w, 0, 16 << 20)) { refused += 1000000; return; }
    for (int i = 0; i < 4000; ++i) {
        for (const Shape& x : shapes) {
            ++launches;
            if (twm_dense_gemm(dtype, a, x.k, w, x.k, c, x.n, x.m, x.n, x.k, TWM_EPI_STORE_F32, 0, 0, s) != TWM_OK) {
                if (refused++ == 0) printf("%s\n", twm_dense_last_error());
            }
        }
        if (i % 64 == 0) cudaStreamSynchronize(s);
    }
    cudaStreamSynchronize(s);
}

int main() {
    for (int dtype : {TWM_DENSE_BF16, TWM_DENSE_F32}) {
        std::thread x(run, dtype, std::vector<Shape>{{100, 2048, 512}, {20, 1024, 512}}), y(run, dtype, std::vector<Shape>{{24, 2048, 512}, {60, 1024, 512}});
        x.join();
        y.join();
    }
    unsigned int word = 0;
    const int device = twm_dense_device_error(nullptr, &word);
    printf("%d launches, %d refused, device status %d, error word %u\n", launches.load(), refused.load(), device, word);
    return refused.load() != 0 || device != 0 || word != 0;
}
