// Threads that ask for the driver's tensor-map encoder at the same time all get it.  The
// look-up is replaced by one that takes a while.
#include <cuda_runtime.h>

#include <chrono>
#include <thread>

static cudaError_t slow_entry_point(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q)
{
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    *p = reinterpret_cast<void*>(1);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
#define cudaGetDriverEntryPoint slow_entry_point
#include "conv_tc_encode.cuh"

#include <cstdio>
#include <vector>

int main()
{
    int missing[8] = {};
    std::vector<std::thread> threads;
    for (int i = 0; i < 8; ++i)
        threads.emplace_back([&, i] {
            std::this_thread::sleep_for(std::chrono::milliseconds(10 * i));
            missing[i] = dcb::encode_tiled_fn() == nullptr;
        });
    int n = 0;
    for (int i = 0; i < 8; ++i)
    {
        threads[(size_t) i].join();
        n += missing[i];
    }
    std::printf("%d\n", n);
    return n != 0;
}
