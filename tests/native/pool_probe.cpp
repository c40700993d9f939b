// The pool's host code (pool.cpp, context_id.cpp) on a CUDA runtime of its own
// that counts: what the pool does is seen without a GPU.
#include "pool.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>

static std::atomic<int> lookups{0};

static CUresult get_current(CUcontext *c)
{
    *c = (CUcontext)0x1;
    return CUDA_SUCCESS;
}
static CUresult get_id(CUcontext, unsigned long long *id)
{
    *id = 7;
    return CUDA_SUCCESS;
}

extern "C" {
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long, cudaDriverEntryPointQueryResult *q)
{
    ++lookups;
    std::this_thread::sleep_for(std::chrono::milliseconds(20));
    *f = strcmp(name, "cuCtxGetId") == 0 ? (void *)get_id : (void *)get_current;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
}

// eight threads that ask for the first time at once: one lookup of each of the
// two functions, and an answer for every thread
static int first_use()
{
    std::atomic<int> ready{0}, answers{0};
    std::vector<std::thread> threads;
    for (int t = 0; t < 8; ++t)
        threads.emplace_back([&] {
            ++ready;
            while (ready < 8) std::this_thread::yield();
            unsigned long long id = 0;
            if (hpr::current_context_id(&id) && id == 7) ++answers;
        });
    for (auto &t : threads) t.join();
    printf("lookups %d answers %d\n", lookups.load(), answers.load());
    return lookups == 2 && answers == 8 ? 0 : 1;
}

int main(int argc, char **argv)
{
    if (argc == 2 && !strcmp(argv[1], "first_use")) return first_use();
    return 2;
}
