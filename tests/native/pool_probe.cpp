// The pool's host code (pool.cpp, context_id.cpp) on a CUDA runtime of its own
// that counts: what the pool does is seen without a GPU.
#include "pool.h"

#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <set>
#include <thread>
#include <vector>

static std::atomic<int> lookups{0};
static bool ids = true;           // the driver answers
static std::set<void *> held;     // blocks, pinned words and streams that exist

static CUresult get_current(CUcontext *c)
{
    *c = (CUcontext)0x1;
    return CUDA_SUCCESS;
}
static CUresult get_id(CUcontext, unsigned long long *id)
{
    *id = 7;
    return ids ? CUDA_SUCCESS : CUDA_ERROR_UNKNOWN;
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
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t bytes)
{
    held.insert(*p = malloc(bytes));
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (p && held.erase(p)) free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned)
{
    held.insert(*p = malloc(bytes));
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned)
{
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p)
{
    return cudaFree(p);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return cudaMalloc((void **)s, 1); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return cudaFree(s); }
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

// a block that the pool has on record, returned while the context's identity
// cannot be read: given back to the device, not forgotten
static int unknown_context()
{
    void *p = hpr::pool_alloc(1000);
    ids = false;
    hpr::pool_free(p);
    printf("%zu blocks still allocated\n", held.size());
    return held.empty() ? 0 : 1;
}

// what the pool keeps can be had back; what is in use stays
static int release()
{
    void *dev = nullptr, *kept[2] = {hpr::pool_alloc(1000), hpr::pool_alloc(5000)}, *used = hpr::pool_alloc(100000);
    cudaStream_t s = hpr::pool_stream();
    void *word = hpr::pool_pinned(&dev);
    for (void *p : kept) hpr::pool_free(p);
    hpr::pool_stream_return(s);
    hpr::pool_pinned_return(word);
    const size_t before = held.size();
    const bool ok = hpr::pool_release(0) && hpr::pool_release(1);
    printf("%zu objects, %zu after the release\n", before, held.size());
    if (!ok || before != 5 || held.size() != 1 || !held.count(used)) return 1;
    hpr::pool_free(used);  // kept again
    return held.size() == 1 && hpr::pool_alloc(100000) == used ? 0 : 1;
}

int main(int argc, char **argv)
{
    if (argc == 2 && !strcmp(argv[1], "first_use")) return first_use();
    if (argc == 2 && !strcmp(argv[1], "unknown_context")) return unknown_context();
    if (argc == 2 && !strcmp(argv[1], "release")) return release();
    return 2;
}
