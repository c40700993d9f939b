#include "pool.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace hpr {

namespace {

struct Key {
    int device = -1;
    unsigned long long ctx = 0;
    bool operator==(const Key &o) const { return device == o.device && ctx == o.ctx; }
};

struct Block {
    Key key;
    size_t bytes = 0;
};

struct Pinned {
    void *host, *dev;
};

struct Cache {  // of one device
    Key key;
    std::multimap<size_t, void *> blocks;  // by size
    size_t bytes = 0;
    std::vector<cudaStream_t> streams;
    std::vector<Pinned> pinned;
};

std::mutex mu;
// never destroyed: handles may be released while the process ends
std::map<int, Cache> &caches()
{
    static auto *c = new std::map<int, Cache>();
    return *c;
}
std::unordered_map<void *, Block> &lent()
{
    static auto *l = new std::unordered_map<void *, Block>();
    return *l;
}
struct Lent {
    Key key;
    void *dev;
};
std::unordered_map<void *, Lent> &lent_objects()  // streams and pinned words
{
    static auto *l = new std::unordered_map<void *, Lent>();
    return *l;
}

bool here(Key &k)
{
    if (cudaGetDevice(&k.device) != cudaSuccess) return false;
    // (makes the primary context current if none is)
    if (cudaFree(nullptr) != cudaSuccess) return false;
    return current_context_id(&k.ctx);
}

// the device's cache, emptied if its context is gone (its objects went with it)
Cache &cache_of(const Key &k)
{
    Cache &c = caches()[k.device];
    if (!(c.key == k)) {
        c = Cache();
        c.key = k;
    }
    return c;
}

}  // namespace

void *pool_alloc(size_t bytes)
{
    bytes = (std::max<size_t>(bytes, 1) + 511) & ~size_t(511);
    Key k;
    const bool keyed = here(k);
    std::lock_guard<std::mutex> lock(mu);
    if (keyed) {
        Cache &c = cache_of(k);
        auto it = c.blocks.lower_bound(bytes);
        if (it != c.blocks.end() && it->first <= bytes + bytes / 4 + 65536) {
            void *p = it->second;
            lent()[p] = {k, it->first};
            c.bytes -= it->first;
            c.blocks.erase(it);
            return p;
        }
    }
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        if (keyed) {
            Cache &c = cache_of(k);
            for (auto &b : c.blocks) cudaFree(b.second);
            c.blocks.clear();
            c.bytes = 0;
        }
        if (cudaMalloc(&p, bytes) != cudaSuccess) return nullptr;
    }
    if (keyed) lent()[p] = {k, bytes};
    return p;
}

void pool_free(void *p)
{
    if (!p) return;
    Key k;
    const bool keyed = here(k);
    std::lock_guard<std::mutex> lock(mu);
    auto it = lent().find(p);
    if (it == lent().end()) {
        cudaFree(p);
        return;
    }
    const Block b = it->second;
    lent().erase(it);
    if (keyed && b.key == k) {
        Cache &c = cache_of(k);
        if (c.bytes + b.bytes <= kPoolBytes) {
            c.blocks.emplace(b.bytes, p);
            c.bytes += b.bytes;
            return;
        }
        cudaFree(p);
    } else if (!keyed || b.key.device != k.device) {
        cudaFree(p);  // another device's block, or no telling whose: freed by address
    }
    // (a block of a context that is gone went with it)
}

cudaStream_t pool_stream()
{
    Key k;
    const bool keyed = here(k);
    std::lock_guard<std::mutex> lock(mu);
    cudaStream_t s = nullptr;
    if (keyed) {
        Cache &c = cache_of(k);
        if (!c.streams.empty()) {
            s = c.streams.back();
            c.streams.pop_back();
            lent_objects()[s] = {k, nullptr};
            return s;
        }
    }
    if (cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
    if (keyed) lent_objects()[s] = {k, nullptr};
    return s;
}

void pool_stream_return(cudaStream_t s)
{
    if (!s) return;
    Key k;
    const bool keyed = here(k);
    std::lock_guard<std::mutex> lock(mu);
    auto it = lent_objects().find(s);
    const bool ours = keyed && it != lent_objects().end() && it->second.key == k;
    if (it != lent_objects().end()) {
        const bool gone = keyed && it->second.key.device == k.device && !(it->second.key == k);
        lent_objects().erase(it);
        if (gone) return;
    }
    if (ours) {
        Cache &c = cache_of(k);
        if (c.streams.size() < kPoolObjects) {
            c.streams.push_back(s);
            return;
        }
    }
    cudaStreamDestroy(s);
}

void *pool_pinned(void **dev)
{
    Key k;
    const bool keyed = here(k);
    std::lock_guard<std::mutex> lock(mu);
    Pinned p = {nullptr, nullptr};
    if (keyed) {
        Cache &c = cache_of(k);
        if (!c.pinned.empty()) {
            p = c.pinned.back();
            c.pinned.pop_back();
        }
    }
    if (!p.host) {
        if (cudaHostAlloc(&p.host, kPinnedBytes, cudaHostAllocMapped) != cudaSuccess) return nullptr;
        if (cudaHostGetDevicePointer(&p.dev, p.host, 0) != cudaSuccess) {
            cudaFreeHost(p.host);
            return nullptr;
        }
    }
    if (keyed) lent_objects()[p.host] = {k, p.dev};
    memset(p.host, 0, kPinnedBytes);
    *dev = p.dev;
    return p.host;
}

void pool_pinned_return(void *host)
{
    if (!host) return;
    Key k;
    const bool keyed = here(k);
    std::lock_guard<std::mutex> lock(mu);
    auto it = lent_objects().find(host);
    if (it != lent_objects().end()) {
        const Lent l = it->second;
        lent_objects().erase(it);
        if (keyed && l.key.device == k.device && !(l.key == k)) return;  // went with its context
        if (keyed && l.key == k) {
            Cache &c = cache_of(k);
            if (c.pinned.size() < kPoolObjects) {
                c.pinned.push_back({host, l.dev});
                return;
            }
        }
    }
    cudaFreeHost(host);
}

bool pool_release(int device)
{
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!caches().count(device)) return true;  // (nothing kept: leaves a device without a context alone)
    }
    int current = -1;
    if (cudaGetDevice(&current) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return false;
    Key k;
    const bool keyed = here(k);
    if (keyed) {
        std::lock_guard<std::mutex> lock(mu);
        Cache &c = cache_of(k);
        for (auto &b : c.blocks) cudaFree(b.second);
        for (auto &s : c.streams) cudaStreamDestroy(s);
        for (auto &p : c.pinned) cudaFreeHost(p.host);
        caches().erase(device);
    }
    cudaSetDevice(current);
    return keyed;
}

}  // namespace hpr
