// pool.cu — see pool.cuh.
#include "pool.cuh"

#include <cuda.h>

#include <mutex>
#include <unordered_map>
#include <vector>

#include "prg_internal.cuh"

namespace prg {

namespace {

// Id of the current context, unique over the process's life (0 = unknown, in
// which case nothing is pooled).  A context that was destroyed and made
// again has another id.
unsigned long long context_id() {
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetId get_id = []() -> GetId {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        return reinterpret_cast<GetId>(f);
    }();
    unsigned long long id = 0;
    if (!get_id) return 0;
    if (get_id(nullptr, &id) != CUDA_SUCCESS) {
        cudaFree(nullptr);  // this thread's first call: makes the device's context current
        if (get_id(nullptr, &id) != CUDA_SUCCESS) return 0;
    }
    return id;
}

template <class T>
struct Entry {
    T item;
    unsigned long long ctx;
};

struct Pool {
    std::mutex mu;
    std::vector<Entry<void *>> slabs;
    std::vector<Entry<cudaStream_t>> streams;
    std::unordered_map<void *, unsigned long long> owner;  // slabs and streams handed out -> their context
};

Pool &pool() {
    static Pool *p = new Pool();  // never destroyed: calls may still run while statics are torn down
    return *p;
}

// Takes the newest entry of context ctx out of v.
template <class T>
bool take(std::vector<Entry<T>> &v, unsigned long long ctx, T *out) {
    for (size_t i = v.size(); i-- > 0;) {
        if (v[i].ctx != ctx) continue;
        *out = v[i].item;
        v.erase(v.begin() + i);
        return true;
    }
    return false;
}

// Makes room for one entry of context ctx: an entry of another context gives
// way first (it may be gone, so it is only forgotten).
template <class T>
bool room(std::vector<Entry<T>> &v, size_t most, unsigned long long ctx) {
    if (v.size() < most) return true;
    for (size_t i = 0; i < v.size(); i++) {
        if (v[i].ctx == ctx) continue;
        v.erase(v.begin() + i);
        return true;
    }
    return false;
}

}  // namespace

void *pinned_acquire() {
    const unsigned long long ctx = context_id();
    Pool &p = pool();
    void *s = nullptr;
    if (ctx) {
        std::lock_guard<std::mutex> lock(p.mu);
        if (take(p.slabs, ctx, &s)) {
            p.owner[s] = ctx;
            return s;
        }
    }
    PRG_CUDA(cudaMallocHost(&s, kSlabBytes));
    std::lock_guard<std::mutex> lock(p.mu);
    p.owner[s] = ctx;
    return s;
}

// Forgets that `item` was handed out; its context, or 0.
static unsigned long long take_back(Pool &p, void *item) {
    auto it = p.owner.find(item);
    if (it == p.owner.end()) return 0;
    const unsigned long long ctx = it->second;
    p.owner.erase(it);
    return ctx;
}

void pinned_release(void *s) {
    if (!s) return;
    Pool &p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        const unsigned long long ctx = take_back(p, s);
        if (ctx && room(p.slabs, kPoolSlabs, ctx)) {
            p.slabs.push_back({s, ctx});
            return;
        }
    }
    cudaFreeHost(s);
}

cudaStream_t stream_acquire() {
    const unsigned long long ctx = context_id();
    Pool &p = pool();
    cudaStream_t s = nullptr;
    if (ctx) {
        std::lock_guard<std::mutex> lock(p.mu);
        if (take(p.streams, ctx, &s)) {
            p.owner[s] = ctx;
            return s;
        }
    }
    PRG_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    std::lock_guard<std::mutex> lock(p.mu);
    p.owner[s] = ctx;
    return s;
}

void stream_release(cudaStream_t s) {
    if (!s) return;
    const bool healthy = cudaStreamSynchronize(s) == cudaSuccess;
    Pool &p = pool();
    {
        std::lock_guard<std::mutex> lock(p.mu);
        const unsigned long long ctx = take_back(p, s);
        if (healthy && ctx && room(p.streams, kPoolStreams, ctx)) {
            p.streams.push_back({s, ctx});
            return;
        }
    }
    cudaStreamDestroy(s);
}

}  // namespace prg
