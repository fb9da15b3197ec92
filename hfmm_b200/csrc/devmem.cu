// Device memory blocks of the library (hfmm::DevBuf). A plan rebuilt for moved points makes
// and drops about 160 buffers; a cudaMalloc and cudaFree pair of each took 26 of the 32 ms of
// such a call at 1e5 points (90 us a call here, and milliseconds at times on a shared host).
// A block of at most MOST_BLOCK bytes that is dropped idle, or inside a KeepBlocks scope, is
// kept, up to MOST_KEPT bytes in all, and serves the next allocation of its size class on its
// device. A scope's block is kept after a wait for the device, so whoever gets one finds no
// kernel of any stream on it. Nothing is kept while no plan is alive, and the last plan's end
// frees all of it.
#include "hfmm_internal.cuh"

#include <map>
#include <mutex>

namespace hfmm {

namespace {

constexpr size_t MOST_BLOCK = (size_t)32 << 20, MOST_KEPT = (size_t)128 << 20;

struct Kept {
    std::mutex mu;
    std::multimap<std::pair<int, size_t>, void*> blocks;   // (device, bytes)
    size_t bytes = 0;
    int plans = 0;
};
Kept& kept() {
    static Kept* k = new Kept;   // outlives every static DevBuf; the driver frees at exit
    return *k;
}

// eight classes an octave, 512 bytes at least; a block too large to be kept has its own size
// (rounded up it could be what no longer fits the device)
size_t size_class(size_t bytes) {
    if (bytes > MOST_BLOCK) return bytes;
    size_t step = 512;
    while (step * 16 < bytes) step *= 2;
    return (bytes + step - 1) / step * step;
}

void free_all() {   // with the lock held
    Kept& k = kept();
    for (auto& b : k.blocks) cudaFree(b.second);
    k.blocks.clear();
    k.bytes = 0;
}

thread_local int t_keep = 0, t_idle = 0;   // scopes, and those whose blocks are idle

}  // namespace

KeepBlocks::KeepBlocks(bool idle_) : idle(idle_) {
    ++t_keep;
    t_idle += idle;
}
KeepBlocks::~KeepBlocks() {
    --t_keep;
    t_idle -= idle;
}
bool keeping_blocks() { return t_keep > 0; }

void* dev_alloc(size_t bytes, size_t* cap, int* device) {
    HFMM_CUDA(cudaGetDevice(device));
    *cap = size_class(bytes);
    Kept& k = kept();
    {
        std::lock_guard<std::mutex> g(k.mu);
        auto it = k.blocks.find({*device, *cap});
        if (it != k.blocks.end()) {
            void* p = it->second;
            k.blocks.erase(it);
            k.bytes -= *cap;
            return p;
        }
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, *cap);
    if (e == cudaErrorMemoryAllocation) {   // what is kept may be what is missing
        cudaGetLastError();
        {
            std::lock_guard<std::mutex> g(k.mu);
            free_all();
        }
        e = cudaMalloc(&p, *cap);
    }
    if (e != cudaSuccess) {
        *cap = 0;
        throw Error{HFMM_ERR_CUDA, std::string("cudaMalloc: ") + cudaGetErrorString(e)};
    }
    return p;
}

void dev_free(void* p, size_t cap, int device, bool idle) noexcept {
    Kept& k = kept();
    int now = -1;
    idle = idle || t_idle > 0;
    if (cap <= MOST_BLOCK && (idle || t_keep > 0) && cudaGetDevice(&now) == cudaSuccess && now == device) {
        // what is counted is what is in the store: the lock is open during the wait, and another
        // thread may empty the store meanwhile
        auto room = [&] { return k.plans > 0 && k.bytes + cap <= MOST_KEPT; };
        std::unique_lock<std::mutex> g(k.mu);
        if (room() && !idle) {
            g.unlock();
            idle = cudaDeviceSynchronize() == cudaSuccess;
            g.lock();
        }
        if (idle && room()) {
            try {
                k.blocks.emplace(std::make_pair(device, cap), p);
                k.bytes += cap;
                return;
            } catch (...) {
            }
        }
    }
    cudaFree(p);
}

void dev_plan_count(int change) {
    Kept& k = kept();
    std::lock_guard<std::mutex> g(k.mu);
    k.plans += change;
    if (k.plans == 0) free_all();
}

}  // namespace hfmm
