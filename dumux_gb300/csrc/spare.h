// spare.h -- device memory that its holder can do without.
//
// Contexts and batches keep packed copies of their ILU(0) factors, which make the sweeps faster and
// nothing else.  Such memory must not be missing elsewhere: an allocation of the library that finds the
// device full asks the other holders on that device to give theirs back and tries once more.  A holder
// that is in a call of its own is left alone; one that gave its memory back goes on without it.
#pragma once

#include <atomic>
#include <cstddef>
#include <mutex>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

namespace dxg {

class Spare {
public:
    Spare() = default;
    Spare(const Spare&) = delete;
    Spare& operator=(const Spare&) = delete;
    virtual ~Spare() = default;   // a derived class leaves first: give() may be running
    // holder side: from here on give() may be called whenever the holder is not in use
    void join(int device)
    {
        if (joined) return;
        Registry& r = registry();
        std::lock_guard<std::mutex> lock(r.m);
        onDevice = device;
        r.all.push_back(this);
        joined = true;
    }
    void leave()
    {
        Registry& r = registry();
        std::lock_guard<std::mutex> lock(r.m);
        for (size_t k = 0; k < r.all.size(); ++k)
            if (r.all[k] == this) {
                r.all.erase(r.all.begin() + (std::ptrdiff_t)k);
                break;
            }
        joined = false;
    }
    // A call of the holder that reads or replaces the memory.  Calls of one holder do not overlap, so
    // this only waits for a give() in progress.
    class Use {
    public:
        explicit Use(Spare& s) : spare(s)
        {
            int idle = 0;
            while (!spare.state.compare_exchange_weak(idle, 1, std::memory_order_acquire)) {
                idle = 0;
                std::this_thread::yield();
            }
        }
        ~Use() { spare.state.store(0, std::memory_order_release); }
        Use(const Use&) = delete;
        Use& operator=(const Use&) = delete;

    private:
        Spare& spare;
    };
    // The spare memory of every idle holder on the device; true when there was some.
    static bool giveAll(int device)
    {
        Registry& r = registry();
        std::lock_guard<std::mutex> lock(r.m);
        bool any = false;
        for (Spare* s : r.all) {
            int idle = 0;
            if (s->onDevice != device || !s->state.compare_exchange_strong(idle, 2, std::memory_order_acquire)) continue;
            any = s->give() || any;
            s->state.store(0, std::memory_order_release);
        }
        return any;
    }

protected:
    // gives the memory back (no work on it is in flight); true when there was some
    virtual bool give() = 0;

private:
    struct Registry {
        std::mutex m;
        std::vector<Spare*> all;
    };
    static Registry& registry()
    {
        static Registry r;
        return r;
    }
    std::atomic<int> state{0};   // 0 idle, 1 in a call of the holder, 2 being given back
    int onDevice = 0;
    bool joined = false;
};

// cudaMalloc that takes spare memory back when the device is full
inline cudaError_t deviceMalloc(void** p, size_t bytes)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    int device = 0;
    if (cudaGetDevice(&device) == cudaSuccess && Spare::giveAll(device)) {
        e = cudaMalloc(p, bytes);
        if (e != cudaSuccess) cudaGetLastError();
    }
    return e;
}

// Spare memory is taken only while this much stays free beside it, for what the driver and the
// library allocate in small pieces (graphs, kernels loaded on first use, argument blocks); small
// pieces of its own without asking, which would take a small problem's first solve 40 us.
constexpr size_t kSpareHeadroom = 64u << 20, kSpareSmall = 1u << 20;
inline cudaError_t spareMalloc(void** p, size_t bytes)
{
    if (bytes > kSpareSmall) {
        size_t free = 0, total = 0;
        const cudaError_t e = cudaMemGetInfo(&free, &total);
        if (e != cudaSuccess) return e;
        if (free < bytes + kSpareHeadroom) return cudaErrorMemoryAllocation;
    }
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

}  // namespace dxg
