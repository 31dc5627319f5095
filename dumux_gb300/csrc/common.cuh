// common.cuh -- shared device/host helpers of the GB300 cc-TPFA library.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <cstdio>
#include <stdexcept>
#include <string>
#include <utility>

#include "../../include/dumux_gb300.h"
#include "spare.h"

namespace dxg {

// Thrown inside the library only; converted to a status code at the C ABI.
struct Error : std::runtime_error {
    int status;
    Error(int st, const std::string& msg) : std::runtime_error(msg), status(st) {}
};

#define DXG_CUDA(call)                                                                       \
    do {                                                                                     \
        cudaError_t e_ = (call);                                                             \
        if (e_ != cudaSuccess)                                                               \
            throw ::dxg::Error(e_ == cudaErrorMemoryAllocation ? DXG_ERR_OOM : DXG_ERR_CUDA, \
                               std::string(#call) + ": " + cudaGetErrorString(e_));          \
    } while (0)

// One device allocation that the buffers of a problem upload are carved from: while a
// thread has a block installed (DevBlockScope), DevBuf::alloc takes 256-byte aligned pieces
// of it instead of calling cudaMalloc once per buffer.  The owner keeps the block alive
// for as long as the buffers carved from it.
struct DevBlock {
    unsigned char* base = nullptr;
    size_t cap = 0, used = 0;
};
inline DevBlock*& currentDevBlock()
{
    thread_local DevBlock* b = nullptr;
    return b;
}
struct DevBlockScope {
    DevBlock* prev;
    explicit DevBlockScope(DevBlock* b) : prev(currentDevBlock()) { currentDevBlock() = b; }
    ~DevBlockScope() { currentDevBlock() = prev; }
};

// Owning device buffer (or a piece of the installed DevBlock, which it does not free).
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    bool owned = true;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    void release()
    {
        if (p && owned) cudaFree(p);
        p = nullptr;
        n = 0;
        owned = true;
    }
    void alloc(size_t count)
    {
        if (count == n && p) return;
        release();
        if (count == 0) return;
        const size_t bytes = (count * sizeof(T) + 255) & ~(size_t)255;
        DevBlock* blk = currentDevBlock();
        if (blk && blk->used + bytes <= blk->cap) {
            p = reinterpret_cast<T*>(blk->base + blk->used);
            blk->used += bytes;
            owned = false;
            n = count;
            return;
        }
        DXG_CUDA(deviceMalloc(reinterpret_cast<void**>(&p), count * sizeof(T)));
        n = count;
    }
    // memory that the owner can do without (spare.h): false where the device does not have it to spare
    bool allocSpare(size_t count)
    {
        release();
        const cudaError_t e = spareMalloc(reinterpret_cast<void**>(&p), count * sizeof(T));
        if (e == cudaErrorMemoryAllocation) {
            p = nullptr;
            return false;
        }
        DXG_CUDA(e);
        n = count;
        return true;
    }
    T* get() const { return p; }
    size_t bytes() const { return n * sizeof(T); }
};

// A launch of the Krylov iteration's chain: a programmatic dependent of the launch before it, whose
// blocks may start (and stop in chainWait) while that one still runs, so its launch latency and
// the ramp of the grid overlap with it.  Every kernel launched this way calls chainWait before it
// touches memory, and reads what the chain writes with plain loads (the read-only path, __ldg or a
// const __restrict__ parameter, is for data that nobody writes while the kernel runs).
template <class... P, class... Q>
inline void launchChained(void (*kern)(P...), dim3 grid, unsigned threads, cudaStream_t st, Q&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    DXG_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<Q>(args)...));
}
// Waits until the launch before has completed and its writes are visible.  A grid of at most `early`
// blocks lets the next launch of the chain start at once.  Its blocks then wait on the SMs that this
// grid leaves free, several to an SM, and share that SM's FP64 pipe when they run; so how large a
// grid may be depends on what follows:
//   * a kernel over the whole GPU (red-black passes, AMG levels): a quarter of the SMs.  Sixteen
//     iterations, never early, early up to 38 and up to 152 blocks: red-black 10x10 mixed 645, 595 and
//     592 us, 24x24x24 FP64 929, 921 and 1011 us, 33x33x33 961, 961 and 1341 us; AMG 30x30x30 2771,
//     2806 and 3750 us;
//   * a cluster sweep, which has few CTAs and needs SMs of its own: up to one block per SM.  24x24x24
//     FP64, never early, up to 38 and up to 152 blocks: 2371, 2322 and 2306 us, 32x32x32 mixed 2090,
//     2090 and 2038 us.
constexpr unsigned kSms = 152;   // of a GB300
constexpr unsigned kEarlyWide = kSms / 4, kEarlySweep = kSms;
__device__ __forceinline__ void chainWait(unsigned early)
{
    if (gridDim.x * gridDim.y <= early) asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

constexpr int kMaxMaterials = 16;

// Derived constants of one regularised Brooks-Corey parameter set
// (BrooksCoreyRegularization::initPcParameters_, brookscorey.hh:477-486).
// Two-point cubic spline of the Van Genuchten regularisation (Spline<Scalar, 2>,
// dumux/common/spline.hh:310-345): end points, values and the moments of the clamped
// spline (dumux/common/splinecommon_.hh:419-440).
struct Spline2 {
    double x0, x1, y0, y1, M0, M1;
};

struct MaterialLaw {
    int kind;                      // 0 regularised Brooks-Corey, 1 regularised Van Genuchten
    double pe, lambda, swr, snr, pcLowSwe;
    double denom;                  // 1.0 - swr - snr
    double expPc;                  // -1.0/lambda
    double expKrw;                 // 2.0/lambda + 3.0
    double expKrn;                 // 2.0/lambda + 1.0
    double pcLowSwePcValue, pcDerivativeLowSw, pcDerivativeHighSwEnd, entryPressure;
    // derivative constants (brookscorey.hh:166-174, 241-249, 295-305; efftoabsdefaultpolicy.hh:135)
    double dsweDsw;                // 1.0/(1.0 - swr - snr)
    double dpcCoef, dpcExp;        // -pe/lambda, -1.0/lambda - 1.0
    double dkrwCoef, dkrwExp;      // 2.0/lambda + 3.0, 2.0/lambda + 2.0
    double lambdaInv, dkrnExp;     // 1.0/lambda, 2*lambdaInv
    // Van Genuchten (vangenuchten.hh:30-300): alpha, n, m = 1 - 1/n, l and the exponents
    // the reference forms at run time; regularisation thresholds and splines
    double vgAlpha, vgN, vgM, vgL;
    double vgNegInvM, vgInvN, vgInvM;       // -1.0/m, 1.0/n, 1.0/m
    double pcHighSwe, krnLowSwe, krwHighSwe;
    Spline2 pcSpline, krwSpline, krnSpline;
};

// Problem constants visible to the kernels.
struct ProblemConsts {
    int dim, b;
    int nx, ny, nz;
    int64_t N;
    int64_t sideOffset[7];
    int gravity;                   // Problem.EnableGravity
    int gravAxisMask;              // bit a set: faces normal to axis a carry gravity terms
    double density[2], viscosity[2];
    double mobility1p;             // 1.0/viscosity (1p)
    double upwindWeight;
    int upwindFull;                // upwind weight != 1
    int method;                    // numeric difference method (3: analytic derivatives)
    double baseEps;
    double magnitude[2];
    int numMaterials;
    int hasSource;
    MaterialLaw law[kMaxMaterials];
};

__host__ __device__ inline int slotOfFace(int dim, int f)
{
    const int a = f >> 1;
    return (f & 1) ? dim + 1 + a : dim - 1 - a;
}

}  // namespace dxg
