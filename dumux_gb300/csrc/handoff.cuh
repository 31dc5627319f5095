// handoff.cuh -- what the packed lane sweeps (lanepack.cu, stencilpack.cu, stencilplane.cu) share: hand-off
// histories polled for an all-ones pattern with bounded waits, record rings filled by bulk
// copies, and asynchronous copies of vector entries.
#pragma once

#include "common.cuh"

namespace dxg {
namespace {

__device__ __forceinline__ unsigned long long lpTimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t lpAddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t lpMapa(uint32_t addr, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
template <class T>
__device__ __forceinline__ T lpEmpty()
{
    if constexpr (sizeof(T) == 8) return __longlong_as_double(-1ll);
    else return __int_as_float(-1);
}
// The upper word alone identifies the pattern: arithmetic never yields a NaN with it, and an
// 8-byte entry is seen whole.
template <class T>
__device__ __forceinline__ bool lpIsEmpty(T v)
{
    if constexpr (sizeof(T) == 8) return __double2hiint(v) == -1;
    else return __float_as_int(v) == -1;
}
// A factor entry for the sweeps.  A NaN keeps its bits through FP64 arithmetic (but for the sign), and
// a caller's matrix may hold one with all bits set: the packed records hold another NaN in its place,
// so no result ever looks like the pattern (a right-hand side with a NaN ends the solve before the
// sweeps).  Told by the bits, off the FP64 pipe.
__device__ __forceinline__ double lpEntry(double v)
{
    return (__double2hiint(v) & 0x7fffffff) == 0x7fffffff ? __longlong_as_double(0x7ff8000000000000ll) : v;
}
__device__ __forceinline__ float lpEntry(float v)
{
    return (__float_as_int(v) & 0x7fffffff) == 0x7fffffff ? __int_as_float(0x7fc00000) : v;
}
// The hand-off stores and polls carry no "memory" clobber: they need no order against the
// step's other memory operations (a poll issued early sees the pattern and repeats).
template <int OFF, class T>
__device__ __forceinline__ void lpStShared(uint32_t dst, T v)
{
    if constexpr (sizeof(T) == 8) asm volatile("st.relaxed.cta.shared::cta.f64 [%0 + %2], %1;" ::"r"(dst), "d"(v), "n"(OFF));
    else asm volatile("st.relaxed.cta.shared::cta.f32 [%0 + %2], %1;" ::"r"(dst), "f"(v), "n"(OFF));
}
template <int OFF, class T>
__device__ __forceinline__ void lpStRemote(uint32_t dst, T v)
{
    if constexpr (sizeof(T) == 8) asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0 + %2], %1;" ::"r"(dst), "d"(v), "n"(OFF));
    else asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0 + %2], %1;" ::"r"(dst), "f"(v), "n"(OFF));
}
template <class T>
__device__ __forceinline__ void lpStGpu(T* p, T v)
{
    if constexpr (sizeof(T) == 8) asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(p), "d"(v));
    else asm volatile("st.relaxed.gpu.global.f32 [%0], %1;" ::"l"(p), "f"(v));
}
// the B values of one line's hand-off entry
template <class T, int B>
struct LpVal {
    T v[B];
    __device__ __forceinline__ bool empty() const
    {
        if constexpr (B == 2) return lpIsEmpty(v[0]) || lpIsEmpty(v[1]);
        else return lpIsEmpty(v[0]);
    }
};
// ... as one relaxed vector load
template <class T, int B, int OFF>
__device__ __forceinline__ LpVal<T, B> lpLdShared(uint32_t p)
{
    LpVal<T, B> r;
    if constexpr (B == 2 && sizeof(T) == 8)
        asm volatile("ld.relaxed.cluster.shared::cta.v2.f64 {%0, %1}, [%2 + %3];" : "=d"(r.v[0]), "=d"(r.v[1]) : "r"(p), "n"(OFF));
    else if constexpr (B == 2)
        asm volatile("ld.relaxed.cluster.shared::cta.v2.f32 {%0, %1}, [%2 + %3];" : "=f"(r.v[0]), "=f"(r.v[1]) : "r"(p), "n"(OFF));
    else if constexpr (sizeof(T) == 8)
        asm volatile("ld.relaxed.cluster.shared::cta.f64 %0, [%1 + %2];" : "=d"(r.v[0]) : "r"(p), "n"(OFF));
    else
        asm volatile("ld.relaxed.cluster.shared::cta.f32 %0, [%1 + %2];" : "=f"(r.v[0]) : "r"(p), "n"(OFF));
    return r;
}
template <class T, int B>
__device__ __forceinline__ LpVal<T, B> lpLdGpu(const T* p)
{
    LpVal<T, B> r;
    if constexpr (B == 2 && sizeof(T) == 8)
        asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(r.v[0]), "=d"(r.v[1]) : "l"(p));
    else if constexpr (B == 2)
        asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(r.v[0]), "=f"(r.v[1]) : "l"(p));
    else if constexpr (sizeof(T) == 8)
        asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(r.v[0]) : "l"(p));
    else
        asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(r.v[0]) : "l"(p));
    return r;
}

// Looked at after every 64 empty polls of a wait: whether it should go on.  False once the CTA's
// sweep has stopped or when the wait's time is up (which records DXG_ERR_TIMEOUT and stops it).
// The limit is each wait's own: its first look starts it.
__device__ __forceinline__ bool lpLook(bool first, unsigned long long* deadline, int* stop, int* err, unsigned long long waitNs)
{
    if (*(volatile int*)stop) return false;
    const unsigned long long now = lpTimer();
    if (first) *deadline = now + waitNs;
    else if (now > *deadline) {
        atomicExch(err, DXG_ERR_TIMEOUT);
        *(volatile int*)stop = 1;
        return false;
    }
    return true;
}
// (the first look told by the polls so far, or by a deadline of 0)
__device__ __noinline__ bool lpGoOn(int n, unsigned long long* deadline, int* stop, int* err, unsigned long long waitNs)
{
    return lpLook(n == 64, deadline, stop, err, waitNs);
}
__device__ __noinline__ bool lpGoOn(unsigned long long* deadline, int* stop, int* err, unsigned long long waitNs)
{
    return lpLook(*deadline == 0, deadline, stop, err, waitNs);
}
// A poll: until no lane's entry is empty any more, bounded; zeros when the wait was given up.  The
// warp decides together, so it stays converged.  How a wait's first look is told moves the code of the
// steps: cleared here in FP64 64x64x32 takes 2% longer (16 iterations: 5020 and 4905 us), by the polls
// in FP32 45x37x23 1% (2225 and 2212 us); set or cleared for every poll 3%.
template <class T, int B, class LOAD>
__device__ __forceinline__ void lpPoll(LpVal<T, B>& r, LOAD&& load, unsigned long long* deadline, int* stop, int* err,
                                       unsigned long long waitNs)
{
    int n = 0;
    while (__any_sync(0xffffffffu, r.empty())) {
        if ((++n & 63) == 0) {
            bool on;
            if constexpr (sizeof(T) == 4) {
                if (n == 64) *deadline = 0;
                on = lpGoOn(deadline, stop, err, waitNs);
            } else {
                on = lpGoOn(n, deadline, stop, err, waitNs);
            }
            if (__any_sync(0xffffffffu, !on)) {
#pragma unroll
                for (int e = 0; e < B; ++e) r.v[e] = 0;
                break;
            }
        }
        r = load();
    }
}

// A record as chunks of 16 bytes per lane (each chunk's 32 lanes contiguous), then one chunk of
// 8 and / or 4 bytes per lane for the rest.
template <class T, int NV>
__device__ __forceinline__ void lpLoadRec(const unsigned char* p, int lane, T (&rec)[NV])
{
    constexpr int bytes = NV * (int)sizeof(T);
    constexpr int n16 = bytes / 16;
    constexpr int per = 16 / (int)sizeof(T);
#pragma unroll
    for (int c = 0; c < n16; ++c) {
        if constexpr (sizeof(T) == 8) {
            const double2 q = *reinterpret_cast<const double2*>(p + c * 512 + lane * 16);
            rec[c * per] = q.x;
            rec[c * per + 1] = q.y;
        } else {
            const float4 q = *reinterpret_cast<const float4*>(p + c * 512 + lane * 16);
            rec[c * per] = q.x;
            rec[c * per + 1] = q.y;
            rec[c * per + 2] = q.z;
            rec[c * per + 3] = q.w;
        }
    }
    constexpr int rem = bytes % 16;
    const unsigned char* q = p + n16 * 512;
    constexpr int at = n16 * per;
    if constexpr (rem == 8 && sizeof(T) == 8) rec[at] = reinterpret_cast<const double*>(q)[lane];
    if constexpr (rem >= 8 && sizeof(T) == 4) {
        const float2 w = reinterpret_cast<const float2*>(q)[lane];
        rec[at] = w.x;
        rec[at + 1] = w.y;
    }
    if constexpr (rem == 12) rec[at + 2] = reinterpret_cast<const float*>(q + 256)[lane];
    if constexpr (rem == 4) rec[at] = reinterpret_cast<const float*>(q)[lane];
}
// byte offset of value k of a lane inside a record of NV values
template <class T, int NV>
__device__ __forceinline__ int lpValueOffset(int k, int lane)
{
    constexpr int bytes = NV * (int)sizeof(T);
    constexpr int n16 = bytes / 16;
    constexpr int per = 16 / (int)sizeof(T);
    if (k < n16 * per) return (k / per) * 512 + lane * 16 + (k % per) * (int)sizeof(T);
    const int q = k - n16 * per;
    if constexpr (bytes % 16 >= 8) {
        constexpr int per8 = 8 / (int)sizeof(T);
        if (q < per8) return n16 * 512 + lane * 8 + q * (int)sizeof(T);
        return n16 * 512 + 256 + lane * 4;
    }
    return n16 * 512 + lane * 4;
}

__device__ __forceinline__ void lpBarInit(uint32_t bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
// one bulk copy of `bytes` into this CTA's shared memory, completing on bar
__device__ __forceinline__ void lpBulk(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ bool lpBarTry(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}
// Bounded wait for a copy of this CTA's own.  A copy always ends, so the limit only guards
// against waiting forever; on expiry the sweep runs out on what is there and reports.
__device__ __noinline__ void lpBarWait(uint32_t bar, uint32_t parity, int* stop, int* err, unsigned long long waitNs)
{
    const unsigned long long deadline = lpTimer() + waitNs + 1000000000ull;
    while (!lpBarTry(bar, parity))
        if (lpTimer() > deadline) {
            atomicExch(err, DXG_ERR_TIMEOUT);
            *(volatile int*)stop = 1;
            return;
        }
}
// asynchronous copy of one vector entry, or zeros
template <int BYTES>
__device__ __forceinline__ void lpCpAsync(uint32_t dst, const void* src, bool valid)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES),
                 "r"(valid ? BYTES : 0)
                 : "memory");
}
__device__ __forceinline__ void lpCpAsync16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void lpCommit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void lpCpWait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace
}  // namespace dxg
