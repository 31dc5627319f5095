// stencilpack.cu -- ILU(0) triangular solves of the 2D scalar 9-point stencil (1p MPFA-O) in one
// launch: the forward and the backward sweep over packed factor records.
//
// Natural order: cell (x, y) sits on level x + 2y.  Forward it needs its own line's cell x-1
// (level -1) and line y-1's cells x+1, x, x-1 (levels -1, -2, -3); backward line y+1's cells x-1,
// x, x+1 and its own line's x+1.  What bounds the sweeps: the chain of nx + 2 ny levels, each at
// least the FP64 instructions of a row (4 forward, 5 backward; on GB300 64 cycles each on the
// sub-partition of the warp, two of them and a shuffle dependent on the level before).  One CTA
// with a line per thread put two warps on every sub-partition at 256 lines and paid a CTA
// barrier a level; so here a CTA holds at most two warps, the CTAs of one cluster hand their
// boundary lines on by distributed shared memory, and a step is kept to its chain as in
// lanepack.cu: factor records packed in the order the sweeps read them and streamed by bulk
// copies, the right-hand side and the forward results in shared memory, polled histories.
//
// Mapping: lane j of a warp holds line j, cell x = t - 1 - 2j at the warp's step t (ascending
// forward, descending backward).  The neighbour line's newest result (slots 2 / 6) comes by
// shuffle, across warps and CTAs through a history indexed by the consumer's step; the two older
// ones (slots 1, 0 / 7, 8) are the lane's own previous two shuffles.  The terms enter the row sum
// oldest first, as in stencilApplyKernel (linalg.cu): same operands, same order, same bits.
// Waits are bounded as in lanepack.cu.
//
// Measured per apply, 256x256: one-CTA line sweeps 0.667 ms, this kernel 0.30 ms.
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"
#include "handoff.cuh"
#include "linalg_kernels.cuh"

namespace cg = cooperative_groups;

namespace dxg {
namespace {

constexpr int kSpLines = 32;             // lines per warp
constexpr int kSpMaxWarps = 2;
constexpr int kSpStageSteps = 4;
constexpr int kSpMaxStages = 6;
constexpr int kSpPad = 2 * kSpLines;     // of the histories: the boundary line's steps without a cell
constexpr int kSpFwd = 4, kSpBwd = 5;    // values of a record: slots 0..3; slots 8, 7, 6, 5 and the pivot
constexpr size_t kSpSmemLimit = 226 * 1024;

// steps of a warp with `lines` lines, padded to whole stages: the first forward and the first
// backward step of a line at the warp's edge only fetch a neighbour value
__host__ __device__ inline int spSteps(int nx, int lines)
{
    return (nx + 2 + 2 * (lines - 1) + kSpStageSteps - 1) / kSpStageSteps * kSpStageSteps;
}

struct SpSmem {
    size_t ring, vbuf, ybuf, zero, sink, total;
};
__host__ __device__ inline SpSmem spSmem(int steps, int W, int stages)
{
    SpSmem s{};
    size_t o = 0;
    s.ring = o;
    o += (size_t)W * stages * kSpStageSteps * kSpBwd * 32 * 8;
    s.vbuf = o;
    o += (size_t)W * steps * 32 * 8;
    s.ybuf = o;
    o += (2 * (size_t)(W + 1) * (kSpPad + steps) + kSpPad) * 8;
    s.zero = o;
    o += 16 * 8;
    s.sink = o;
    o += 16 * 8;
    s.total = o;
    return s;
}

}  // namespace

// The packed records of both sweeps (blockIdx.y), zeros where a lane has no cell or neighbour.
__global__ void __launch_bounds__(256) stencilPackKernel(StencilArgs a, StencilPackPlan p)
{
    const bool fwd = blockIdx.y == 0;
    const int NV = fwd ? kSpFwd : kSpBwd;
    double* const out = reinterpret_cast<double*>(a.pack[fwd ? 0 : 1]);
    const int64_t total = (int64_t)p.ctas * p.warps * p.steps * 32;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
        const int lane = (int)(k & 31);
        const int64_t rec = k >> 5;
        const int s = (int)(rec % p.steps), cw = (int)(rec / p.steps);
        const int y = cw * kSpLines + lane;
        const int x = (fwd ? s : p.steps - 1 - s) - 1 - 2 * lane;
        double v[kSpBwd] = {0.0, 0.0, 0.0, 0.0, 0.0};
        if (y < a.ny && x >= 0 && x < a.nx) {
            const int64_t i = (int64_t)y * a.nx + x;
            const uint32_t m = a.mask[i];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int slot = fwd ? e : 8 - e;
                if ((m >> slot) & 1u) v[e] = lpEntry(a.LU[(int64_t)slot * a.N + i]);
            }
            if (!fwd) v[4] = lpEntry(a.Dinv[i]);
        }
        // values in pairs (16 bytes per lane), the last one alone
        double* dst = out + rec * (NV * 32);
        dst[lane * 2] = v[0];
        dst[lane * 2 + 1] = v[1];
        dst[64 + lane * 2] = v[2];
        dst[64 + lane * 2 + 1] = v[3];
        if (!fwd) dst[128 + lane] = v[4];
    }
}

__global__ void __launch_bounds__((kSpMaxWarps + 1) * 32) stencilPackApply(StencilArgs a, StencilPackPlan pl,
                                                                            const double* d, double* v)
{
    constexpr int SS = kSpStageSteps, STAGE = SS * kSpBwd * 32 * 8, LPW = kSpLines;
    extern __shared__ __align__(128) unsigned char spRaw[];
    __shared__ int stopFlag;
    __shared__ volatile int consumed[kSpMaxWarps];   // blocks each warp has read out of its ring
    __shared__ __align__(8) unsigned long long bars[kSpMaxWarps][kSpMaxStages];

    cg::cluster_group cluster = cg::this_cluster();
    const int nx = a.nx, ny = a.ny, W = pl.warps, steps = pl.steps, stages = pl.stages;
    const SpSmem lay = spSmem(steps, W, stages);
    const int cta = (int)blockIdx.x, lane = threadIdx.x & 31;
    // through a shuffle, so that what depends on it is known to be uniform over the warp
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const bool producer = warp == W;
    const int tileLine = cta * W * LPW;
    const int y = tileLine + warp * LPW + lane;
    const bool lineOk = !producer && y < ny;
    const bool hasLo = cta > 0, hasHi = cta + 1 < pl.ctas;
    auto blocksOf = [&](int w) {
        const int lines = min(LPW, ny - (tileLine + w * LPW));
        return lines > 0 ? spSteps(nx, lines) / SS : 0;
    };
    double* const ybuf = reinterpret_cast<double*>(spRaw + lay.ybuf);
    const int yRow = kSpPad + steps, yDir = (W + 1) * yRow;
    const unsigned long long waitNs = a.waitNs ? a.waitNs : 500000000ull;

    // histories: empty where a value will arrive, zero elsewhere.  Entry t forward: cell x = t of
    // the line before; backward: cell x = t - 64 of the line after
    if (!producer) {
        for (int k = threadIdx.x; k < 2 * yDir; k += W * 32) {
            const int x = k % yRow - kSpPad - (k < yDir ? 0 : 2 * LPW);
            ybuf[k] = x >= 0 && x < nx ? lpEmpty<double>() : 0.0;
        }
        if (lane < 16) {
            reinterpret_cast<double*>(spRaw + lay.zero)[lane] = 0.0;
        }
        if (lane < kSpMaxStages) lpBarInit(lpAddr(&bars[warp][lane]));
        if (lane == 0) consumed[warp] = 0;
    } else if (lane == 0) {
        stopFlag = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cluster.sync();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool skip = a.ks && a.ks->status != KS_RUNNING;

    if (producer) {
        if (lane == 0 && !skip) {
            int issued[kSpMaxWarps] = {};
            bool more = true;
            while (more) {
                more = false;
#pragma unroll
                for (int w = 0; w < kSpMaxWarps; ++w) {
                    const int n = w < W ? blocksOf(w) : 0;
                    if (issued[w] >= 2 * n) continue;
                    more = true;
                    if (issued[w] - consumed[w] >= stages) continue;
                    const int b = issued[w]++;
                    const bool fwd = b < n;
                    const uint32_t bytes = SS * (fwd ? kSpFwd : kSpBwd) * 32 * 8;
                    const size_t all = steps / SS;   // blocks a warp has room for; the backward ones end there
                    const size_t at = (((size_t)cta * W + w) * all + (fwd ? b : b - n + all - n)) * bytes;
                    lpBulk(lpAddr(spRaw + lay.ring + ((size_t)w * stages + b % stages) * STAGE), a.pack[fwd ? 0 : 1] + at,
                           bytes, lpAddr(&bars[w][b % stages]));
                }
                __nanosleep(64);
            }
        }
        __syncwarp();
    } else if (!skip && tileLine + warp * LPW < ny) {
        unsigned char* const ring = spRaw + lay.ring + (size_t)warp * stages * STAGE;
        const uint32_t barAddr = lpAddr(&bars[warp][0]);
        double* const vb = reinterpret_cast<double*>(spRaw + lay.vbuf) + (size_t)warp * steps * 32 + lane;   // + t * 32
        const int jx = lineOk ? 1 + 2 * lane : 0x40000000;   // t - jx: the lane's cell, when below nx unsigned
        const int64_t lineBase = lineOk ? (int64_t)y * nx : 0;
        unsigned long long deadlineOfWait = 0, *const deadline = &deadlineOfWait;
        const int myBlocks = blocksOf(warp);
        int block = 0, stage = 0;
        uint32_t parity = 0;
        // the right-hand side, zeros where the lane has no cell
        for (int t = 0; t < myBlocks * SS; ++t) {
            const int x = t - jx;
            const bool valid = (unsigned)x < (unsigned)nx;
            lpCpAsync<8>(lpAddr(vb + t * 32), valid ? d + lineBase + x : d, valid);
        }
        lpCommit();
        lpCpWait<0>();

        auto sweep = [&](auto dirC) {
            constexpr int DIR = decltype(dirC)::value;
            constexpr int NV = DIR > 0 ? kSpFwd : kSpBwd;
            constexpr int REC = NV * 32 * 8;
            const int t0 = DIR > 0 ? 0 : myBlocks * SS - 1;
            const bool edge = lane == (DIR > 0 ? 0 : LPW - 1);
            const int yWarp = DIR > 0 ? (warp > 0 ? warp - 1 : W) : (warp < W - 1 ? warp + 1 : W);
            const bool src = edge && lineOk && (DIR > 0 ? warp > 0 || hasLo : (warp < W - 1 ? y + 1 < ny : hasHi));
            double* const dirBuf = ybuf + (DIR > 0 ? 0 : yDir) + kSpPad;
            uint32_t yIn = src ? lpAddr(dirBuf + yWarp * yRow + t0) : lpAddr(spRaw + lay.zero) + 64;
            const uint32_t yInStep = src ? (uint32_t)(DIR * SS * 8) : 0u;
            // the boundary line's results: cell x of the last line (forward) at entry x, of the
            // first line (backward) at entry x + 64; every lane stores every step (others to a sink)
            const bool pub = lineOk && lane == (DIR > 0 ? LPW - 1 : 0) && (DIR > 0 ? warp < W - 1 || hasHi : warp > 0 || hasLo);
            const bool far = DIR > 0 ? warp == W - 1 && hasHi : warp == 0 && hasLo;   // to another CTA
            uint32_t yOut = lpAddr(spRaw + lay.sink) + 64;
            if (pub) yOut = lpAddr(dirBuf + (far ? W : warp) * yRow + t0 + (DIR > 0 ? -(2 * LPW - 1) : 2 * LPW - 1));
            if (far) yOut = lpMapa(yOut, pub ? cta + DIR : cta);
            const uint32_t yOutStep = pub ? (uint32_t)(DIR * SS * 8) : 0u;
            double* dst = v + lineBase + t0 - (1 + 2 * lane);   // dereferenced where the lane has a cell
            double* vt = vb + t0 * 32;

            if (!lpBarTry(barAddr + 8 * stage, parity)) lpBarWait(barAddr + 8 * stage, parity, &stopFlag, a.err, waitNs);
            double c[NV], cV = vt[0], prev = 0.0, n2 = 0.0, n3 = 0.0;
            lpLoadRec<double, NV>(ring + stage * STAGE, lane, c);

            auto step = [&](int t, auto kC, const unsigned char* next) {
                constexpr int K = DIR * decltype(kC)::value;
                const double up = DIR > 0 ? __shfl_up_sync(0xffffffffu, prev, 1) : __shfl_down_sync(0xffffffffu, prev, 1);
                LpVal<double, 1> yp = lpLdShared<double, 1, K * 8>(yIn);
                double acc = fma(-c[0], n3, cV);
                acc = fma(-c[1], n2, acc);
                double n[NV];
                lpLoadRec<double, NV>(next, lane, n);
                const double nV = vt[(K + DIR) * 32];
                lpPoll<double, 1>(yp, [&] { return lpLdShared<double, 1, K * 8>(yIn); }, deadline, &stopFlag, a.err, waitNs);
                const double n1 = edge ? yp.v[0] : up;
                acc = fma(-c[2], n1, acc);
                acc = fma(-c[3], prev, acc);
                const double res = DIR > 0 ? acc : c[NV - 1] * acc;
                if (far) lpStRemote<K * 8>(yOut, res);
                else lpStShared<K * 8>(yOut, res);
                if (DIR > 0) vt[K * 32] = res;
                else if ((unsigned)(t + K - jx) < (unsigned)nx) dst[K] = res;
                n3 = n2;
                n2 = n1;
                prev = res;
                cV = nV;
#pragma unroll
                for (int e = 0; e < NV; ++e) c[e] = n[e];
            };
            for (int b = 0; b < myBlocks; ++b) {
                const unsigned char* cur = ring + stage * STAGE;
                const int t = t0 + DIR * b * SS;
                const int after = stage + 1 == stages ? 0 : stage + 1;
                const uint32_t afterParity = after == 0 ? parity ^ 1 : parity;
                const bool ready = b + 1 == myBlocks || lpBarTry(barAddr + 8 * after, afterParity);
                step(t, std::integral_constant<int, 0>{}, cur + REC);
                step(t, std::integral_constant<int, 1>{}, cur + 2 * REC);
                step(t, std::integral_constant<int, 2>{}, cur + 3 * REC);
                // the block's records are in registers: hand its stage back
                ++block;
                __syncwarp();
                if (lane == 0) consumed[warp] = block;
                stage = after;
                parity = afterParity;
                if (!ready) lpBarWait(barAddr + 8 * stage, parity, &stopFlag, a.err, waitNs);
                step(t, std::integral_constant<int, SS - 1>{}, ring + stage * STAGE);
                yIn += yInStep;
                yOut += yOutStep;
                dst += DIR * SS;
                vt += DIR * SS * 32;
            }
        };
        sweep(std::integral_constant<int, 1>{});
        sweep(std::integral_constant<int, -1>{});
    }
    // no CTA may leave while another can still write into its shared memory
    cluster.sync();
}

static void spConfig(const StencilPackPlan& p, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr)
{
    cfg.gridDim = dim3(p.ctas);
    cfg.blockDim = dim3((p.warps + 1) * 32);
    cfg.dynamicSmemBytes = spSmem(p.steps, p.warps, p.stages).total;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

// Two warps per CTA (one where the lines are too long for two): the producer warp and each
// sweeping warp then have a sub-partition of their own.
StencilPackPlan makeStencilPackPlan(const StencilArgs& a)
{
    StencilPackPlan best{};
    if (a.b != 1 || a.S != 9 || a.nx < 1 || a.ny < 1) return best;
    DXG_CUDA(cudaFuncSetAttribute(stencilPackApply, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    DXG_CUDA(cudaFuncSetAttribute(stencilPackApply, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSpSmemLimit));
    for (int w : {2, 1}) {
        StencilPackPlan p{};
        p.warps = w;
        p.ctas = (a.ny + w * kSpLines - 1) / (w * kSpLines);
        if (p.ctas > 16) continue;
        p.steps = spSteps(a.nx, std::min(kSpLines, a.ny));
        p.stages = kSpMaxStages;
        while (p.stages > 1 && spSmem(p.steps, w, p.stages).total > kSpSmemLimit) --p.stages;
        if (p.stages < 2) continue;
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr[1];
        spConfig(p, cfg, attr);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, stencilPackApply, &cfg) != cudaSuccess) {
            cudaGetLastError();
            continue;
        }
        p.ok = fit > 0;
        if (p.ok) return p;
    }
    return best;
}

size_t stencilPackBytes(const StencilPackPlan& p, int dir)
{
    return (size_t)p.ctas * p.warps * p.steps * (dir > 0 ? kSpFwd : kSpBwd) * 32 * 8;
}

void launchStencilPack(const StencilArgs& a, const StencilPackPlan& p, cudaStream_t st)
{
    const int64_t total = (int64_t)p.ctas * p.warps * p.steps * 32;
    stencilPackKernel<<<dim3((unsigned)std::min<int64_t>((total + 255) / 256, 2048), 2), 256, 0, st>>>(a, p);
    DXG_CUDA(cudaGetLastError());
}

void launchStencilPackApply(const StencilArgs& a, const StencilPackPlan& p, const double* d, double* v, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    spConfig(p, cfg, attr);
    cfg.stream = st;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    DXG_CUDA(cudaLaunchKernelEx(&cfg, stencilPackApply, a, p, d, v));
}

}  // namespace dxg
