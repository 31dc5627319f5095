// lanepack.cu -- natural-order ILU(0) triangular solves of cc-TPFA systems (2D and 3D, 1x1 and
// 2x2 blocks) in one launch: the forward and the backward sweep over packed factor records.
//
// What bounds the sweeps: a chain of nx+ny+nz-2 dependent levels each way.  On GB300 a
// dependent FP64 FMA takes 64 cycles and an FP64 warp instruction holds its SM sub-partition as
// long, so a level costs at least (dim x block size) x 64 cycles; with FP32 factors the chain is
// ~25 cycles and everything else a step does is what it costs.  So a step is kept to the chain:
//   * the factor is re-laid once per factorisation (lanePackKernel) into the order the sweeps
//     read it, one contiguous record per warp and step with zeros for lanes without a cell; a
//     producer warp streams the records into a shared-memory ring with bulk copies, so a
//     sweeping warp issues no global loads, addresses or predicates for them;
//   * a lane reads the record of the next step while it works on this one;
//   * the sweep's right-hand side is copied into shared memory at the start, overwritten there
//     by the forward results and read back by the same lane in the backward sweep;
//   * neighbour values arrive in histories indexed by the consumer's own step, zero where a
//     lane has no cell, so polls need no predicates; lanes without a hand-off poll a zero;
//   * a zero multiplier times a zero value leaves the accumulator's bits, so there is no
//     branch on missing neighbours.
//
// Mapping: a lane holds R rows of one grid line (R = 1: FP64, whose row chains run best on
// lanes of their own; R = B: FP32), 32 R / B lines per warp; line j handles cell x = t - j at
// the warp's step t, forward with t ascending, backward with t descending.  A CTA holds a tile
// of W warps of one z-plane; tiles and planes are spread over thread-block clusters, all of them
// resident.  Dependencies of cell (x, y, z), all of the level before (mirrored backward):
//   * x: the lane's previous result (R < B: the other row by shuffle);
//   * y: inside a warp by shuffle; across warps the boundary line's results in a shared-memory
//     history; across CTAs of a plane the same history by remote stores;
//   * z: the neighbouring plane is another CTA: inside a cluster its results are stored straight
//     into this CTA's history [step][lane] (same step and lane on both sides); across clusters
//     they go through a hand-off buffer in global memory, prefetched a ring depth ahead by a
//     consumer that starts once its producer is that far ahead.
// A plane starts its backward sweep as soon as its forward sweep is done (one cluster barrier:
// the z history is used in both directions), so the turn costs no launch.
// So a cluster waits for clusters of lower and of higher index, and a launch whose clusters are not
// all resident would wait for itself: the plan counts them (cudaOccupancyMaxActiveClusters), a
// batched launch takes no more problems than fit, and a launch of several clusters is a cooperative
// one, which CUDA runs with all its CTAs resident whatever else the GPU is doing.  (The count
// alone does not give that: placed around the CTAs of the kernel before it or of another stream,
// the clusters leave gaps that no cluster fits.  4x4x700 cells, FP64 1x1: 88 clusters of 8 where
// 89 fit, and the waits of a plain dependent launch expired.  The attribute costs nothing: 24
// iterations on 64x64x32 FP64 take 7.52 ms either way.)
// Every history starts filled with an all-ones pattern (a NaN that no arithmetic produces)
// which the consumer waits to see replaced: each entry is one aligned 4- or 8-byte relaxed
// store, seen whole, so no fence, flag or barrier sits on the chain.  The consumer puts the
// pattern back into the z history and the global hand-off buffer.  Waits are bounded: one that
// expires records DXG_ERR_TIMEOUT and stops the CTA's sweep (its remaining waits return at once).
//
// The arithmetic per row is that of wave.cu (same operands, same order, explicit FMAs), so the
// results are those of the cluster wavefront bit for bit.
//
// Measured per apply against the lane sweeps that read the factor in place (lanewave.cu) and the
// cluster wavefront: 64x64x32, 2x2 blocks, FP64 0.129 ms (0.195, 0.345), FP32 0.068 ms (0.156,
// 0.207); 45x37x23 FP32 0.049 ms (0.097, 0.152); 100x100 1x1 FP64 0.056 ms (0.193 for the
// wavefront).  A 64x64 plane alone takes 0.35 us a step in FP64 (its FMA chain: 0.23 us) and
// 0.18 us in FP32.
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"
#include "handoff.cuh"
#include "linalg.cuh"
#include "wave.cuh"

namespace cg = cooperative_groups;

namespace dxg {

namespace {

constexpr int kLpMaxWarps = 4;
constexpr size_t kLpSmemLimit = 226 * 1024;

// values of one lane's record: the off-diagonal rows in the order x, y, z, then (backward) the
// rows of the inverted pivot
template <int B, int R, int DIR, int DIM>
struct LpRec {
    static constexpr int n = R * B * (DIM + (DIR < 0 ? 1 : 0));
};
// rows of a line that one lane holds
template <class T, int B>
constexpr int lpRows() { return sizeof(T) == 8 ? 1 : B; }

// steps per stage of the record ring (two where shared memory is short), its largest depth in
// stages, and the depth in steps of the ring of hand-offs across clusters
template <class T, int B, int DIM>
constexpr int lpStageSteps() { return sizeof(T) == 8 && B == 2 && DIM == 3 ? 2 : 4; }
constexpr int kLpMaxStages = 8;
template <class T>
constexpr int lpZDepth() { return sizeof(T) == 8 ? 4 : 8; }

// steps of a warp's sweep at most, padded to whole stages
inline int lpSteps(int nx, int linesPerWarp) { return (nx + linesPerWarp - 1 + 3) / 4 * 4; }

struct LpSmem {
    size_t ring, vbuf, zin, zring, ybuf, zero, sink, total;
};
// ring [W][stages][stage], vbuf and zin [W][steps][32 R], zring [W][depth][32 R], ybuf
// [2 directions][W + 1][pad + steps][B] (entry W: from the neighbouring CTA; pad: room for the
// boundary line's steps without a cell), and for the lanes without a hand-off zeros to poll and
// a sink to store to (of a block's steps either way)
__host__ __device__ inline int lpYPad(int B, int R) { return 32 * R / B; }
__host__ __device__ inline LpSmem lpSmem(int steps, int W, int stages, int stageSteps, int B, int R, int dim, int tsize)
{
    LpSmem s{};
    size_t o = 0;
    s.ring = o;
    o += (size_t)W * stages * stageSteps * (R * B * (dim + 1) * 32 * tsize);
    s.vbuf = o;
    o += (size_t)W * steps * 32 * R * tsize;
    s.zin = o;
    if (dim == 3) o += (size_t)W * steps * 32 * R * tsize;
    s.zring = o;
    if (dim == 3) o += (size_t)W * 8 * 32 * R * tsize;
    s.ybuf = o;
    o += (2 * (size_t)(W + 1) * (lpYPad(B, R) + steps) + lpYPad(B, R)) * B * tsize;
    o = (o + 15) & ~(size_t)15;
    s.zero = o;
    o += 64 * (size_t)tsize;
    s.sink = o;
    o += (size_t)2 * stageSteps * 32 * R * tsize;
    s.total = o;
    return s;
}

// lane `lane` of warp w of CTA `cta`: its plane, line, line within the warp and first row
struct LpWhere {
    int z, y, j, r;
};
template <int B, int R>
__device__ __forceinline__ LpWhere lpWhere(int cta, int nyb, int W, int w, int lane)
{
    constexpr int per = B / R, lpw = 32 / per;
    LpWhere p;
    p.z = cta / nyb;
    p.j = lane / per;
    p.r = lane % per * R;
    p.y = (cta % nyb) * W * lpw + w * lpw + p.j;
    return p;
}

}  // namespace

// The packed records of both sweeps from the factor (L, A's upper slots, Dinv): per sweep
// (blockIdx.y) one thread per (CTA, warp, step, lane); zeros where the lane has no cell or no
// neighbour.  The backward records run in the order of the backward steps.  Bandwidth bound: the
// factor read once and the records written once (64x64x32, 2x2 blocks, FP64: 20 us for 66 MB).
template <class T, int B, int DIR, int DIM>
__device__ __forceinline__ void lpPackSweep(const LanePackArgs<T>& a, int64_t first, int64_t stride)
{
    constexpr int R = lpRows<T, B>();
    constexpr int NV = LpRec<B, R, DIR, DIM>::n;
    constexpr int BB = B * B;
    const int64_t total = (int64_t)a.ctas * a.warps * a.steps * 32;
    for (int64_t k = first; k < total; k += stride) {
        const int lane = (int)(k & 31);
        const int64_t rec = k >> 5;
        const int s = (int)(rec % a.steps);
        const int64_t cw = rec / a.steps;
        const int w = (int)(cw % a.warps), cta = (int)(cw / a.warps);
        const LpWhere p = lpWhere<B, R>(cta, a.nyb, a.warps, w, lane);
        const int x = (DIR > 0 ? s : a.steps - 1 - s) - p.j;
        T out[NV];
#pragma unroll
        for (int e = 0; e < NV; ++e) out[e] = 0;
        if (p.y < a.ny && x >= 0 && x < a.nx) {
            const int64_t i = ((int64_t)p.z * a.ny + p.y) * a.nx + x;
            // slots: -z -y -x centre +x +y +z (2D without z)
            const int c[3] = {x, p.y, p.z}, n[3] = {a.nx, a.ny, a.nz};
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int ax = 0; ax < DIM; ++ax) {
                    if (c[ax] == (DIR > 0 ? 0 : n[ax] - 1)) continue;
                    const T* row = (DIR > 0 ? a.Lf + ((int64_t)(DIM - 1 - ax) * a.N + i) * BB
                                            : a.A + ((int64_t)(DIM + 1 + ax) * a.N + i) * BB) + (p.r + r) * B;
#pragma unroll
                    for (int e = 0; e < B; ++e) out[(ax * R + r) * B + e] = lpEntry(row[e]);
                }
                if (DIR < 0)
#pragma unroll
                    for (int e = 0; e < B; ++e) out[(DIM * R + r) * B + e] = lpEntry(a.Dinv[i * BB + (p.r + r) * B + e]);
            }
        }
        unsigned char* dst = a.pack[DIR > 0 ? 0 : 1] + rec * (NV * 32 * (int64_t)sizeof(T));
#pragma unroll
        for (int e = 0; e < NV; ++e) *reinterpret_cast<T*>(dst + lpValueOffset<T, NV>(e, lane)) = out[e];
    }
}
template <class T, int B, int DIM>
__global__ void __launch_bounds__(256) lanePackKernel(LanePackArgs<T> a)
{
    const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (blockIdx.y == 0) lpPackSweep<T, B, 1, DIM>(a, first, stride);
    else lpPackSweep<T, B, -1, DIM>(a, first, stride);
}

// v = (LU)^-1 rhs: z_i = d_i - L_ix z_x - L_iy z_y - L_iz z_z, then
// y_i = D_i^-1 (z_i - U_ix y_x - U_iy y_y - U_iz y_z).
// BATCH: block k works as CTA map[k].y of problem map[k].x (whole clusters per problem).
template <class T, int B, int DIM, bool BATCH>
__global__ void __launch_bounds__((kLpMaxWarps + 1) * 32) lanePackApply(LanePackArgs<T> a0, const LanePackArgs<T>* batch,
                                                                        const uint2* map)
{
    uint2 who = make_uint2(0u, blockIdx.x);
    if constexpr (BATCH) {
        who = map[blockIdx.x];
        a0 = batch[who.x];
    }
    const LanePackArgs<T>& a = a0;
    constexpr int R = lpRows<T, B>();
    constexpr int NF = LpRec<B, R, 1, DIM>::n, NB = LpRec<B, R, -1, DIM>::n;
    constexpr int TS = (int)sizeof(T);
    constexpr int LPW = 32 * R / B;          // lines per warp
    constexpr int SLAB = 32 * R;             // values of one step of a warp
    constexpr int SS = lpStageSteps<T, B, DIM>(), ZD = lpZDepth<T>();
    constexpr int STAGE = SS * NB * 32 * TS;   // bytes of a ring stage (the larger, backward records)
    constexpr int YP = LPW;                  // padding of the y histories
    extern __shared__ __align__(128) unsigned char lpRaw[];
    __shared__ int stopFlag;
    __shared__ volatile int consumed[kLpMaxWarps];   // blocks each warp has read out of its ring
    __shared__ __align__(8) unsigned long long bars[kLpMaxWarps][kLpMaxStages];

    cg::cluster_group cluster = cg::this_cluster();
    // Every hand-off inside a cluster goes to a rank of the plan's: launched with other clusters (a
    // profiler repeats a cooperative launch without its cluster dimension) the kernel does nothing and
    // says so, and the solve goes on with the sweeps that read the factor in place.
    if (cluster.num_blocks() != (unsigned)a.clusterSize) {
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (threadIdx.x == 0) atomicExch(a.err, DXG_ERR_CUDA);
        return;
    }
    const int nx = a.nx, ny = a.ny, W = a.warps, steps = a.steps, stages = a.stages;
    const LpSmem lay = lpSmem(steps, W, stages, SS, B, R, DIM, TS);
    const int cta = (int)who.y;
    const int lane = threadIdx.x & 31;
    // through a shuffle, so that what depends on it is known to be uniform over the warp
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    const bool working = cta < a.ctas;
    // the last warp fetches the records; a batched launch has more sweeping warps than some of its
    // problems use
    const bool producer = warp == (BATCH ? (int)(blockDim.x >> 5) - 1 : W), idle = BATCH && !producer && warp >= W;
    const LpWhere p = lpWhere<B, R>(working ? cta : 0, a.nyb, W, warp, lane);
    const int yb = working ? cta % a.nyb : 0;
    const bool lineOk = working && !producer && !idle && p.y < ny;
    const int cs = a.clusterSize;
    // neighbouring CTAs: the planes below and above, the tiles before and after in y
    const int zLo = cta - a.nyb, zHi = cta + a.nyb;
    const bool hasZLo = DIM == 3 && working && p.z > 0, hasZHi = DIM == 3 && working && zHi < a.ctas;
    const bool zLoLocal = hasZLo && zLo / cs == cta / cs, zHiLocal = hasZHi && zHi / cs == cta / cs;
    const bool hasYLo = working && yb > 0, hasYHi = working && yb + 1 < a.nyb;
    const int tileLine = yb * W * LPW;       // first line of this CTA
    const int blocks = steps / SS;           // record blocks of one warp and sweep ...
    // ... and how many of them hold cells: a warp with fewer lines ends (and starts back) early
    auto blocksOf = [&](int w) {
        const int lines = min(LPW, ny - (tileLine + w * LPW));
        return lines > 0 ? (nx + lines - 1 + SS - 1) / SS : 0;
    };

    T* const zin = reinterpret_cast<T*>(lpRaw + lay.zin);
    T* const ybuf = reinterpret_cast<T*>(lpRaw + lay.ybuf);
    const int yRow = (YP + steps) * B, yDir = (W + 1) * yRow;

    // the histories: empty where a value will arrive, zero where the lane has no cell
    if (!producer && !idle) {
        if (DIM == 3)
            for (int t = 0; t < steps; ++t) {
                const int x = t - p.j;
                const T v = zLoLocal && lineOk && x >= 0 && x < nx ? lpEmpty<T>() : T(0);
#pragma unroll
                for (int r = 0; r < R; ++r) zin[((size_t)warp * steps + t) * SLAB + lane * R + r] = v;
            }
        for (int k = threadIdx.x; k < 2 * yDir; k += W * 32) {
            // forward entries hold cell x = t of the line before, backward ones x = t - (LPW - 1)
            // of the line after (t counted behind the padding)
            const int t = (k / B) % (YP + steps) - YP, x = t - (k < yDir ? 0 : LPW - 1);
            ybuf[k] = x >= 0 && x < nx ? lpEmpty<T>() : T(0);
        }
        T* zero = reinterpret_cast<T*>(lpRaw + lay.zero);
        for (int k = threadIdx.x; k < 64; k += W * 32) zero[k] = 0;
        if (lane < kLpMaxStages) lpBarInit(lpAddr(&bars[warp][lane]));
        if (lane == 0) consumed[warp] = 0;
    } else if (producer && lane == 0) {
        stopFlag = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cluster.sync();
    // This launch is a programmatic dependent of the kernel before it: its CTAs may have been
    // filling their histories while that one ran.  Wait until it has completed and its writes
    // (the right-hand side, the Krylov state) are visible.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool skip = a.ks && a.ks->status != KS_RUNNING;

    if (producer || idle) {
        // barrier 2 of 3 (the turn): nothing of this warp's orders with it
        asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
        if (producer && lane == 0 && working && !skip) {
            int issued[kLpMaxWarps];
#pragma unroll
            for (int w = 0; w < kLpMaxWarps; ++w) issued[w] = 0;
            bool more = true;
            while (more) {
                more = false;
#pragma unroll
                for (int w = 0; w < kLpMaxWarps; ++w) {
                    const int n = w < W ? blocksOf(w) : 0;
                    if (issued[w] >= 2 * n) continue;
                    more = true;
                    if (issued[w] - consumed[w] >= stages) continue;
                    const int b = issued[w]++;
                    const bool fwd = b < n;
                    const uint32_t bytes = SS * (fwd ? NF : NB) * 32 * TS;
                    const size_t at = (((size_t)cta * W + w) * blocks + (fwd ? b : b - n + blocks - n)) * bytes;
                    const int st = b % stages;
                    lpBulk(lpAddr(lpRaw + lay.ring + ((size_t)w * stages + st) * STAGE), a.pack[fwd ? 0 : 1] + at, bytes,
                           lpAddr(&bars[w][st]));
                }
                __nanosleep(64);
            }
        }
        __syncwarp();
        asm volatile("barrier.cluster.wait;" ::: "memory");
    } else {
        const bool warpWorks = working && !skip && tileLine + warp * LPW < ny;
        unsigned char* const ring = lpRaw + lay.ring + (size_t)warp * stages * STAGE;
        const uint32_t barAddr = lpAddr(&bars[warp][0]);
        T* const vb = reinterpret_cast<T*>(lpRaw + lay.vbuf) + (size_t)warp * steps * SLAB + lane * R;   // + t * SLAB
        const int jx = lineOk ? p.j : 0x40000000;   // t - jx: the lane's cell, when below nx unsigned
        const int64_t lineBase = lineOk ? ((int64_t)p.z * ny + p.y) * nx : 0;
        const size_t slab = ((size_t)(working ? cta : 0) * W + warp) * steps * SLAB;
        const size_t handoffDir = (size_t)a.ctas * W * steps * SLAB;
        unsigned long long deadlineOfWait = 0, *const deadline = &deadlineOfWait;
        const int lineOff = p.j * B;             // this line's entry within a slab
        const int myBlocks = blocksOf(warp);
        int block = 0, stage = 0;                // of the record ring, over both sweeps
        uint32_t parity = 0;

        if (warpWorks) {
            // the right-hand side, zeros where the lane has no cell
            const T* src = a.rhs + lineBase * B + p.r;
            for (int t = 0; t < myBlocks * SS; ++t) {
                const int x = t - jx;
                const bool valid = (unsigned)x < (unsigned)nx;
                lpCpAsync<R * TS>(lpAddr(vb + t * SLAB), valid ? src + (int64_t)x * B : src, valid);
            }
            lpCommit();
        }

        auto sweep = [&](auto dirC, auto viaGlobal) {
            constexpr int DIR = decltype(dirC)::value;
            constexpr bool GZ = decltype(viaGlobal)::value;
            constexpr int NV = DIR > 0 ? NF : NB;
            constexpr int REC = NV * 32 * TS;
            const bool yEdge = p.j == (DIR > 0 ? 0 : LPW - 1);
            [[maybe_unused]] const bool up = DIR > 0 ? zLoLocal : zHiLocal;   // z values arrive in zin
            const bool downLocal = DIR > 0 ? zHiLocal : zLoLocal, down = DIR > 0 ? hasZHi : hasZLo;
            const int downCta = DIR > 0 ? zHi : zLo;
            const int t0 = DIR > 0 ? 0 : myBlocks * SS - 1;              // first slot of the sweep
            // where the y and z neighbour values arrive, per step of this warp
            const int yWarp = DIR > 0 ? (warp > 0 ? warp - 1 : W) : (warp < W - 1 ? warp + 1 : W);
            const bool ySrc = yEdge && lineOk &&
                              (DIR > 0 ? warp > 0 || hasYLo : (warp < W - 1 ? p.y + 1 < ny : hasYHi));
            T* const yDirBuf = ybuf + (DIR > 0 ? 0 : yDir) + YP * B;
            uint32_t yIn = ySrc ? lpAddr(yDirBuf + yWarp * yRow + t0 * B) : lpAddr(lpRaw + lay.zero) + 32 * TS;
            const uint32_t yInStep = ySrc ? (uint32_t)(DIR * SS * B * TS) : 0u;
            uint32_t zIn = lpAddr(zin + ((size_t)warp * steps + t0) * SLAB + lineOff);
            T* const zFrom = a.handoff + (DIR > 0 ? 0 : handoffDir) + slab;
            // ... and where this lane's results go: what a lane has no hand-off for goes to a sink
            // (every lane stores every step; steps without a cell store a zero to a slot that holds
            // one or is padding)
            const uint32_t sink = lpAddr(lpRaw + lay.sink);
            const bool yPub = lineOk && p.j == (DIR > 0 ? LPW - 1 : 0) &&
                              (DIR > 0 ? warp < W - 1 || hasYHi : warp > 0 || hasYLo);
            const bool yFar = DIR > 0 ? warp == W - 1 && hasYHi : warp == 0 && hasYLo;   // to another CTA
            uint32_t yOut = sink + SS * SLAB * TS;
            const uint32_t yOutStep = yPub ? (uint32_t)(DIR * SS * B * TS) : 0u;
            if (yPub) {
                const uint32_t to = lpAddr(yDirBuf + (yFar ? W : warp) * yRow);
                yOut = (yFar ? lpMapa(to, (cta + DIR) % cs) : to) +
                       (uint32_t)((((DIR > 0 ? -(LPW - 1) : LPW - 1) + t0) * B + p.r) * TS);   // x = t - j
            } else if (yFar) {
                yOut = lpMapa(yOut, cta % cs);
            }
            uint32_t zOut = lpMapa(downLocal ? lpAddr(zin + ((size_t)warp * steps + t0) * SLAB + lane * R)
                                             : sink + SS * SLAB * TS,
                                   downLocal ? downCta % cs : cta % cs);
            const uint32_t zOutStep = downLocal ? (uint32_t)(DIR * SS * SLAB * TS) : 0u;
            uint32_t zOwn = lpAddr(zin + ((size_t)warp * steps + t0) * SLAB + lane * R);
            T* const zTo = a.handoff + (DIR > 0 ? 0 : handoffDir) +
                           ((size_t)max(downCta, 0) * W + warp) * steps * SLAB + lane * R;
            T* dst = a.v + (lineBase + t0 - p.j) * B + p.r;   // dereferenced where the lane has a cell
            T* vt = vb + t0 * SLAB;

            const T* const zring = reinterpret_cast<const T*>(lpRaw + lay.zring) + (size_t)warp * ZD * SLAB;
            const uint32_t zringAddr = lpAddr(zring) + 16 * lane;
            // copies of slot t's hand-offs across clusters, one group per step
            auto fetchZ = [&](int t) {
                if (t >= 0 && t < steps && lane < SLAB * TS / 16)
                    lpCpAsync16(zringAddr + (t & (ZD - 1)) * (SLAB * TS),
                                reinterpret_cast<const unsigned char*>(zFrom + (size_t)t * SLAB) + 16 * lane);
                lpCommit();
            };
            if constexpr (GZ) {
                // start once the producer is a ring depth ahead, so that the prefetched entries
                // of the steps that follow hold their values: line 0 (forward) or the warp's
                // last line (backward) of a slot that many cells on
                const int lines = min(LPW, ny - (tileLine + warp * LPW));
                const int on = min(ZD + 1, nx - 1);
                const T* w = DIR > 0 ? zFrom + (size_t)on * SLAB
                                     : zFrom + (size_t)(nx - 1 + lines - 1 - on) * SLAB + (lines - 1) * B;
                LpVal<T, B> first = lpLdGpu<T, B>(w);
                lpPoll<T, B>(first, [&] { return lpLdGpu<T, B>(w); }, deadline, &stopFlag, a.err, a.waitNs);
#pragma unroll 1
                for (int k = 0; k < ZD; ++k) fetchZ(t0 + DIR * k);
                lpCpWait<ZD - 1>();
                __syncwarp();
            }
            if (!lpBarTry(barAddr + 8 * stage, parity)) lpBarWait(barAddr + 8 * stage, parity, &stopFlag, a.err, a.waitNs);
            // the record and the vector entry of the step at hand, loaded a step ahead
            T c[NV], cV[R], prev[R];
            LpVal<T, B> cz{};
            lpLoadRec<T, NV>(ring + stage * STAGE, lane, c);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                cV[r] = vt[r];
                prev[r] = 0;
            }
            if constexpr (GZ)
#pragma unroll
                for (int e = 0; e < B; ++e) cz.v[e] = zring[(t0 & (ZD - 1)) * SLAB + lineOff + e];

            // step KC of a block whose first slot is t; `next`: the record of the step that follows
            auto step = [&](int tBlock, auto kC, const unsigned char* next) {
                constexpr int K = DIR * decltype(kC)::value;
                const int t = tBlock + K;
                T xv[B], yv[B], acc[R];
                if constexpr (R < B) {
                    // both rows of this line and of the neighbour line, each by a shuffle of its own
                    // (a select between this row and the other would follow the shuffle on the chain)
#pragma unroll
                    for (int e = 0; e < B; ++e) xv[e] = __shfl_sync(0xffffffffu, prev[0], (lane & ~1) + e);
#pragma unroll
                    for (int e = 0; e < B; ++e) yv[e] = __shfl_sync(0xffffffffu, prev[0], ((lane & ~1) - 2 * DIR + e) & 31);
                } else {
#pragma unroll
                    for (int e = 0; e < B; ++e) {
                        xv[e] = prev[e];
                        yv[e] = DIR > 0 ? __shfl_up_sync(0xffffffffu, prev[e], 1)
                                        : __shfl_down_sync(0xffffffffu, prev[e], 1);
                    }
                }
                LpVal<T, B> yp = lpLdShared<T, B, K * B * TS>(yIn);
                [[maybe_unused]] LpVal<T, B> zv{}, nz{};
                T n[NV], nV[R];
                lpLoadRec<T, NV>(next, lane, n);
                // slot t + DIR; at a sweep's end a slot of the neighbouring buffers, not used
#pragma unroll
                for (int r = 0; r < R; ++r) nV[r] = vt[(K + DIR) * SLAB + r];
                auto term = [&](int at, const T (&v)[B]) {
#pragma unroll
                    for (int e = 0; e < B; ++e)
#pragma unroll
                        for (int r = 0; r < R; ++r) acc[r] = fma(-c[(at + r) * B + e], v[e], acc[r]);
                };
#pragma unroll
                for (int r = 0; r < R; ++r) acc[r] = cV[r];
                term(0, xv);
                lpPoll<T, B>(yp, [&] { return lpLdShared<T, B, K * B * TS>(yIn); }, deadline,
                             &stopFlag, a.err, a.waitNs);
                // the z values are looked at as late as the chain allows: a plane follows the one
                // before it that much closer
                if constexpr (DIM == 3 && !GZ) zv = lpLdShared<T, B, K * SLAB * TS>(zIn);
#pragma unroll
                for (int e = 0; e < B; ++e) yv[e] = yEdge ? yp.v[e] : yv[e];
                term(R, yv);
                const bool act = (unsigned)(t - jx) < (unsigned)nx;
                if constexpr (DIM == 3) {
                    if constexpr (GZ) {
                        fetchZ(t + DIR * ZD);
                        lpCpWait<ZD - 1>();
                        __syncwarp();
                        T* src = zFrom + (size_t)t * SLAB;
#pragma unroll
                        for (int e = 0; e < B; ++e) {
                            zv.v[e] = act ? cz.v[e] : T(0);
                            nz.v[e] = zring[((t + DIR) & (ZD - 1)) * SLAB + lineOff + e];
                        }
                        lpPoll<T, B>(zv, [&] {
                            LpVal<T, B> v = lpLdGpu<T, B>(src + lineOff);
#pragma unroll
                            for (int e = 0; e < B; ++e) v.v[e] = act ? v.v[e] : T(0);
                            return v;
                        }, deadline, &stopFlag, a.err, a.waitNs);
                        // every lane of the line holds its values: put the pattern back
                        if (act)
#pragma unroll
                            for (int r = 0; r < R; ++r) lpStGpu<T>(src + lane * R + r, lpEmpty<T>());
                    } else {
                        // (the poll also orders the two lanes' reads of an entry before its reset)
                        lpPoll<T, B>(zv, [&] { return lpLdShared<T, B, K * SLAB * TS>(zIn); },
                                     deadline, &stopFlag, a.err, a.waitNs);
                    }
                    term(2 * R, zv.v);
                }
                T res[R];
                if constexpr (DIR > 0) {
#pragma unroll
                    for (int r = 0; r < R; ++r) res[r] = acc[r];
                } else {
                    T full[B];
                    if constexpr (R < B) {
#pragma unroll
                        for (int e = 0; e < B; ++e) full[e] = __shfl_sync(0xffffffffu, acc[0], (lane & ~1) + e);
                    } else {
#pragma unroll
                        for (int e = 0; e < B; ++e) full[e] = acc[e];
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        res[r] = c[(DIM * R + r) * B] * full[0];
#pragma unroll
                        for (int e = 1; e < B; ++e) res[r] = fma(c[(DIM * R + r) * B + e], full[e], res[r]);
                    }
                }
                auto publish = [&](auto rC) {
                    constexpr int r = decltype(rC)::value;
                    if constexpr (DIM == 3) {
                        lpStRemote<K * SLAB * TS + r * TS>(zOut, res[r]);
                        if (DIR > 0) lpStShared<K * SLAB * TS + r * TS>(zOwn, act && up ? lpEmpty<T>() : T(0));
                    }
                    if (yFar) lpStRemote<K * B * TS + r * TS>(yOut, res[r]);
                    else lpStShared<K * B * TS + r * TS>(yOut, res[r]);
                    if (DIR > 0) vt[K * SLAB + r] = res[r];
                    else if (act) dst[K * B + r] = res[r];
                    prev[r] = res[r];
                };
                publish(std::integral_constant<int, 0>{});
                if constexpr (R > 1) publish(std::integral_constant<int, 1>{});
                if (DIM == 3 && !downLocal && down && act)
#pragma unroll
                    for (int r = 0; r < R; ++r) lpStGpu<T>(zTo + (size_t)t * SLAB + r, res[r]);
#pragma unroll
                for (int e = 0; e < NV; ++e) c[e] = n[e];
#pragma unroll
                for (int r = 0; r < R; ++r) cV[r] = nV[r];
                cz = nz;
            };
            for (int b = 0; b < myBlocks; ++b) {
                const unsigned char* cur = ring + stage * STAGE;
                const int t = t0 + DIR * b * SS;
                const int after = stage + 1 == stages ? 0 : stage + 1;
                const uint32_t afterParity = after == 0 ? parity ^ 1 : parity;
                const bool ready = b + 1 == myBlocks || lpBarTry(barAddr + 8 * after, afterParity);
                step(t, std::integral_constant<int, 0>{}, cur + REC);
                if constexpr (SS == 4) {
                    step(t, std::integral_constant<int, 1>{}, cur + 2 * REC);
                    step(t, std::integral_constant<int, 2>{}, cur + 3 * REC);
                }
                // the block's records are in registers: hand its stage back
                ++block;
                __syncwarp();
                if (lane == 0) consumed[warp] = block;
                stage = after;
                parity = afterParity;
                if (!ready) lpBarWait(barAddr + 8 * stage, parity, &stopFlag, a.err, a.waitNs);
                step(t, std::integral_constant<int, SS - 1>{}, ring + stage * STAGE);
                yIn += yInStep;
                zIn += (uint32_t)(DIR * SS * SLAB * TS);
                zOut += zOutStep;
                zOwn += (uint32_t)(DIR * SS * SLAB * TS);
                yOut += yOutStep;
                dst += DIR * SS * B;
                vt += DIR * SS * SLAB;
            }
            if constexpr (GZ) lpCpWait<0>();
        };
        using Fwd = std::integral_constant<int, 1>;
        using Bwd = std::integral_constant<int, -1>;
        if (warpWorks) {
            lpCpWait<0>();
            if (DIM == 3 && hasZLo && !zLoLocal) sweep(Fwd{}, std::true_type{});
            else sweep(Fwd{}, std::false_type{});
        }
        // the turn: z histories that no forward values arrived in start empty for the backward ones,
        // the others have been put back (barrier 2 of 3)
        if (DIM == 3 && zHiLocal && !zLoLocal && warpWorks)
            for (int t = 0; t < steps; ++t) {
                const T v = (unsigned)(t - jx) < (unsigned)nx ? lpEmpty<T>() : T(0);
#pragma unroll
                for (int r = 0; r < R; ++r) zin[((size_t)warp * steps + t) * SLAB + lane * R + r] = v;
            }
        if (DIM == 3 && zLoLocal && !zHiLocal && warpWorks)
            for (int t = 0; t < steps; ++t)
#pragma unroll
                for (int r = 0; r < R; ++r) zin[((size_t)warp * steps + t) * SLAB + lane * R + r] = 0;
        asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
        if (warpWorks) {
            if (DIM == 3 && hasZHi && !zHiLocal) sweep(Bwd{}, std::true_type{});
            else sweep(Bwd{}, std::false_type{});
        }
    }
    // no CTA may leave while another can still write into its shared memory
    cluster.sync();
}

// ---------------------------------------------------------------- host side
namespace {

// One problem's launch, a batched one (map), or with `fits` the number of its clusters that are
// resident at once.
struct LpShape {
    unsigned grid;
    int clusterSize, warps;
    size_t smem;
};
template <class T, int B, int DIM, bool BATCH>
cudaError_t lpLaunch(const LpShape& p, const LanePackArgs<T>& a, const LanePackArgs<T>* batch, const uint2* map,
                     cudaStream_t st, int* fits)
{
    auto kern = lanePackApply<T, B, DIM, BATCH>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLpSmemLimit);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.grid);
    cfg.blockDim = dim3((p.warps + 1) * 32);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[3];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.clusterSize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    // the clusters wait for one another: all of them resident
    attr[2].id = cudaLaunchAttributeCooperative;
    attr[2].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = fits ? 1 : p.grid > (unsigned)p.clusterSize ? 3 : 2;
    if (fits) {
        int n = 0;
        e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
        *fits = e == cudaSuccess ? n : 0;
        if (e != cudaSuccess) cudaGetLastError();
        return cudaSuccess;
    }
    return cudaLaunchKernelEx(&cfg, kern, a, batch, map);
}
template <class T, bool BATCH>
cudaError_t lpDispatch(int dim, int b, const LpShape& s, const LanePackArgs<T>& a, const LanePackArgs<T>* batch,
                       const uint2* map, cudaStream_t st, int* fits)
{
    if (dim == 3)
        return b == 2 ? lpLaunch<T, 2, 3, BATCH>(s, a, batch, map, st, fits)
                      : lpLaunch<T, 1, 3, BATCH>(s, a, batch, map, st, fits);
    return b == 2 ? lpLaunch<T, 2, 2, BATCH>(s, a, batch, map, st, fits)
                  : lpLaunch<T, 1, 2, BATCH>(s, a, batch, map, st, fits);
}
template <class T>
int lpStepsPerStage(int dim, int b)
{
    return dim == 3 ? (b == 2 ? lpStageSteps<T, 2, 3>() : lpStageSteps<T, 1, 3>()) : lpStageSteps<T, 1, 2>();
}
template <class T>
size_t lpSmemOf(const LanePackPlan& p)
{
    return lpSmem(p.steps, p.warps, p.stages, lpStepsPerStage<T>(p.dim, p.b), p.b, p.rows, p.dim, (int)sizeof(T)).total;
}
}  // namespace

size_t lanePackBytes(const LanePackPlan& p, int dir, size_t tsize)
{
    const size_t rec = (size_t)p.rows * p.b * (p.dim + (dir < 0 ? 1 : 0)) * 32 * tsize;
    return ((size_t)p.ctas * p.warps * p.steps * rec + 255) & ~(size_t)255;
}
size_t laneHandoffBytes(const LanePackPlan& p, size_t tsize)
{
    return 2 * (size_t)p.ctas * p.warps * p.steps * 32 * p.rows * tsize;
}

template <class T, bool BATCH>
static int lpResident(const LanePackPlan& p, int warps, size_t smem)
{
    int n = 0;
    lpDispatch<T, BATCH>(p.dim, p.b, LpShape{(unsigned)p.grid, p.clusterSize, warps, smem}, LanePackArgs<T>{}, nullptr,
                         nullptr, 0, &n);
    return n;
}

// whole: clusters of exactly maxCluster CTAs, and where possible little enough shared memory for
// two CTAs on an SM (a batched launch: its problems share one cluster size and the SMs)
template <class T>
static LanePackPlan lpPlanFor(int dim, int nx, int ny, int nz, int b, int warps, int maxCluster, bool whole = false)
{
    LanePackPlan p{};
    p.dim = dim;
    p.b = b;
    p.rows = b == 2 ? lpRows<T, 2>() : 1;
    const int lpw = 32 * p.rows / b;
    p.steps = lpSteps(nx, std::min(lpw, ny));
    p.warps = warps;
    const int tile = warps * lpw;
    p.nyb = (ny + tile - 1) / tile;
    const int64_t ctas = (int64_t)p.nyb * (dim == 3 ? nz : 1);
    if (p.nyb > maxCluster || (whole && maxCluster % p.nyb != 0) || ctas > 4096) return p;
    // whole planes, split evenly over as few clusters as hold them
    const int planes = (int)ctas / p.nyb, most = maxCluster / p.nyb;
    const int clusters = (planes + most - 1) / most;
    const int clusterSize = whole ? maxCluster : (planes + clusters - 1) / clusters * p.nyb;
    // the deepest record ring that fits, at least two stages
    auto deepest = [&](size_t limit) {
        p.stages = kLpMaxStages;
        while (p.stages > 1 && lpSmemOf<T>(p) > limit) --p.stages;
        return p.stages >= 2;
    };
    if (!(whole && deepest(112 * 1024)) && !deepest(kLpSmemLimit)) return p;
    p.ctas = (int)ctas;
    p.clusterSize = clusterSize;
    p.grid = (p.ctas + clusterSize - 1) / clusterSize * clusterSize;
    // every cluster of the launch resident at once
    const int resident = whole ? lpResident<T, true>(p, p.warps, lpSmemOf<T>(p))
                               : lpResident<T, false>(p, p.warps, lpSmemOf<T>(p));
    p.ok = resident >= p.grid / clusterSize;
    return p;
}

// Warps per CTA: the fewest CTAs per plane that up to three warps give (a fourth would share its
// sub-partition with the producer warp, which costs more than a hand-off between CTAs: 64x64x16
// in FP64, 0.105 ms per apply with two warps and two CTAs per plane, 0.126 ms with four and
// one), and of those the fewest warps; four where only that keeps every cluster resident.
// Clusters of up to 16 CTAs, smaller where only those are resident: a hand-off across clusters
// costs ~3 us (the consumer keeps a prefetch depth behind), one inside ~0.4 us.
template <class T>
LanePackPlan makeLanePackPlan(int dim, int nx, int ny, int nz, int b)
{
    if ((dim != 2 && dim != 3) || (b != 1 && b != 2) || nx < 1 || ny < 1 || nz < 1) return LanePackPlan{};
    const int lpw = 32 * (b == 2 ? lpRows<T, 2>() : 1) / b;
    auto perPlane = [&](int w) { return (ny + w * lpw - 1) / (w * lpw); };
    int order[4] = {1, 2, 3, 4};
    std::stable_sort(order, order + 3, [&](int p, int q) { return perPlane(p) < perPlane(q); });
    for (int maxCluster : {16, 8, 4})
        for (int w : order) {
            const LanePackPlan p = lpPlanFor<T>(dim, nx, ny, nz, b, w, maxCluster);
            if (p.ok) return p;
        }
    return LanePackPlan{};
}
template <class T>
LanePackPlan makeLanePackBatchPlan(int dim, int nx, int ny, int nz, int b)
{
    if ((dim != 2 && dim != 3) || (b != 1 && b != 2) || nx < 1 || ny < 1 || nz < 1) return LanePackPlan{};
    const int lpw = 32 * (b == 2 ? lpRows<T, 2>() : 1) / b;
    auto perPlane = [&](int w) { return (ny + w * lpw - 1) / (w * lpw); };
    int order[3] = {1, 2, 3};
    std::stable_sort(order, order + 3, [&](int p, int q) { return perPlane(p) < perPlane(q); });
    for (int w : order) {
        const LanePackPlan p = lpPlanFor<T>(dim, nx, ny, nz, b, w, kLanePackBatchCluster, true);
        if (p.ok) return p;
    }
    return LanePackPlan{};
}
template <class T>
int lanePackResident(const LanePackPlan& p, int warps, size_t smem)
{
    return lpResident<T, true>(p, warps, smem);
}
template <class T>
size_t lanePackSmem(const LanePackPlan& p)
{
    return lpSmemOf<T>(p);
}
template <class T>
void launchLanePackApplyBatch(const LanePackArgs<T>* batch, const uint2* map, unsigned blocks, int warps, size_t smem,
                              int dim, int b, cudaStream_t st)
{
    const LpShape shape{blocks, kLanePackBatchCluster, warps, smem};
    DXG_CUDA((lpDispatch<T, true>(dim, b, shape, LanePackArgs<T>{}, batch, map, st, nullptr)));
}

template <class T>
void launchLanePack(const LanePackPlan& p, const LanePackArgs<T>& a, cudaStream_t st)
{
    const int64_t total = (int64_t)p.ctas * p.warps * p.steps * 32;
    const dim3 grid((unsigned)std::min<int64_t>((total + 255) / 256, 4096), 2);
    if (p.dim == 3) {
        if (p.b == 2) lanePackKernel<T, 2, 3><<<grid, 256, 0, st>>>(a);
        else lanePackKernel<T, 1, 3><<<grid, 256, 0, st>>>(a);
    } else {
        if (p.b == 2) lanePackKernel<T, 2, 2><<<grid, 256, 0, st>>>(a);
        else lanePackKernel<T, 1, 2><<<grid, 256, 0, st>>>(a);
    }
    DXG_CUDA(cudaGetLastError());
}
template <class T>
void launchLanePackApply(const LanePackPlan& p, const LanePackArgs<T>& a, cudaStream_t st)
{
    const LpShape shape{(unsigned)p.grid, p.clusterSize, p.warps, lpSmemOf<T>(p)};
    DXG_CUDA((lpDispatch<T, false>(p.dim, p.b, shape, a, nullptr, nullptr, st, nullptr)));
}

template LanePackPlan makeLanePackPlan<double>(int, int, int, int, int);
template LanePackPlan makeLanePackBatchPlan<double>(int, int, int, int, int);
template size_t lanePackSmem<double>(const LanePackPlan&);
template int lanePackResident<double>(const LanePackPlan&, int, size_t);
template void launchLanePackApplyBatch<double>(const LanePackArgs<double>*, const uint2*, unsigned, int, size_t, int, int,
                                           cudaStream_t);
template LanePackPlan makeLanePackPlan<float>(int, int, int, int, int);
template LanePackPlan makeLanePackBatchPlan<float>(int, int, int, int, int);
template size_t lanePackSmem<float>(const LanePackPlan&);
template int lanePackResident<float>(const LanePackPlan&, int, size_t);
template void launchLanePackApplyBatch<float>(const LanePackArgs<float>*, const uint2*, unsigned, int, size_t, int, int,
                                           cudaStream_t);
template void launchLanePack<double>(const LanePackPlan&, const LanePackArgs<double>&, cudaStream_t);
template void launchLanePack<float>(const LanePackPlan&, const LanePackArgs<float>&, cudaStream_t);
template void launchLanePackApply<double>(const LanePackPlan&, const LanePackArgs<double>&, cudaStream_t);
template void launchLanePackApply<float>(const LanePackPlan&, const LanePackArgs<float>&, cudaStream_t);

}  // namespace dxg
