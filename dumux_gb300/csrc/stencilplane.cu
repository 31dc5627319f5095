// stencilplane.cu -- ILU(0) triangular solves of the 3D 27-point stencil (MPFA-O, 1x1 or 2x2
// blocks) in one launch: the forward and the backward sweep over packed factor records, one
// z-plane per CTA of a cluster.
//
// Natural order: cell (x, y, z) sits on level x + 2y + 4z.  Its 13 lower terms enter the row sum in
// ascending slot order (0..8: the cells of plane z-1 around it; 9, 10, 11: line y-1's x-1, x, x+1;
// 12: x-1), backward the mirrored ones.  What bounds the sweeps: a row is 13 B dependent FP64 FMAs
// (backward B more for the pivot), and on GB300 each takes ~64 cycles, as long as the FP64
// instruction of a warp holds its sub-partition.  One warp per tile of lines doing whole rows
// (stencillane.cu) takes at least 26 of them a level and leaves sub-partitions idle.  But only the
// last terms of a row are of the level before; so here four warps share a tile, each adding the
// terms of some slots (0..2, 3..6, 7..8, 9..12 and the pivot) and handing the partial sum of a row
// on through a ring in shared memory.  Same operands, same order, same bits, and with 7 B of them on
// each of a tile's two sub-partitions a level costs little more than 7 B FMAs: two warps on one
// sub-partition hide each other's polls and loads (with two warps per tile, each alone on its
// sub-partition, a step of 32 lines of 2x2 blocks takes 0.79 us, with four 0.63 us; 14 FMAs: 0.46 us).
// Everything else is as in lanepack.cu and stencilpack.cu: records in the order the sweeps read
// them, streamed by bulk copies (each warp its own, a copy issued as a stage is read out); the
// right-hand side, overwritten by the forward results, in shared memory; histories of the
// neighbours' results polled for an all-ones pattern, loaded a step ahead.
//
// Mapping: 32 / B lines per tile, lane = line and block row; line j of a tile handles cell
// x = t - 1 - 2j at its warps' step t (ascending forward, descending backward).  Plane z-1 (z+1)
// stores its results straight into this CTA's copy of it; of each row of that copy only the newest
// cell is read in a step, the older ones are the lane's values of the steps before, as are the
// line before's (shuffles; across tiles a history indexed by the consumer's step).  Waits are
// bounded as in lanepack.cu.
//
// Measured per apply, 32x32x16 2x2 blocks: whole rows per warp 0.56 ms, this kernel 0.20 ms.
#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"
#include "handoff.cuh"
#include "linalg_kernels.cuh"

namespace cg = cooperative_groups;

namespace dxg {
namespace {

constexpr int kPlMaxTiles = 4;
constexpr int kPlStageSteps = 2;
constexpr int kPlMaxStages = 4;
constexpr int kPlAhead = 8;              // steps a warp of a tile may be ahead of the next
constexpr int kPlRoles = 4;              // warps of a tile: slots 0..2, 3..6, 7..8, 9..12 (backward and the pivot)
constexpr int kPlAll = 14;
constexpr size_t kPlSmemLimit = 226 * 1024;

// steps of a tile, padded to whole stages: a line's first step each way only fetches its
// neighbours' first cells
__host__ __device__ inline int plSteps(int nx, int lines)
{
    return (nx + 2 + 2 * (lines - 1) + kPlStageSteps - 1) / kPlStageSteps * kPlStageSteps;
}
// the first slot of a role; a record has plTerms(role) * b values per lane
__host__ __device__ constexpr int plFirst(int role) { return role == 0 ? 0 : role == 1 ? 3 : role == 2 ? 7 : 9; }
__host__ __device__ constexpr int plTerms(int role, bool fwd)
{
    return role == 0 ? 3 : role == 1 ? 4 : role == 2 ? 2 : fwd ? 4 : 5;
}
__host__ __device__ constexpr int plAll(bool fwd) { return fwd ? kPlAll - 1 : kPlAll; }

struct PlSmem {
    size_t ring, vbuf, zin, ybuf, part, zero, total;
};
__host__ __device__ inline PlSmem plSmem(int nx, int ny, int b, int tiles, int steps, int stages)
{
    PlSmem s{};
    size_t o = 0;
    s.ring = o;
    o += (size_t)tiles * stages * kPlStageSteps * kPlAll * b * 32 * 8;
    s.vbuf = o;
    o += (size_t)tiles * steps * 32 * 8;
    s.part = o;
    o += (size_t)tiles * (kPlRoles - 1) * kPlAhead * 32 * 8;
    s.zin = o;
    o += (size_t)2 * nx * (ny + 2) * b * 8;
    o = (o + 15) / 16 * 16;
    s.ybuf = o;
    o += (size_t)2 * (tiles - 1) * steps * b * 8;
    o = (o + 15) / 16 * 16;
    s.zero = o;
    o += 16;
    s.total = o;
    return s;
}

}  // namespace

// The packed records of both sweeps (blockIdx.y), zeros where a lane has no cell or neighbour.
template <int B>
__global__ void __launch_bounds__(256) stencilPlanePackKernel(StencilArgs a, StencilPlanePlan p)
{
    constexpr int LPW = 32 / B;
    const bool fwd = blockIdx.y == 0;
    double* const out = reinterpret_cast<double*>(a.pack[fwd ? 0 : 1]);
    const int64_t total = (int64_t)a.nz * p.tiles * kPlRoles * p.steps * 32;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < total; k += (int64_t)gridDim.x * blockDim.x) {
        const int lane = (int)(k & 31);
        const int64_t rec = k >> 5;
        const int s = (int)(rec % p.steps);
        const int64_t wz = rec / p.steps, tz = wz / kPlRoles;
        const int role = (int)(wz % kPlRoles), tile = (int)(tz % p.tiles), z = (int)(tz / p.tiles);
        const int y = tile * LPW + lane / B, r = lane % B;
        const int x = (fwd ? s : p.steps - 1 - s) - 1 - 2 * (lane / B);
        const bool cell = y < a.ny && x >= 0 && x < a.nx;
        const int64_t i = cell ? ((int64_t)z * a.ny + y) * a.nx + x : 0;
        const uint32_t m = cell ? a.mask[i] : 0u;
        const int NV = plTerms(role, fwd) * B;
        double* const dst = out + ((tz * plAll(fwd) + plFirst(role)) * B * p.steps + (int64_t)s * NV) * 32;
        for (int e = 0; e < NV; ++e) {
            const int q = plFirst(role) + e / B, c = e % B;
            double val = 0.0;
            if (q < 13) {
                const int slot = fwd ? q : 26 - q;
                if ((m >> slot) & 1u) val = lpEntry(a.LU[((int64_t)slot * a.N + i) * (B * B) + r * B + c]);
            } else if (cell) {
                val = lpEntry(a.Dinv[i * (B * B) + r * B + c]);
            }
            dst[NV * 8 % 16 != 0 && e == NV - 1 ? (NV - 1) * 32 + lane : (e / 2) * 64 + lane * 2 + e % 2] = val;
        }
    }
}

template <int B>
__global__ void __launch_bounds__(kPlRoles * kPlMaxTiles * 32) stencilPlaneApply(StencilArgs a, StencilPlanePlan pl,
                                                                               const double* d, double* v)
{
    using Val = LpVal<double, B>;
    constexpr int LPW = 32 / B, SS = kPlStageSteps, REC1 = B * 32 * 8;   // bytes of one term of a record
    extern __shared__ __align__(128) unsigned char plRaw[];
    __shared__ int stopFlag;
    __shared__ __align__(8) unsigned long long bars[kPlRoles * kPlMaxTiles][kPlMaxStages];

    cg::cluster_group cluster = cg::this_cluster();
    const int nx = a.nx, ny = a.ny, nz = a.nz, W = pl.tiles, steps = pl.steps, stages = pl.stages;
    const PlSmem lay = plSmem(nx, ny, B, W, steps, stages);
    const int z = (int)blockIdx.x, lane = threadIdx.x & 31;   // the grid is one cluster
    // through a shuffle, so that what depends on it is known to be uniform over the warp
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    // warps 4 k, 4 k + 2 (roles 0, 1) and 4 k + 1, 4 k + 3 (roles 2, 3) of a pair of tiles: the roles
    // of a tile that add 7 terms together share a sub-partition
    const int tile = (warp >> 3) * 2 + (warp & 2) / 2, role = (warp & 1) * 2 + (warp >> 2 & 1);
    const int blocks = steps / SS;
    const int zRow = (ny + 2) * B, zDir = nx * zRow, yDir = (W - 1) * steps * B;
    double* const zin = reinterpret_cast<double*>(plRaw + lay.zin);
    double* const ybuf = reinterpret_cast<double*>(plRaw + lay.ybuf);
    double* const part = reinterpret_cast<double*>(plRaw + lay.part);
    const unsigned long long waitNs = a.waitNs ? a.waitNs : 500000000ull;

    // histories: empty where a value will arrive, zero elsewhere.  The plane before: [x][y + 1]; the
    // tile before: entry t forward cell x = t of its last line, backward cell x = t - 2 LPW of the
    // first line of the tile after
    for (int k = threadIdx.x; k < 2 * zDir; k += blockDim.x) {
        const int yy = k % zRow / B;
        const bool plane = k < zDir ? z > 0 : z + 1 < nz;
        zin[k] = plane && yy >= 1 && yy <= ny ? lpEmpty<double>() : 0.0;
    }
    for (int k = threadIdx.x; k < 2 * yDir; k += blockDim.x) {
        const int x = k / B % steps - (k < yDir ? 0 : 2 * LPW);
        ybuf[k] = x >= 0 && x < nx ? lpEmpty<double>() : 0.0;
    }
    for (int k = threadIdx.x; k < W * (kPlRoles - 1) * kPlAhead * 32; k += blockDim.x) part[k] = lpEmpty<double>();
    if (threadIdx.x < 2) reinterpret_cast<double*>(plRaw + lay.zero)[threadIdx.x] = 0.0;
    if (lane < kPlMaxStages) lpBarInit(lpAddr(&bars[warp][lane]));
    if (threadIdx.x == 0) stopFlag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    cluster.sync();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const bool skip = a.ks && a.ks->status != KS_RUNNING;

    if (!skip && tile < W) {
        const int stageBytes = SS * plTerms(role, false) * REC1;
        unsigned char* const ring = plRaw + lay.ring + ((size_t)tile * kPlAll + plFirst(role)) * stages * SS * REC1;
        const uint32_t barAddr = lpAddr(&bars[warp][0]);
        double* const vb = reinterpret_cast<double*>(plRaw + lay.vbuf) + (size_t)tile * steps * 32 + lane;   // + t * 32
        // the partial sums that this warp passes on, + t % ahead * 256; those of the role before lie in front
        const uint32_t partOut = lpAddr(part + (tile * (kPlRoles - 1) + min(role, kPlRoles - 2)) * kPlAhead * 32 + lane);
        const uint32_t partIn = role == 0 ? partOut : lpAddr(part + (tile * (kPlRoles - 1) + role - 1) * kPlAhead * 32 + lane);
        const uint32_t zero = lpAddr(plRaw + lay.zero);
        const int jl = lane / B, r = lane % B, y = tile * LPW + jl;
        const bool lineOk = y < ny;
        const int jx = lineOk ? 1 + 2 * jl : 0x40000000;   // t - jx: the lane's cell, when below nx unsigned
        const int64_t lineBase = lineOk ? ((int64_t)z * ny + y) * nx : 0;
        unsigned long long deadlineOfWait = 0, *const deadline = &deadlineOfWait;
        int block = 0, stage = 0;
        uint32_t parity = 0;
        // the copies of this warp's records: block b of both sweeps into its stage
        const unsigned char* from[2];
        uint32_t size[2];
        for (int k = 0; k < 2; ++k) {
            from[k] = a.pack[k] + (((size_t)z * W + tile) * plAll(k == 0) + plFirst(role)) * steps * REC1;
            size[k] = SS * plTerms(role, k == 0) * REC1;
        }
        auto fetch = [&](int b, int into) {
            if (lane != 0 || b >= 2 * blocks) return;
            const bool fwd = b < blocks;
            lpBulk(lpAddr(ring + into * stageBytes), fwd ? from[0] + (size_t)b * size[0] : from[1] + (size_t)(b - blocks) * size[1],
                   fwd ? size[0] : size[1], barAddr + 8 * into);
        };
        for (int k = 0; k < stages; ++k) fetch(k, k);
        if (role == 0) {
            // the right-hand side, zeros where the lane has no cell
            for (int t = 0; t < steps; ++t) {
                const int x = t - jx;
                const bool valid = (unsigned)x < (unsigned)nx;
                lpCpAsync<8>(lpAddr(vb + t * 32), valid ? d + (lineBase + x) * B + r : d, valid);
            }
            lpCommit();
            lpCpWait<0>();
        }

        // waits until busy() holds for no lane, calling again() in between; false when given up
        auto await = [&](auto&& busy, auto&& again) {
            int n = 0;
            while (__any_sync(0xffffffffu, busy())) {
                if ((++n & 63) == 0) {
                    const bool on = lpGoOn(n, deadline, &stopFlag, a.err, waitNs);
                    if (__any_sync(0xffffffffu, !on)) return false;
                }
                again();
            }
            return true;
        };
        auto term = [](double acc, const double* m, const Val& x) {
            acc = fma(-m[0], x.v[0], acc);
            if constexpr (B == 2) acc = fma(-m[1], x.v[1], acc);
            return acc;
        };
        // the steps of one sweep: step(t, record) with the records of NV values streamed through
        auto run = [&](auto dirC, auto nvC, auto&& step) {
            constexpr int DIR = decltype(dirC)::value, NV = decltype(nvC)::value, REC = NV * 32 * 8;
            int t = DIR > 0 ? 0 : steps - 1;
            if (!lpBarTry(barAddr + 8 * stage, parity)) lpBarWait(barAddr + 8 * stage, parity, &stopFlag, a.err, waitNs);
            double c[NV], n[NV];
            lpLoadRec<double, NV>(ring + stage * stageBytes, lane, c);
            for (int b = 0; b < blocks; ++b) {
                const int after = stage + 1 == stages ? 0 : stage + 1;
                const uint32_t afterParity = after == 0 ? parity ^ 1 : parity;
                const bool ready = b + 1 == blocks || lpBarTry(barAddr + 8 * after, afterParity);
                static_assert(SS == 2, "two steps a stage");
                lpLoadRec<double, NV>(ring + stage * stageBytes + REC, lane, n);
                step(t, c);
                // the block's records are in registers: its stage takes the next one
                __syncwarp();
                fetch(block + stages, stage);
                ++block;
                stage = after;
                parity = afterParity;
                if (!ready) lpBarWait(barAddr + 8 * stage, parity, &stopFlag, a.err, waitNs);
                // (behind the sweep's last block: not read any more)
                lpLoadRec<double, NV>(ring + stage * stageBytes, lane, c);
                step(t + DIR, n);
                t += 2 * DIR;
            }
        };
        auto sweep = [&](auto dirC) {
            constexpr int DIR = decltype(dirC)::value;
            const uint32_t zb = lpAddr(zin + (DIR > 0 ? 0 : zDir)) + (uint32_t)(lineOk ? y + 1 : 0) * (B * 8);
            const uint32_t zx = (uint32_t)zRow * 8;   // to the next x
            // the partial sum of step t, and room for this role's
            LpVal<double, 1> sum{}, room{};
            auto lookSums = [&](int t) {
                const uint32_t at = (uint32_t)(t & (kPlAhead - 1)) * 256u;
                if (role > 0) sum = lpLdShared<double, 1, 0>(partIn + at);
                if (role < kPlRoles - 1) room = lpLdShared<double, 1, 0>(partOut + at);
            };
            auto passOn = [&](int t, double acc) { lpStShared<0>(partOut + (uint32_t)(t & (kPlAhead - 1)) * 256u, acc); };
            auto takeOver = [&](int t) { lpStShared<0>(partIn + (uint32_t)(t & (kPlAhead - 1)) * 256u, lpEmpty<double>()); };
            // what a step waits for (the newest cells of its rows, the partial sum, room for its own) is
            // loaded a step ahead
            auto cellAt = [&](int x, int row) {   // of the plane before, row y + row
                return lpLdShared<double, B, 0>((unsigned)x < (unsigned)nx ? zb + (uint32_t)x * zx + (uint32_t)(row * B * 8) : zero);
            };
            const int tFirst = DIR > 0 ? 0 : steps - 1;
            if (role == 0) {
                Val w0{}, w1{}, z2;   // row y-1: cells x-1, x and x+1
                auto look = [&](int t) {
                    z2 = cellAt(t - jx + DIR, -DIR);
                    lookSums(t);
                };
                look(tFirst);
                run(dirC, std::integral_constant<int, 3 * B>{}, [&](int t, const double* c) {
                    const double rhs = vb[t * 32];
                    if (!await([&] { return z2.empty() || !room.empty(); }, [&] { look(t); })) z2 = Val{};
                    const Val a2 = z2;
                    look(t + DIR);
                    double acc = term(rhs, c, w0);
                    acc = term(acc, c + B, w1);
                    acc = term(acc, c + 2 * B, a2);
                    passOn(t, acc);
                    w0 = w1;
                    w1 = a2;
                });
            } else if (role == 1) {
                Val u0{}, u1{}, z5, z6;   // row y: cells x-1, x and x+1; row y+1: x-1
                auto look = [&](int t) {
                    z5 = cellAt(t - jx + DIR, 0);
                    z6 = cellAt(t - jx - DIR, DIR);
                    lookSums(t);
                };
                look(tFirst);
                run(dirC, std::integral_constant<int, 4 * B>{}, [&](int t, const double* c) {
                    if (!await([&] { return z5.empty() || z6.empty() || sum.empty() || !room.empty(); }, [&] { look(t); })) {
                        z5 = z6 = Val{};
                        sum.v[0] = 0.0;
                    }
                    takeOver(t);
                    const Val a5 = z5, a6 = z6;
                    double acc = term(sum.v[0], c, u0);
                    look(t + DIR);
                    acc = term(acc, c + B, u1);
                    acc = term(acc, c + 2 * B, a5);
                    acc = term(acc, c + 3 * B, a6);
                    passOn(t, acc);
                    u0 = u1;
                    u1 = a5;
                });
            } else if (role == 2) {
                Val w7{}, z8;   // row y+1: cells x and x+1
                auto look = [&](int t) {
                    z8 = cellAt(t - jx + DIR, DIR);
                    lookSums(t);
                };
                look(tFirst);
                run(dirC, std::integral_constant<int, 2 * B>{}, [&](int t, const double* c) {
                    if (!await([&] { return z8.empty() || sum.empty() || !room.empty(); }, [&] { look(t); })) {
                        z8 = Val{};
                        sum.v[0] = 0.0;
                    }
                    takeOver(t);
                    const Val a8 = z8;
                    double acc = term(sum.v[0], c, w7);
                    look(t + DIR);
                    acc = term(acc, c + B, a8);
                    passOn(t, acc);
                    w7 = a8;
                });
            } else {
                const bool edge = jl == (DIR > 0 ? 0 : LPW - 1);
                const bool src = edge && lineOk && (DIR > 0 ? tile > 0 : y + 1 < ny);
                double* const dirBuf = ybuf + (DIR > 0 ? 0 : yDir);
                // boundary k lies between tiles k and k + 1
                const uint32_t yIn = src ? lpAddr(dirBuf + (size_t)(DIR > 0 ? tile - 1 : tile) * steps * B) : zero;
                const bool pub = lineOk && (DIR > 0 ? jl == LPW - 1 && tile + 1 < W : jl == 0 && tile > 0);
                const uint32_t yOut = lpAddr(dirBuf + ((size_t)(DIR > 0 ? tile : tile - 1) * steps + (DIR > 0 ? 0 : 2 * LPW)) * B + r);
                const bool next = DIR > 0 ? z + 1 < nz : z > 0;
                const uint32_t zOut = lpMapa(zb, next ? z + DIR : z) + r * 8;
                const int l0 = (lane - r - DIR * B) & 31;
                double* const dst = v + lineBase * B + r;
                Val n2{}, n3{}, yp;   // line before: cells x, x-1 and, for the tile's first line, x+1
                double prev = 0.0;
                auto look = [&](int t) {
                    yp = lpLdShared<double, B, 0>(src && (unsigned)t < (unsigned)steps ? yIn + (uint32_t)t * (B * 8) : zero);
                    lookSums(t);
                };
                look(tFirst);
                run(dirC, std::integral_constant<int, plTerms(3, DIR > 0) * B>{}, [&](int t, const double* c) {
                    const int x = t - jx;
                    const bool act = (unsigned)x < (unsigned)nx;
                    Val n1, own;
                    n1.v[0] = __shfl_sync(0xffffffffu, prev, l0);
                    if constexpr (B == 2) n1.v[1] = __shfl_sync(0xffffffffu, prev, l0 + 1);
                    double partner = 0.0;
                    if constexpr (B == 2) partner = __shfl_xor_sync(0xffffffffu, prev, 1);
                    if (!await([&] { return sum.empty() || yp.empty(); }, [&] { look(t); })) {
                        sum.v[0] = 0.0;
                        yp = Val{};
                    }
                    takeOver(t);
                    const Val ay = yp;
                    double acc = term(sum.v[0], c, n3);
                    look(t + DIR);
                    acc = term(acc, c + B, n2);
                    if (edge) n1 = ay;
                    acc = term(acc, c + 2 * B, n1);
                    own.v[0] = B == 1 || r == 0 ? prev : partner;
                    if constexpr (B == 2) own.v[1] = r == 0 ? partner : prev;
                    acc = term(acc, c + 3 * B, own);
                    double res = acc;
                    if constexpr (DIR < 0) {
                        if constexpr (B == 2) {
                            const double other = __shfl_xor_sync(0xffffffffu, acc, 1);
                            res = c[4 * B] * (r == 0 ? acc : other);
                            res = fma(c[4 * B + 1], r == 0 ? other : acc, res);
                        } else {
                            res = c[4] * acc;
                        }
                    }
                    if (act) {
                        if (next) lpStRemote<0>(zOut + (uint32_t)x * zx, res);
                        if (pub) lpStShared<0>(yOut + (uint32_t)x * (B * 8), res);
                        if (DIR < 0) dst[x * B] = res;
                    }
                    prev = act ? res : 0.0;
                    if (DIR > 0) vb[t * 32] = prev;
                    n3 = n2;
                    n2 = n1;
                });
            }
        };
        sweep(std::integral_constant<int, 1>{});
        // role 0 reads the forward results of role 3
        asm volatile("bar.sync 1, %0;" ::"r"(kPlRoles * W * 32) : "memory");
        sweep(std::integral_constant<int, -1>{});
    }
    // no CTA may leave while another can still write into its shared memory
    cluster.sync();
}

static void plConfig(const StencilArgs& a, const StencilPlanePlan& p, cudaLaunchConfig_t& cfg, cudaLaunchAttribute* attr)
{
    cfg.gridDim = dim3(a.nz);
    cfg.blockDim = dim3((p.tiles + 1) / 2 * 2 * kPlRoles * 32);
    cfg.dynamicSmemBytes = plSmem(a.nx, a.ny, a.b, p.tiles, p.steps, p.stages).total;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = a.nz;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
}

template <int B>
static bool plResident(const StencilArgs& a, const StencilPlanePlan& p)
{
    auto kern = stencilPlaneApply<B>;
    DXG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    DXG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPlSmemLimit));
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    plConfig(a, p, cfg, attr);
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return fit > 0;
}

StencilPlanePlan makeStencilPlanePlan(const StencilArgs& a)
{
    StencilPlanePlan p{};
    if ((a.b != 1 && a.b != 2) || a.S != 27 || a.nz > 16 || a.nx < 1 || a.ny < 1 || a.nz < 1) return p;
    const int lpw = 32 / a.b;
    if (a.nx > 4096 || a.ny > kPlMaxTiles * lpw) return p;
    p.tiles = (a.ny + lpw - 1) / lpw;
    p.steps = plSteps(a.nx, std::min(lpw, a.ny));
    p.stages = kPlMaxStages;
    while (p.stages > 1 && plSmem(a.nx, a.ny, a.b, p.tiles, p.steps, p.stages).total > kPlSmemLimit) --p.stages;
    if (p.stages >= 2) p.ok = a.b == 2 ? plResident<2>(a, p) : plResident<1>(a, p);
    return p;
}

size_t stencilPlaneBytes(const StencilArgs& a, const StencilPlanePlan& p, int dir)
{
    return (size_t)a.nz * p.tiles * p.steps * plAll(dir > 0) * a.b * 32 * 8;
}

void launchStencilPlanePack(const StencilArgs& a, const StencilPlanePlan& p, cudaStream_t st)
{
    const int64_t total = (int64_t)a.nz * p.tiles * kPlRoles * p.steps * 32;
    const dim3 grid((unsigned)std::min<int64_t>((total + 255) / 256, 4096), 2);
    if (a.b == 2) stencilPlanePackKernel<2><<<grid, 256, 0, st>>>(a, p);
    else stencilPlanePackKernel<1><<<grid, 256, 0, st>>>(a, p);
    DXG_CUDA(cudaGetLastError());
}

void launchStencilPlaneApply(const StencilArgs& a, const StencilPlanePlan& p, const double* d, double* v, cudaStream_t st)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    plConfig(a, p, cfg, attr);
    cfg.stream = st;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    if (a.b == 2) DXG_CUDA(cudaLaunchKernelEx(&cfg, stencilPlaneApply<2>, a, p, d, v));
    else DXG_CUDA(cudaLaunchKernelEx(&cfg, stencilPlaneApply<1>, a, p, d, v));
}

}  // namespace dxg
