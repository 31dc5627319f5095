// amg.cu -- aggregation AMG kernels (setup and V-cycle) on the structured stencil.
#include "amg.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace dxg {

namespace {

constexpr int kAmgThreads = 256;

// neighbour of (x, y, z) through slot s (3D: -z,-y,-x,diag,+x,+y,+z; 2D: -y,-x,diag,+x,+y):
// false when it leaves the grid; *d = index offset
template <int DIM>
__device__ __forceinline__ bool neighbour(int s, int x, int y, int z, int nx, int ny, int nz, int64_t* d)
{
    const int axis = s < DIM ? DIM - 1 - s : s - DIM - 1;
    const int sign = s < DIM ? -1 : 1;
    const int c = axis == 0 ? x : (axis == 1 ? y : z);
    const int n = axis == 0 ? nx : (axis == 1 ? ny : nz);
    const int64_t stride = axis == 0 ? 1 : (axis == 1 ? (int64_t)nx : (int64_t)nx * ny);
    *d = sign * stride;
    return sign < 0 ? c > 0 : c < n - 1;
}

template <int B, class T>
__device__ __forceinline__ void ldBlk(const T* p, T* o)
{
#pragma unroll
    for (int e = 0; e < B * B; ++e) o[e] = p[e];
}
template <int B, class T>
__device__ __forceinline__ bool invBlk(const T* A, T* inv)
{
    if (B == 1) {
        inv[0] = (T)1 / A[0];
        return A[0] != (T)0;
    } else {
        const T det = A[0] * A[3] - A[1] * A[2];
        if (det == (T)0) return false;
        const T r = (T)1 / det;
        inv[0] = A[3] * r;
        inv[1] = -A[1] * r;
        inv[2] = -A[2] * r;
        inv[3] = A[0] * r;
        return true;
    }
}
// y = M v (B x B block times B-vector)
template <int B, class T>
__device__ __forceinline__ void mv(const T* M, const T* v, T* y)
{
#pragma unroll
    for (int r = 0; r < B; ++r) {
        T t = M[r * B] * v[0];
#pragma unroll
        for (int c = 1; c < B; ++c) t = fma(M[r * B + c], v[c], t);
        y[r] = t;
    }
}

#define AMG_LOOP(L)                                                                                 \
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < (L).N;                   \
         i += (int64_t)gridDim.x * blockDim.x)

__device__ __forceinline__ void coordOf(int64_t i, int nx, int ny, int& x, int& y, int& z)
{
    // cell counts fit 32 bits (checked at upload); a 64-bit division would cost more than the row
    const unsigned q = (unsigned)i / (unsigned)nx;
    x = (int)((unsigned)i - q * (unsigned)nx);
    z = (int)(q / (unsigned)ny);
    y = (int)(q - (unsigned)z * (unsigned)ny);
}

template <int B, class T>
__device__ __forceinline__ void diagInvCell(const AmgLevel<T>& L, int64_t i, int dim, int* singular)
{
    constexpr int BB = B * B;
    T D[BB], inv[BB];
    ldBlk<B>(L.A + ((int64_t)dim * L.N + i) * BB, D);
    if (!invBlk<B>(D, inv)) *singular = 1;
#pragma unroll
    for (int e = 0; e < BB; ++e) L.Dinv[i * BB + e] = inv[e];
}

template <int B, class T>
__global__ void amgDiagInvKernel(AmgLevel<T> L, int dim, int* singular)
{
    AMG_LOOP(L) diagInvCell<B, T>(L, i, dim, singular);
}

// coarse cell C = block sums over its aggregate's fine cells (fixed order: z, y, x, slot)
template <int B, int DIM, class T>
__device__ __forceinline__ void coarsenCell(const AmgLevel<T>& F, const AmgLevel<T>& C, int64_t i, int* singular)
{
    constexpr int BB = B * B, S = 2 * DIM + 1;
    T* Ac = const_cast<T*>(C.A);
    {
        int cx, cy, cz;
        coordOf(i, C.nx, C.ny, cx, cy, cz);
        T acc[S][BB];
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int e = 0; e < BB; ++e) acc[s][e] = 0;
        for (int dz = 0; dz < (DIM == 3 ? 2 : 1); ++dz) {
            const int z = 2 * cz + dz;
            if (z >= F.nz) continue;
            for (int dy = 0; dy < 2; ++dy) {
                const int y = 2 * cy + dy;
                if (y >= F.ny) continue;
                for (int dx = 0; dx < 2; ++dx) {
                    const int x = 2 * cx + dx;
                    if (x >= F.nx) continue;
                    const int64_t f = x + (int64_t)F.nx * (y + (int64_t)F.ny * z);
#pragma unroll
                    for (int s = 0; s < S; ++s) {
                        int target = DIM;
                        if (s != DIM) {
                            int64_t d;
                            if (!neighbour<DIM>(s, x, y, z, F.nx, F.ny, F.nz, &d)) continue;
                            // leaves the aggregate when the neighbour's coarse coordinate differs
                            const int axis = s < DIM ? DIM - 1 - s : s - DIM - 1;
                            const int c = axis == 0 ? x : (axis == 1 ? y : z);
                            const int cn = c + (s < DIM ? -1 : 1);
                            if ((cn >> 1) != (c >> 1)) target = s;
                        }
                        const T* blk = F.A + ((int64_t)s * F.N + f) * BB;
#pragma unroll
                        for (int e = 0; e < BB; ++e) acc[target][e] += blk[e];
                    }
                }
            }
        }
#pragma unroll
        for (int s = 0; s < S; ++s)
#pragma unroll
            for (int e = 0; e < BB; ++e) Ac[((int64_t)s * C.N + i) * BB + e] = acc[s][e];
        T inv[BB];
        if (!invBlk<B>(acc[DIM], inv)) *singular = 1;
#pragma unroll
        for (int e = 0; e < BB; ++e) C.Dinv[i * BB + e] = inv[e];
    }
}

template <int B, int DIM, class T>
__global__ void amgCoarsenKernel(AmgLevel<T> F, AmgLevel<T> C, int* singular)
{
    AMG_LOOP(C) coarsenCell<B, DIM, T>(F, C, i, singular);
}

// sum_s A_is x_j over the existing neighbours and the diagonal
template <int B, int DIM, class T>
__device__ __forceinline__ void rowTimes(const AmgLevel<T>& L, int64_t i, const T* xv, const T* xc, int cnx, int cny,
                                         T* out)
{
    constexpr int BB = B * B, S = 2 * DIM + 1;
    int x, y, z;
    coordOf(i, L.nx, L.ny, x, y, z);
#pragma unroll
    for (int e = 0; e < B; ++e) out[e] = 0;
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int64_t d = 0;
        int jx = x, jy = y, jz = z;
        if (s != DIM) {
            if (!neighbour<DIM>(s, x, y, z, L.nx, L.ny, L.nz, &d)) continue;
            const int axis = s < DIM ? DIM - 1 - s : s - DIM - 1;
            const int sg = s < DIM ? -1 : 1;
            if (axis == 0) jx += sg;
            else if (axis == 1) jy += sg;
            else jz += sg;
        }
        const int64_t j = i + d;
        T v[B];
#pragma unroll
        for (int e = 0; e < B; ++e) v[e] = xv[j * B + e];
        if (xc) {   // prolongation on the fly: x~_j = x_j + xc[aggregate of j]
            const int64_t C = (jx >> 1) + (int64_t)cnx * ((jy >> 1) + (int64_t)cny * (jz >> 1));
#pragma unroll
            for (int e = 0; e < B; ++e) v[e] += xc[C * B + e];
        }
        T blk[BB], t[B];
        ldBlk<B>(L.A + ((int64_t)s * L.N + i) * BB, blk);
        mv<B>(blk, v, t);
#pragma unroll
        for (int e = 0; e < B; ++e) out[e] += t[e];
    }
}

template <class T>
__device__ __forceinline__ bool stopped(const KrylovState* ks)
{
    return ks && ks->status != KS_RUNNING;
}

// ---- per-cell bodies of the V-cycle passes (shared by the per-level kernels and the
// cluster kernel of the small levels)

// out = omega D^-1 b
template <int B, class T>
__device__ __forceinline__ void firstCell(const AmgLevel<T>& L, int64_t i, T* out, T omega)
{
    constexpr int BB = B * B;
    T D[BB], bi[B], y[B];
    ldBlk<B>(L.Dinv + i * BB, D);
#pragma unroll
    for (int e = 0; e < B; ++e) bi[e] = L.b[i * B + e];
    mv<B>(D, bi, y);
#pragma unroll
    for (int e = 0; e < B; ++e) out[i * B + e] = omega * y[e];
}

// out = x~ + omega D^-1 (b - A x~), x~ = xin (+ prolongated xc when given)
template <int B, int DIM, class T>
__device__ __forceinline__ void jacobiCell(const AmgLevel<T>& L, int64_t i, const T* xin, const T* xc, int cnx, int cny,
                                           T* out, T omega)
{
    constexpr int BB = B * B;
    T ax[B], res[B], D[BB], y[B];
    rowTimes<B, DIM, T>(L, i, xin, xc, cnx, cny, ax);
#pragma unroll
    for (int e = 0; e < B; ++e) res[e] = L.b[i * B + e] - ax[e];
    ldBlk<B>(L.Dinv + i * BB, D);
    mv<B>(D, res, y);
    int x, yy, z;
    coordOf(i, L.nx, L.ny, x, yy, z);
    const int64_t C = xc ? (x >> 1) + (int64_t)cnx * ((yy >> 1) + (int64_t)cny * (z >> 1)) : 0;
#pragma unroll
    for (int e = 0; e < B; ++e) {
        T xi = xin[i * B + e];
        if (xc) xi += xc[C * B + e];
        out[i * B + e] = xi + omega * y[e];
    }
}

// r = b - A x
template <int B, int DIM, class T>
__device__ __forceinline__ void residualCell(const AmgLevel<T>& L, int64_t i, const T* xin)
{
    T ax[B];
    rowTimes<B, DIM, T>(L, i, xin, nullptr, 0, 0, ax);
#pragma unroll
    for (int e = 0; e < B; ++e) L.r[i * B + e] = L.b[i * B + e] - ax[e];
}

// coarse b = sum of the aggregate's fine residuals (fixed order)
template <int B, int DIM, class T>
__device__ __forceinline__ void restrictCell(const AmgLevel<T>& F, const AmgLevel<T>& C, int64_t i)
{
    int cx, cy, cz;
    coordOf(i, C.nx, C.ny, cx, cy, cz);
    T acc[B];
#pragma unroll
    for (int e = 0; e < B; ++e) acc[e] = 0;
    for (int dz = 0; dz < (DIM == 3 ? 2 : 1); ++dz) {
        const int z = 2 * cz + dz;
        if (z >= F.nz) continue;
        for (int dy = 0; dy < 2; ++dy) {
            const int y = 2 * cy + dy;
            if (y >= F.ny) continue;
            for (int dx = 0; dx < 2; ++dx) {
                const int x = 2 * cx + dx;
                if (x >= F.nx) continue;
                const int64_t f = x + (int64_t)F.nx * (y + (int64_t)F.ny * z);
#pragma unroll
                for (int e = 0; e < B; ++e) acc[e] += F.r[f * B + e];
            }
        }
    }
#pragma unroll
    for (int e = 0; e < B; ++e) C.b[i * B + e] = acc[e];
}

// row i of x = Ainv b on the last level (the inverse is stored by columns, so that the threads
// of consecutive rows read consecutive entries)
template <class T>
__device__ __forceinline__ void coarseRow(const AmgLevel<T>& L, int n, int i)
{
    T t = 0;
#pragma unroll 8
    for (int j = 0; j < n; ++j) t = fma(L.Ainv[(int64_t)j * n + i], L.b[j], t);
    L.x[i] = t;
}

template <int B, class T>
__global__ void amgFirstKernel(AmgLevel<T> L, T* out, T omega, const KrylovState* ks)
{
    chainWait(kEarlyWide);
    if (stopped<T>(ks)) return;
    AMG_LOOP(L) firstCell<B, T>(L, i, out, omega);
}

template <int B, int DIM, class T>
__global__ void amgJacobiKernel(AmgLevel<T> L, const T* xin, const T* xc, int cnx, int cny, T* out, T omega,
                                const KrylovState* ks)
{
    chainWait(kEarlyWide);
    if (stopped<T>(ks)) return;
    AMG_LOOP(L) jacobiCell<B, DIM, T>(L, i, xin, xc, cnx, cny, out, omega);
}

template <int B, int DIM, class T>
__global__ void amgResidualKernel(AmgLevel<T> L, const T* xin, const KrylovState* ks)
{
    chainWait(kEarlyWide);
    if (stopped<T>(ks)) return;
    AMG_LOOP(L) residualCell<B, DIM, T>(L, i, xin);
}

template <int B, int DIM, class T>
__global__ void amgRestrictKernel(AmgLevel<T> F, AmgLevel<T> C, const KrylovState* ks)
{
    chainWait(kEarlyWide);
    if (stopped<T>(ks)) return;
    AMG_LOOP(C) restrictCell<B, DIM, T>(F, C, i);
}

// The V-cycle below a level of at most kAmgClusterLevel cells as one launch of one thread block
// cluster.  Such a level's passes are a few thousand rows each, so what they cost is the way to
// the data and the barrier between them (run from global memory, 16 CTAs: ~3 us a pass, 41 us for
// the levels 2048, 256 and 32 of a 64x64x32 grid; from shared memory 11 us).  So the
// top level is spread over the CTAs' shared memory -- matrix, pivots, right-hand side and both
// Jacobi buffers, one thread per row, neighbour rows' values by distributed shared memory -- and
// the levels below run in CTA 0 alone, out of its shared memory (their matrices too, where they
// fit) with CTA barriers.  Same per-row arithmetic and pass order as the per-level kernels.
constexpr int kAmgMaxClusterLevels = 12;
constexpr int kAmgClusterCtas = 16;
constexpr int kAmgClusterThreads = 512;
// Largest second level, in cells, for the cycle to start from the level above it.  A BiCGSTAB iteration
// in us, started there and started from the second level itself, 2x2 blocks: FP64 245 cells (grid
// 14x14x10) 131 and 136, 256 (16x16x8) 123 and 129, 256 (64x64x32) 259 and 259, 288 (18x16x8) 134 and
// 130, 512 (16x16x16) 193 and 138; FP32 500 (40x40x20) 129 and 133, 512 98 and 104, 625 (50x50) 93 and
// 120, 1024 (64x64) 104 and 119.  Beyond the lines 1x1 blocks and FP32 could still take it: FP64 1x1 512
// cells 88 and 91, 1024 103 and 109.
constexpr int64_t kAmgOneCtaLevel64 = 256, kAmgOneCtaLevel32 = 640;
constexpr size_t kAmgClusterSmem = 220 * 1024;
// What the cycle holds without the matrices of the lower levels always fits: a sixteenth of the top
// level with its matrix (3D, 2x2 blocks: 40 elements a cell), and the levels below, 12 elements a cell
// of a second level that is limited, each further one about half of the one before at most.
static_assert((kAmgClusterLevel / kAmgClusterCtas * 40 + 3 * kAmgOneCtaLevel64 * 12) * 8 <= (int64_t)kAmgClusterSmem &&
                  (kAmgClusterLevel / kAmgClusterCtas * 40 + 3 * kAmgOneCtaLevel32 * 12) * 4 <= (int64_t)kAmgClusterSmem,
              "");
template <class T>
struct AmgCycle {
    AmgLevel<T> lv[kAmgMaxClusterLevels];
    int count;
    // the level's matrix (last level: the dense inverse) is held in shared memory
    unsigned char matrixShared[kAmgMaxClusterLevels];
};
// Elements of the shared-memory areas: the top level's part of a CTA, then CTA 0's levels with
// or without their matrices.
template <int B, int DIM, class T>
__host__ __device__ inline size_t amgTopElems(int64_t N)
{
    constexpr int BB = B * B, S = 2 * DIM + 1;
    const size_t cpc = (size_t)((N + kAmgClusterCtas - 1) / kAmgClusterCtas);
    return cpc * (S * BB + BB + 4 * B);
}
template <int B, int DIM, class T>
__host__ __device__ inline size_t amgSubElems(int64_t N, bool last, bool matrix)
{
    constexpr int BB = B * B, S = 2 * DIM + 1;
    const size_t n = (size_t)N * B;
    if (last) return (matrix ? n * n : 0) + 2 * n;
    return (size_t)N * ((matrix ? S * BB : 0) + BB + 4 * B);
}

template <int B, int DIM, class T>
__global__ void __launch_bounds__(kAmgClusterThreads) amgClusterCycle(AmgCycle<T> cy, const KrylovState* ks)
{
    constexpr int BB = B * B, S = 2 * DIM + 1;
    extern __shared__ __align__(16) unsigned char amgRaw[];
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), tid = (int)threadIdx.x;
    const T omega = (T)kAmgOmega;
    const int last = cy.count - 1;
    const AmgLevel<T>& top = cy.lv[0];
    const int N = (int)top.N;
    const int cpc = (N + kAmgClusterCtas - 1) / kAmgClusterCtas;

    // shared memory: this CTA's cells of the top level ...
    T* As = reinterpret_cast<T*>(amgRaw);      // [S][cpc][BB]
    T* Ds = As + (size_t)S * cpc * BB;         // [cpc][BB]
    T* bs = Ds + (size_t)cpc * BB;             // [cpc][B]
    T* xs = bs + (size_t)cpc * B;              // [2][cpc][B]
    T* rs = xs + (size_t)2 * cpc * B;          // [cpc][B]
    const int first = rank * cpc, mine = max(0, min(cpc, N - first));
    // One decision for the whole cluster: a CTA must not leave while another reads its shared memory.
    __shared__ int stop;
    chainWait(kEarlyWide);
    if (tid == 0) stop = ks ? __ldcg(&ks->status) != KS_RUNNING : 0;
    cl.sync();
    const int stopAll = *cl.map_shared_rank(&stop, 0);
    if (stopAll) {
        cl.sync();
        return;
    }
    // ... and CTA 0's levels below it
    __shared__ AmgLevel<T> sub[kAmgMaxClusterLevels];
    __shared__ const T* pre[kAmgMaxClusterLevels];
    __shared__ int xcAt;       // where level 1's result lies in CTA 0's area
    auto copy = [&](T* dst, const T* src, size_t k) {
        constexpr size_t per = 16 / sizeof(T);
        size_t e0 = 0;
        if ((((size_t)src | (size_t)dst) & 15) == 0) {
            e0 = k / per * per;
            for (size_t e = tid * per; e < e0; e += blockDim.x * per)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst + e)),
                             "l"(src + e) : "memory");
        }
        for (size_t e = e0 + tid; e < k; e += blockDim.x) dst[e] = src[e];
    };
    if (rank == 0) {
        T* p = reinterpret_cast<T*>(amgRaw) + (last > 0 ? amgTopElems<B, DIM, T>(N) : 0);
        auto take = [&](size_t k) {
            T* q = p;
            p += k;
            return q;
        };
        for (int l = last > 0 ? 1 : 0; l <= last; ++l) {
            AmgLevel<T> L = cy.lv[l];
            const size_t n = (size_t)L.N;
            if (l == last) {
                const unsigned m = (unsigned)(n * B);
                if (cy.matrixShared[l]) {
                    T* inv = take((size_t)m * m);
                    copy(inv, cy.lv[l].Ainv, (size_t)m * m);
                    L.Ainv = inv;
                }
                L.b = take(m);
                if (l > 0) L.x = take(m);
            } else {
                if (cy.matrixShared[l]) {
                    T* m = take(n * S * BB);
                    copy(m, cy.lv[l].A, n * S * BB);
                    L.A = m;
                }
                T* d = take(n * BB);
                copy(d, cy.lv[l].Dinv, n * BB);
                L.Dinv = d;
                L.b = take(n * B);
                L.x = take(n * B);
                L.tmp = take(n * B);
                L.r = take(n * B);
            }
            if (tid == 0) {
                sub[l] = L;
                if (l == 1) xcAt = (int)(L.x - reinterpret_cast<T*>(amgRaw));
            }
        }
    }
    if (last == 0) {
        // one level only: the direct solve
        if (rank == 0) {
            const int n = N * B;
            __syncthreads();
            for (int i = tid; i < n; i += blockDim.x) sub[0].b[i] = top.b[i];
            asm volatile("cp.async.wait_all;" ::: "memory");
            __syncthreads();
            for (int i = tid; i < n; i += blockDim.x) coarseRow<T>(sub[0], n, i);
        }
        cl.sync();
        return;
    }
#pragma unroll
    for (int s = 0; s < S; ++s)
        copy(As + (size_t)s * cpc * BB, top.A + ((int64_t)s * N + first) * BB, (size_t)mine * BB);
    copy(Ds, top.Dinv + (int64_t)first * BB, (size_t)mine * BB);

    // this thread's row of the top level and where its neighbours' values are
    const int lc = tid / B, r = tid % B;
    const bool row = lc < mine;
    int x = 0, y = 0, z = 0;
    if (row) coordOf(first + lc, top.nx, top.ny, x, y, z);
    const T* nb[S];            // the neighbours' entries in Jacobi buffer 0
    int agg[S];                // the neighbours' aggregates
    unsigned has = 0;
    const AmgLevel<T>& C1 = cy.lv[1];
#pragma unroll
    for (int s = 0; s < S; ++s) {
        int64_t d = 0;
        const bool ok = row && (s == DIM || neighbour<DIM>(s, x, y, z, top.nx, top.ny, top.nz, &d));
        const int j = ok ? first + lc + (int)d : first;
        const int axis = s < DIM ? DIM - 1 - s : s - DIM - 1, sg = s < DIM ? -1 : 1;
        const int jx = x + (s != DIM && axis == 0 ? sg : 0), jy = y + (s != DIM && axis == 1 ? sg : 0),
                  jz = z + (s != DIM && axis == 2 ? sg : 0);
        agg[s] = ok ? (jx >> 1) + C1.nx * ((jy >> 1) + C1.ny * (jz >> 1)) : 0;
        const int owner = j / cpc;
        nb[s] = cl.map_shared_rank(xs, owner) + (size_t)(j - owner * cpc) * B;
        has |= ok ? 1u << s : 0u;
    }
    const T* xc = nullptr;     // the coarse correction, in CTA 0
    // row r of A x~, x~ the values of Jacobi buffer w (plus the prolongated correction)
    auto rowTop = [&](int w) -> T {
        T out = 0;
#pragma unroll
        for (int s = 0; s < S; ++s) {
            if (!((has >> s) & 1u)) continue;
            const T* q = nb[s] + (size_t)w * cpc * B;
            T v[B];
#pragma unroll
            for (int e = 0; e < B; ++e) v[e] = q[e];
            if (xc)
#pragma unroll
                for (int e = 0; e < B; ++e) v[e] += xc[agg[s] * B + e];
            const T* m = As + ((size_t)s * cpc + lc) * BB + r * B;
            T t = m[0] * v[0];
#pragma unroll
            for (int e = 1; e < B; ++e) t = fma(m[e], v[e], t);
            out += t;
        }
        return out;
    };
    // row r of D^-1 times the cell's values, this row's in `own`
    auto rowPivot = [&](T own) -> T {
        T v[B];
        v[0] = own;
        if constexpr (B == 2) {
            const T other = __shfl_xor_sync(0xffffffffu, own, 1);
            v[0] = r == 0 ? own : other;
            v[1] = r == 0 ? other : own;
        }
        const T* m = Ds + (size_t)(row ? lc : 0) * BB + r * B;
        T t = m[0] * v[0];
#pragma unroll
        for (int e = 1; e < B; ++e) t = fma(m[e], v[e], t);
        return t;
    };
    auto jacobiTop = [&](int w, T* out) {
        T res = 0;
        if (row) res = bs[lc * B + r] - rowTop(w);
        const T yv = rowPivot(res);
        if (row) {
            T xi = xs[((size_t)w * cpc + lc) * B + r];
            if (xc) xi += xc[agg[DIM] * B + r];
            out[lc * B + r] = xi + omega * yv;
        }
    };
    for (int e = tid; e < mine * B; e += blockDim.x) bs[e] = top.b[(int64_t)first * B + e];
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    // down on the top level: sweeps alternate between the buffers
    {
        const T yv = rowPivot(row ? bs[lc * B + r] : T(0));
        if (row) xs[lc * B + r] = omega * yv;
    }
    cl.sync();
    int w = 0;
    for (int k = 1; k < top.sweeps; ++k, w ^= 1) {
        jacobiTop(w, xs + (size_t)(w ^ 1) * cpc * B);
        cl.sync();
    }
    if (row) rs[lc * B + r] = bs[lc * B + r] - rowTop(w);
    cl.sync();

    if (rank == 0) {
        // restriction from the CTAs' residuals (the aggregate's cells in fixed order) ...
        for (int i = tid; i < (int)C1.N; i += blockDim.x) {
            int cx, cy_, cz;
            coordOf(i, C1.nx, C1.ny, cx, cy_, cz);
            T acc[B];
#pragma unroll
            for (int e = 0; e < B; ++e) acc[e] = 0;
            for (int dz = 0; dz < (DIM == 3 ? 2 : 1); ++dz) {
                if (2 * cz + dz >= top.nz) continue;
                for (int dy = 0; dy < 2; ++dy) {
                    if (2 * cy_ + dy >= top.ny) continue;
                    for (int dx = 0; dx < 2; ++dx) {
                        if (2 * cx + dx >= top.nx) continue;
                        const int f = 2 * cx + dx + top.nx * (2 * cy_ + dy + top.ny * (2 * cz + dz));
                        const int owner = f / cpc;
                        const T* q = cl.map_shared_rank(rs, owner) + (size_t)(f - owner * cpc) * B;
#pragma unroll
                        for (int e = 0; e < B; ++e) acc[e] += q[e];
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < B; ++e) sub[1].b[i * B + e] = acc[e];
        }
        __syncthreads();
        // ... and the cycle below
        for (int l = 1; l < last; ++l) {
            const AmgLevel<T>& L = sub[l];
            T* buf[2] = {L.tmp, L.x};
            int v = 0;
            for (int i = tid; i < (int)L.N; i += blockDim.x) firstCell<B, T>(L, i, buf[0], omega);
            __syncthreads();
            for (int k = 1; k < L.sweeps; ++k, ++v) {
                for (int i = tid; i < (int)L.N; i += blockDim.x)
                    jacobiCell<B, DIM, T>(L, i, buf[v & 1], nullptr, 0, 0, buf[(v + 1) & 1], omega);
                __syncthreads();
            }
            if (tid == 0) pre[l] = buf[v & 1];
            for (int i = tid; i < (int)L.N; i += blockDim.x) residualCell<B, DIM, T>(L, i, buf[v & 1]);
            __syncthreads();
            for (int i = tid; i < (int)sub[l + 1].N; i += blockDim.x) restrictCell<B, DIM, T>(L, sub[l + 1], i);
            __syncthreads();
        }
        {
            const AmgLevel<T>& L = sub[last];
            const int n = (int)L.N * B;
            for (int i = tid; i < n; i += blockDim.x) coarseRow<T>(L, n, i);
            __syncthreads();
        }
        for (int l = last - 1; l >= 1; --l) {
            const AmgLevel<T>& L = sub[l];
            const AmgLevel<T>& C = sub[l + 1];
            T* buf[2] = {L.tmp, L.x};
            int v = L.sweeps - 1;   // index of the last pre-smoothing write
            for (int i = tid; i < (int)L.N; i += blockDim.x)
                jacobiCell<B, DIM, T>(L, i, pre[l], C.x, C.nx, C.ny, buf[(v + 1) & 1], omega);
            ++v;
            __syncthreads();
            for (int k = 1; k < L.sweeps; ++k, ++v) {
                for (int i = tid; i < (int)L.N; i += blockDim.x)
                    jacobiCell<B, DIM, T>(L, i, buf[v & 1], nullptr, 0, 0, buf[(v + 1) & 1], omega);
                __syncthreads();
            }
        }
    }
    cl.sync();
    // up: the correction out of CTA 0 into the first sweep; the last one writes the result
    xc = cl.map_shared_rank(reinterpret_cast<T*>(amgRaw), 0) + *cl.map_shared_rank(&xcAt, 0);
    T* const result = top.x + (int64_t)first * B;
    jacobiTop(w, top.sweeps > 1 ? xs + (size_t)(w ^ 1) * cpc * B : result);
    w ^= 1;
    cl.sync();
    xc = nullptr;
    for (int k = 1; k < top.sweeps; ++k, w ^= 1) {
        const bool end = k + 1 == top.sweeps;
        jacobiTop(w, end ? result : xs + (size_t)(w ^ 1) * cpc * B);
        cl.sync();
    }
}

// Dense inverse of a level of at most kAmgCoarsest cells: the block stencil is expanded
// into an n x n matrix (n = N*b) in shared memory and inverted in place by Gauss-Jordan
// elimination with partial pivoting (row exchanges, undone as column exchanges in reverse
// order at the end); one CTA.
template <int B, int DIM, class T>
__device__ void coarseInvertCta(const AmgLevel<T>& L, int* singular, unsigned char* smemRaw)
{
    constexpr int BB = B * B, S = 2 * DIM + 1;
    const int n = (int)L.N * B;
    T* a = reinterpret_cast<T*>(smemRaw);   // [n][n]
    T* f = a + n * n;                       // column k before the elimination
    int* swapRow = reinterpret_cast<int*>(f + n);
    __shared__ int piv;
    __shared__ bool bad;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) a[e] = 0;
    if (threadIdx.x == 0) bad = false;
    __syncthreads();
    for (int i = threadIdx.x; i < (int)L.N; i += blockDim.x) {
        int x, y, z;
        coordOf(i, L.nx, L.ny, x, y, z);
        for (int s = 0; s < S; ++s) {
            int64_t d = 0;
            if (s != DIM && !neighbour<DIM>(s, x, y, z, L.nx, L.ny, L.nz, &d)) continue;
            const int j = i + (int)d;
            const T* blk = L.A + ((int64_t)s * L.N + i) * BB;
            for (int r = 0; r < B; ++r)
                for (int c = 0; c < B; ++c) a[(i * B + r) * n + j * B + c] = blk[r * B + c];
        }
    }
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        if (threadIdx.x < 32) {
            // pivot: the largest magnitude in column k at or below row k (lowest row on ties)
            T best = -1;
            int row = k;
            for (int i = k + threadIdx.x; i < n; i += 32) {
                const T v = fabs(a[i * n + k]);
                if (v > best) { best = v; row = i; }
            }
            for (int o = 16; o > 0; o >>= 1) {
                const T ob = __shfl_down_sync(0xffffffffu, best, o);
                const int orow = __shfl_down_sync(0xffffffffu, row, o);
                if (ob > best || (ob == best && orow < row)) { best = ob; row = orow; }
            }
            if (threadIdx.x == 0) {
                piv = row;
                swapRow[k] = row;
                if (!(best > 0)) bad = true;
            }
        }
        __syncthreads();
        if (bad) break;
        if (piv != k)
            for (int c = threadIdx.x; c < n; c += blockDim.x) {
                const T t = a[k * n + c];
                a[k * n + c] = a[piv * n + c];
                a[piv * n + c] = t;
            }
        __syncthreads();
        const T dinv = (T)1 / a[k * n + k];
        __syncthreads();
        for (int c = threadIdx.x; c < n; c += blockDim.x) a[k * n + c] = c == k ? dinv : a[k * n + c] * dinv;
        for (int i = threadIdx.x; i < n; i += blockDim.x) f[i] = i == k ? (T)0 : a[i * n + k];
        __syncthreads();
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
            const int i = e / n, c = e % n;
            if (i == k) continue;
            a[e] = c == k ? -f[i] * a[k * n + k] : a[e] - f[i] * a[k * n + c];
        }
        __syncthreads();
    }
    if (bad) {
        if (threadIdx.x == 0) *singular = 1;
        return;
    }
    for (int k = n - 1; k >= 0; --k) {
        const int p = swapRow[k];
        if (p != k)
            for (int i = threadIdx.x; i < n; i += blockDim.x) {
                const T t = a[i * n + k];
                a[i * n + k] = a[i * n + p];
                a[i * n + p] = t;
            }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) L.Ainv[e] = a[e % n * n + e / n];   // by columns
}

template <int B, int DIM, class T>
__global__ void amgCoarseInvertKernel(AmgLevel<T> L, int* singular)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    coarseInvertCta<B, DIM, T>(L, singular, smemRaw);
}

// x = Ainv b on the last level (one row per thread, fixed order)
template <class T>
__global__ void amgCoarseSolveKernel(AmgLevel<T> L, int n, const KrylovState* ks)
{
    chainWait(kEarlyWide);
    if (stopped<T>(ks)) return;
    for (int i = threadIdx.x; i < n; i += blockDim.x) coarseRow<T>(L, n, i);
}

// ---- batched passes: one launch runs one pass for several problems, block k of the
// grid working on problem map[k].x as its block map[k].y of amgPassBlocks(items)
__host__ __device__ __forceinline__ int64_t passItems(int kind, int64_t LN, int64_t CN, int b)
{
    return (kind == AMG_RESTRICT || kind == AMG_COARSEN) ? CN : (kind == AMG_COARSE ? LN * b : LN);
}

template <int B, int DIM, class T, int KIND>
__global__ void __launch_bounds__(kAmgThreads) amgPassBatch(const AmgPass<T>* passes, const uint2* map)
{
    const uint2 m = map[blockIdx.x];
    const AmgPass<T>& P = passes[m.x];
    if (stopped<T>(P.ks)) return;
    const int64_t n = passItems(KIND, P.L.N, P.C.N, B);
    const unsigned nblk = amgPassBlocks(n);
    if (m.y >= nblk) return;
    for (int64_t i = m.y * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)nblk * blockDim.x) {
        if constexpr (KIND == AMG_FIRST) firstCell<B, T>(P.L, i, P.out, P.omega);
        else if constexpr (KIND == AMG_JACOBI)
            jacobiCell<B, DIM, T>(P.L, i, P.in, P.prolong ? P.C.x : nullptr, P.C.nx, P.C.ny, P.out, P.omega);
        else if constexpr (KIND == AMG_RESIDUAL) residualCell<B, DIM, T>(P.L, i, P.in);
        else if constexpr (KIND == AMG_RESTRICT) restrictCell<B, DIM, T>(P.L, P.C, i);
        else if constexpr (KIND == AMG_COARSE) coarseRow<T>(P.L, (int)n, (int)i);
        else if constexpr (KIND == AMG_DIAGINV) diagInvCell<B, T>(P.L, i, DIM, P.singular);
        else coarsenCell<B, DIM, T>(P.L, P.C, i, P.singular);
    }
}

// one CTA per problem: dense inverse of its last level
template <int B, int DIM, class T>
__global__ void amgInvertBatch(const AmgPass<T>* passes)
{
    extern __shared__ __align__(16) unsigned char smemRaw[];
    const AmgPass<T>& P = passes[blockIdx.x];
    coarseInvertCta<B, DIM, T>(P.L, P.singular, smemRaw);
}

unsigned gridFor(int64_t n)
{
    int64_t g = (n + kAmgThreads - 1) / kAmgThreads;
    if (g > 4096) g = 4096;
    return (unsigned)(g < 1 ? 1 : g);
}

template <class T, int B, int DIM>
int64_t vcycle(const std::vector<AmgLevel<T>>& Ls, size_t l, const KrylovState* ks, cudaStream_t st)
{
    const AmgLevel<T>& L = Ls[l];
    const unsigned g = gridFor(L.N);
    // the level after the top one runs in one CTA: where it is large, in FP64 above all, a pass costs
    // that SM more than a launch spread over the GPU, and the cluster starts a level further down
    const bool oneCta = l + 1 >= Ls.size() || Ls[l + 1].N <= (sizeof(T) == 8 ? kAmgOneCtaLevel64 : kAmgOneCtaLevel32);
    if (L.N <= kAmgClusterLevel && Ls.size() - l <= (size_t)kAmgMaxClusterLevels && oneCta) {
        // this level and all below: one cluster launch
        const size_t last = Ls.size() - 1;
        size_t elems = last > l ? amgTopElems<B, DIM, T>(L.N) : 0;
        for (size_t k = last > l ? l + 1 : l; k <= last; ++k) elems += amgSubElems<B, DIM, T>(Ls[k].N, k == last, false);
        AmgCycle<T> cy{};
        cy.count = (int)(Ls.size() - l);
        for (int k = 0; k < cy.count; ++k) cy.lv[k] = Ls[l + k];
        // the matrices of the levels below, the coarsest first, while they fit
        for (int k = cy.count - 1; k >= (cy.count > 1 ? 1 : 0); --k) {
            const size_t more = amgSubElems<B, DIM, T>(cy.lv[k].N, k + 1 == cy.count, true) -
                                amgSubElems<B, DIM, T>(cy.lv[k].N, k + 1 == cy.count, false);
            if ((elems + more) * sizeof(T) > kAmgClusterSmem) break;
            cy.matrixShared[k] = 1;
            elems += more;
        }
        auto kern = amgClusterCycle<B, DIM, T>;
        DXG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        DXG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAmgClusterSmem));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kAmgClusterCtas);
        cfg.blockDim = dim3(kAmgClusterThreads);
        cfg.dynamicSmemBytes = elems * sizeof(T);
        cfg.stream = st;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kAmgClusterCtas;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        DXG_CUDA(cudaLaunchKernelEx(&cfg, kern, cy, ks));
        return 1;
    }
    if (l + 1 == Ls.size()) {
        launchChained(amgCoarseSolveKernel<T>, dim3(1), kAmgThreads, st, L, (int)L.N * B, ks);   // exact solve
        return 1;
    }
    const AmgLevel<T>& C = Ls[l + 1];
    const T omega = (T)kAmgOmega;
    int64_t n = 0;
    // 2*sweeps writes alternate between tmp and x, the last one into x
    T* buf[2] = {L.tmp, L.x};
    int w = 0;
    launchChained(amgFirstKernel<B, T>, dim3(g), kAmgThreads, st, L, buf[w & 1], omega, ks);
    ++n;
    for (int k = 1; k < L.sweeps; ++k, ++w, ++n)
        launchChained(amgJacobiKernel<B, DIM, T>, dim3(g), kAmgThreads, st, L, buf[w & 1], nullptr, 0, 0, buf[(w + 1) & 1], omega,
                                                              ks);
    const T* pre = buf[w & 1];
    launchChained(amgResidualKernel<B, DIM, T>, dim3(g), kAmgThreads, st, L, pre, ks);
    launchChained(amgRestrictKernel<B, DIM, T>, dim3(gridFor(C.N)), kAmgThreads, st, L, C, ks);
    n += 2;
    n += vcycle<T, B, DIM>(Ls, l + 1, ks, st);
    // prolongation fused into the first post-sweep
    launchChained(amgJacobiKernel<B, DIM, T>, dim3(g), kAmgThreads, st, L, pre, C.x, C.nx, C.ny, buf[(w + 1) & 1], omega, ks);
    ++w;
    ++n;
    for (int k = 1; k < L.sweeps; ++k, ++w, ++n)
        launchChained(amgJacobiKernel<B, DIM, T>, dim3(g), kAmgThreads, st, L, buf[w & 1], nullptr, 0, 0, buf[(w + 1) & 1], omega,
                                                              ks);
    return n;
}

}  // namespace

std::vector<std::array<int, 3>> amgLevelDims(int dim, int nx, int ny, int nz)
{
    std::vector<std::array<int, 3>> out;
    int n[3] = {nx, ny, dim == 3 ? nz : 1};
    while (n[0] * (int64_t)n[1] * n[2] > kAmgCoarsest) {
        for (int a = 0; a < 3; ++a) n[a] = (n[a] + 1) / 2;
        out.push_back({n[0], n[1], n[2]});
    }
    return out;
}

template <class T>
void launchAmgDiagInv(const AmgLevel<T>& L, int dim, int b, int* singular, cudaStream_t st)
{
    const unsigned g = gridFor(L.N);
    if (b == 1) amgDiagInvKernel<1, T><<<g, kAmgThreads, 0, st>>>(L, dim, singular);
    else amgDiagInvKernel<2, T><<<g, kAmgThreads, 0, st>>>(L, dim, singular);
    DXG_CUDA(cudaGetLastError());
}

template <class T>
void launchAmgCoarsen(const AmgLevel<T>& fine, AmgLevel<T>& coarse, int dim, int b, int* singular, cudaStream_t st)
{
    const unsigned g = gridFor(coarse.N);
    if (b == 1) {
        if (dim == 2) amgCoarsenKernel<1, 2, T><<<g, kAmgThreads, 0, st>>>(fine, coarse, singular);
        else amgCoarsenKernel<1, 3, T><<<g, kAmgThreads, 0, st>>>(fine, coarse, singular);
    } else {
        if (dim == 2) amgCoarsenKernel<2, 2, T><<<g, kAmgThreads, 0, st>>>(fine, coarse, singular);
        else amgCoarsenKernel<2, 3, T><<<g, kAmgThreads, 0, st>>>(fine, coarse, singular);
    }
    DXG_CUDA(cudaGetLastError());
}

template <class T>
void launchAmgCoarseInvert(const AmgLevel<T>& L, int dim, int b, int* singular, cudaStream_t st)
{
    const int n = (int)L.N * b;
    const size_t smem = (size_t)n * n * sizeof(T) + (size_t)n * sizeof(T) + (size_t)n * sizeof(int);
    auto go = [&](auto kern) {
        DXG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<1, kAmgThreads, smem, st>>>(L, singular);
    };
    if (b == 1) dim == 2 ? go(amgCoarseInvertKernel<1, 2, T>) : go(amgCoarseInvertKernel<1, 3, T>);
    else dim == 2 ? go(amgCoarseInvertKernel<2, 2, T>) : go(amgCoarseInvertKernel<2, 3, T>);
    DXG_CUDA(cudaGetLastError());
}

template <class T>
int64_t launchAmgVcycle(const std::vector<AmgLevel<T>>& levels, int dim, int b, const KrylovState* ks,
                        cudaStream_t st)
{
    int64_t n;
    if (b == 1) n = dim == 2 ? vcycle<T, 1, 2>(levels, 0, ks, st) : vcycle<T, 1, 3>(levels, 0, ks, st);
    else n = dim == 2 ? vcycle<T, 2, 2>(levels, 0, ks, st) : vcycle<T, 2, 3>(levels, 0, ks, st);
    DXG_CUDA(cudaGetLastError());
    return n;
}

template <class T, int B, int DIM>
static void passDispatch(int kind, const AmgPass<T>* p, const uint2* map, unsigned blocks, cudaStream_t st)
{
    switch (kind) {
        case AMG_FIRST: amgPassBatch<B, DIM, T, AMG_FIRST><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
        case AMG_JACOBI: amgPassBatch<B, DIM, T, AMG_JACOBI><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
        case AMG_RESIDUAL: amgPassBatch<B, DIM, T, AMG_RESIDUAL><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
        case AMG_RESTRICT: amgPassBatch<B, DIM, T, AMG_RESTRICT><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
        case AMG_COARSE: amgPassBatch<B, DIM, T, AMG_COARSE><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
        case AMG_DIAGINV: amgPassBatch<B, DIM, T, AMG_DIAGINV><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
        default: amgPassBatch<B, DIM, T, AMG_COARSEN><<<blocks, kAmgThreads, 0, st>>>(p, map); break;
    }
}

template <class T>
void launchAmgPassBatch(int kind, const AmgPass<T>* passes, const uint2* map, unsigned blocks, int dim, int b,
                        cudaStream_t st)
{
    if (b == 1) dim == 2 ? passDispatch<T, 1, 2>(kind, passes, map, blocks, st)
                         : passDispatch<T, 1, 3>(kind, passes, map, blocks, st);
    else dim == 2 ? passDispatch<T, 2, 2>(kind, passes, map, blocks, st)
                  : passDispatch<T, 2, 3>(kind, passes, map, blocks, st);
    DXG_CUDA(cudaGetLastError());
}

template <class T>
void launchAmgInvertBatch(const AmgPass<T>* passes, int count, int maxN, int dim, int b, cudaStream_t st)
{
    const int n = maxN * b;
    const size_t smem = (size_t)n * n * sizeof(T) + (size_t)n * sizeof(T) + (size_t)n * sizeof(int);
    auto go = [&](auto kern) {
        DXG_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<count, kAmgThreads, smem, st>>>(passes);
    };
    if (b == 1) dim == 2 ? go(amgInvertBatch<1, 2, T>) : go(amgInvertBatch<1, 3, T>);
    else dim == 2 ? go(amgInvertBatch<2, 2, T>) : go(amgInvertBatch<2, 3, T>);
    DXG_CUDA(cudaGetLastError());
}

template void launchAmgPassBatch<double>(int, const AmgPass<double>*, const uint2*, unsigned, int, int, cudaStream_t);
template void launchAmgPassBatch<float>(int, const AmgPass<float>*, const uint2*, unsigned, int, int, cudaStream_t);
template void launchAmgInvertBatch<double>(const AmgPass<double>*, int, int, int, int, cudaStream_t);
template void launchAmgInvertBatch<float>(const AmgPass<float>*, int, int, int, int, cudaStream_t);
template void launchAmgDiagInv<double>(const AmgLevel<double>&, int, int, int*, cudaStream_t);
template void launchAmgDiagInv<float>(const AmgLevel<float>&, int, int, int*, cudaStream_t);
template void launchAmgCoarseInvert<double>(const AmgLevel<double>&, int, int, int*, cudaStream_t);
template void launchAmgCoarseInvert<float>(const AmgLevel<float>&, int, int, int*, cudaStream_t);
template void launchAmgCoarsen<double>(const AmgLevel<double>&, AmgLevel<double>&, int, int, int*, cudaStream_t);
template void launchAmgCoarsen<float>(const AmgLevel<float>&, AmgLevel<float>&, int, int, int*, cudaStream_t);
template int64_t launchAmgVcycle<double>(const std::vector<AmgLevel<double>>&, int, int, const KrylovState*,
                                         cudaStream_t);
template int64_t launchAmgVcycle<float>(const std::vector<AmgLevel<float>>&, int, int, const KrylovState*,
                                        cudaStream_t);

}  // namespace dxg
