// sl_tma.cu -- the BDF2 trace+gather with x along the lanes and the gather's
// source boxes staged in shared memory by the Tensor Memory Accelerator
// (sm_100a).
//
// Why: the gather issues O^3 eight-byte loads per foot per arrival point and is
// bound by the L1 / shared-memory data pipe, so what a warp's load costs decides.
// With 32 z levels along the lanes (the fields' contiguous direction) the feet
// of a warp spread: the mean profile alone shifts neighbouring levels by
// different numbers of cells, the levels' heights differ, and each lane reads
// its own entries of the z tables.  Along x the flow is homogeneous: the lanes'
// feet keep together whatever the step (their spread is the fluctuations',
// not the profile's), the z tables' entries are the same for nearly all lanes
// (one wavefront instead of three), and a box long in x fits at large steps.
// The fields' layout has z fastest, so the kernel reads copies with x fastest:
// k_mid_pack writes U* and halo-padded copies of V^n and V^{n-1} that way in one
// transposing pass (node (i, j, k) at padded (i + q nx, j + r ny, k), x and y
// extended by one box, so a box never wraps).
//
// How: a block is a tile of 32 (x) x 2 (y) x 4 (z) arrival points, one warp
// per row of 32.  The near foot is traced (the iterated midpoint rule of
// sl_device.cuh), located, staged and gathered, then the far foot, through one
// box buffer, so a thread holds one foot's state at a time and a block one box.
// Warp reductions and shared-memory integer min/max of the feet's stencil bases
// give each foot's bounding box.  If it fits Box<O>, one thread issues a 3-D
// cp.async.bulk.tensor load of it (no multicast) onto an mbarrier; a block
// whose feet spread wider gathers through L1 from the same padded copy.
// Weights, the contraction order and the epilogue are those of k_sl, so the
// results are bit-identical to it.
#include <cuda.h>

#include <climits>
#include <mutex>

#include "slc_grid.h"
#include "slc_tma.cuh"

namespace {

constexpr int kThreads = 256;

#include "sl_device.cuh"

constexpr int kTI = 32, kTJ = 2, kTK = 4;    // arrival tile (x, y, z)
static_assert(kTI * kTJ * kTK == kThreads, "one thread per arrival point");

// Staged box (x, y, z) in nodes and resident blocks per SM, per order.  The x
// extent sets the row stride in shared memory: 48 doubles = 384 bytes, a
// multiple of the 128-byte bank cycle, so lanes whose stencil base moved one
// row in y or z keep their banks.
// At 256^3, order 6, per component: 10 x 12 rows at four blocks (64 registers)
// 2.58 ms, at three 2.80, 11 x 13 at three 2.85; z along the lanes 3.05 ms (order
// 4: 0.64 ms at 128^3 against k_sl's 0.58, which the step therefore uses).
template <int O>
struct Box {
    static constexpr int X = 48;
    static constexpr int Y = O == 4 ? 8 : 10;
    static constexpr int Z = O == 4 ? 10 : 12;
    static constexpr int elems = X * Y * Z;
    static constexpr size_t bytes = (size_t)elems * sizeof(double);
    static constexpr int min_blocks = O == 4 ? 5 : 4;
};
// the padded copies' halo: the largest box
constexpr int kBX = Box<6>::X;
constexpr int kBY = Box<6>::Y > Box<4>::Y ? Box<6>::Y : Box<4>::Y;
constexpr int kBZ = Box<6>::Z > Box<4>::Z ? Box<6>::Z : Box<4>::Z;
static_assert((kBX * sizeof(double)) % 128 == 0, "box rows of whole bank cycles");

// Extents of the padded copies (x fastest; an even row, for the tensor map's
// strides) and of U* (no halo).
__host__ __device__ inline int padded_nx(int nx) { return (nx + kBX + 1) & ~1; }
__host__ __device__ inline int padded_ny(int ny) { return ny + kBY; }

// Unwrapped stencil base of one coordinate relative to the tile origin; NaN and
// bases 4096 cells or more away give kFar, which box_fits refuses (the wrapping
// L1 gather serves such feet).
constexpr int kFar = 1 << 20;
__device__ __forceinline__ int rel_base(double f, int h, int origin)
{
    const double r = f - (double)h - (double)origin;
    if (!(r > -4096.0 && r < 4096.0)) return kFar;
    return (int)r;
}

struct Foot {
    double z;      // clamped z
    double tx, ty;
    int rx, ry;    // unwrapped x, y base (minus O/2 - 1) relative to the tile
    int k0;        // z base
};

template <int C, int O>
__device__ __forceinline__ Foot locate_foot(const SlcParams &P, double xd, double yd, double zd,
                                            int i0, int j0, unsigned &ncl)
{
    constexpr int h = O / 2 - 1;
    if (zd < P.z_lo || zd > P.z_hi) ncl += 1;
    Foot F;
    F.z = clampz(P, zd);
    double s = fma(xd, P.inv_dx, Comp<C>::shift_x);
    double f = floor(s);
    F.tx = s - f;
    F.rx = rel_base(f, h, i0);
    s = fma(yd, P.inv_dy, Comp<C>::shift_y);
    f = floor(s);
    F.ty = s - f;
    F.ry = rel_base(f, h, j0);
    const int NZ = Comp<C>::centers ? P.nz + 2 : P.nz + 1;
    const int m0 = locate_m0(Comp<C>::centers, half_cell(P, F.z));
    F.k0 = min(max(m0 - h, 0), NZ - O);
    return F;
}

// Gather from a staged box: weights and contraction order as gather_sum.
template <int C, int O>
__device__ __forceinline__ double gather_box(const SlcParams &P, const double *box, const Foot &F,
                                             int ox, int oy, int oz)
{
    double wx[O], wy[O], wz[O];
    uniform_weights<O, double>(P, F.tx, wx);
    uniform_weights<O, double>(P, F.ty, wy);
    const double *zn = Comp<C>::centers ? P.zc : P.zf;
    const double *dinv = Comp<C>::centers ? P.dinv_c[O] : P.dinv_f[O];
    z_weights<O, double>(zn, dinv, denom_rows(Comp<C>::centers, P.nz, O), F.k0, F.z, wz);
    const double *b = box + (oz * Box<O>::Y + oy) * Box<O>::X + ox;
    double acc[O];
#pragma unroll
    for (int k = 0; k < O; ++k) acc[k] = 0.0;
#pragma unroll
    for (int i = 0; i < O; ++i) {
#pragma unroll
        for (int j = 0; j < O; ++j) {
            const double w = wx[i] * wy[j];
#pragma unroll
            for (int k = 0; k < O; ++k) acc[k] = fma(w, b[(k * Box<O>::Y + j) * Box<O>::X + i], acc[k]);
        }
    }
    double r = 0.0;
#pragma unroll
    for (int k = 0; k < O; ++k) r = fma(wz[k], acc[k], r);
    return r;
}

// Gather through L1 from the padded copy.
template <int C, int O>
__device__ __forceinline__ double gather_global(const SlcParams &P, const NodeViewX &V, double xd, double yd,
                                                const Foot &F)
{
    Stencil<O, double> st;
    build_stencil<C, O, double>(P, 1, V.sy, xd, yd, F.z, half_cell(P, F.z), st);
    return gather_sum<O, double, double>(V.p, st, V.sz);
}

__device__ __forceinline__ void block_minmax3(int *red, bool act, int a, int b, int c)
{
    const int v[3] = {a, b, c};
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const int lo = __reduce_min_sync(0xffffffffu, act ? v[q] : INT_MAX);
        const int hi = __reduce_max_sync(0xffffffffu, act ? v[q] : INT_MIN);
        if ((threadIdx.x & 31) == 0) {
            atomicMin(&red[2 * q], lo);
            atomicMax(&red[2 * q + 1], hi);
        }
    }
}

// Store a tile's values: the output has z fastest, so they change threads
// through shared memory and a group of four threads stores four levels, 32
// bytes.
template <int C>
__device__ __forceinline__ void store_tile(const SlcParams &P, double val, int i0, int j0, double *__restrict__ out)
{
    __shared__ double res[kTK][kTI * kTJ + 1];
    const int tid = threadIdx.x;
    res[tid >> 6][tid & 63] = val;
    __syncthreads();
    const int q = tid >> 2, k = blockIdx.z * kTK + (tid & 3);  // q: the two rows of 32 x
    const int i = i0 + (q & 31), j = j0 + (q >> 5);
    const GhostShape g = ghost_shape(C, P.nx, P.ny, P.nz);
    if (k < ((C == 2) ? P.nz - 1 : P.nz) && j < P.ny && i < P.nx)
        out[(size_t)(i + 1) * g.Y * g.Z + (size_t)(j + 1) * g.Z + (k + 1)] = res[tid & 3][q];
}

// Whether the feet with stencil bases in [r0, r1] x [r2, r3] (relative to the
// tile) x [r4, r5] fit the box; X0, Y0, Z0 its first node in the padded copy (X0
// even: a 16-byte aligned inner coordinate), ox the first base's place in it.
template <int O>
__device__ __forceinline__ bool box_fits(const int *r, int i0, int j0, const SlcParams &P, int &X0, int &Y0,
                                         int &Z0, int &ox)
{
    const bool fit = r[0] <= r[1] && r[1] - r[0] + O + 1 <= Box<O>::X && r[3] - r[2] + O <= Box<O>::Y &&
                     r[5] - r[4] + O <= Box<O>::Z && r[1] < kFar && r[3] < kFar;
    X0 = Y0 = Z0 = ox = 0;
    if (fit) {
        X0 = (i0 + r[0]) % P.nx;
        if (X0 < 0) X0 += P.nx;
        ox = X0 & 1;
        X0 -= ox;
        Y0 = (j0 + r[2]) % P.ny;
        if (Y0 < 0) Y0 += P.ny;
        Z0 = r[4];
    }
    return fit;
}

// VN, VM: the padded copies of V^n and V^{n-1}.  TO, NI: trajectory order and
// iterations, 0 to read them from P.  Tricubic trajectories take two blocks' 128
// registers (step at 96x96x96: 1.42 ms at two blocks, 1.47 at three, 1.50 at four;
// 1.47 with k_sl).
template <int C, int O, int TO, int NI>
__global__ void __launch_bounds__(kThreads, TO == 4 ? 2 : Box<O>::min_blocks)
    k_sl_tma(const __grid_constant__ SlcParams P, const __grid_constant__ Vel3X M, const __grid_constant__ NodeViewX VN,
             const __grid_constant__ NodeViewX VM, double dt, double *__restrict__ out, unsigned long long *nclamp,
             unsigned long long *stats, const __grid_constant__ CUtensorMap tmN,
             const __grid_constant__ CUtensorMap tmM)
{
    extern __shared__ unsigned char smraw[];
    __shared__ __align__(8) unsigned long long mbar[2];
    __shared__ int red[12];  // per foot: min/max of rx, ry, k0
    __shared__ int near_lost;  // the near copy did not complete: the box is not reused
    double *box = (double *)(((uintptr_t)smraw + 127) & ~(uintptr_t)127);
    const int tid = threadIdx.x;
    const int i0 = blockIdx.x * kTI, j0 = blockIdx.y * kTJ;
    const int i = i0 + (tid & 31);
    const int j = j0 + ((tid >> 5) & (kTJ - 1));
    const int k = blockIdx.z * kTK + (tid >> 6);
    const int nzi = (C == 2) ? P.nz - 1 : P.nz;
    const bool act = k < nzi && j < P.ny && i < P.nx;
    const unsigned barN = smem_u32(&mbar[0]), barM = smem_u32(&mbar[1]);
    overlap_begin();
    if (tid == 0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            red[2 * q] = INT_MAX;
            red[2 * q + 1] = INT_MIN;
        }
        near_lost = 0;
        mbar_init(barN, 1);
        mbar_init(barM, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    unsigned ncl = 0;
    double xa = 0.0, ya = 0.0, za = 0.0, us0 = 0.0, vs0 = 0.0, ws0 = 0.0, xd = 0.0, yd = 0.0, zd = 0.0;
    Foot F{};
    if (act) {
        arrival_point<C>(P, i, j, k, xa, ya, za);
        first_sample<C, TO>(P, M, i, j, k, xa, ya, za, us0, vs0, ws0);
        trace_foot<TO, NI>(P, M, xa, ya, za, 0.5 * dt, us0, vs0, ws0, xd, yd, zd);
        F = locate_foot<C, O>(P, xd, yd, zd, i0, j0, ncl);
    }
    block_minmax3(red, act, F.rx, F.ry, F.k0);
    __syncthreads();
    int X0, Y0, Z0, ox;
    const bool fitN = box_fits<O>(red, i0, j0, P, X0, Y0, Z0, ox);
    if (tid == 0) {
        // stats: [0] time-outs, [1] blocks, [2] near boxes staged, [3] far boxes staged
        atomicAdd(stats + 1, 1ull);
        if (fitN) {
            atomicAdd(stats + 2, 1ull);
            mbar_expect_tx(barN, (unsigned)Box<O>::bytes);
            tma_load_3d(smem_u32(box), &tmN, X0, Y0, Z0, barN);
        }
    }
    double ubar = 0.0;
    if (act) {
        const bool staged = fitN && mbar_wait(barN);
        if (fitN && !staged) atomicAdd(stats, 1ull);
        if (staged)
            ubar = gather_box<C, O>(P, box, F, F.rx - red[0] + ox, F.ry - red[2], F.k0 - Z0);
        else
            ubar = gather_global<C, O>(P, VN, xd, yd, F);
    }
    __syncthreads();  // every thread is done with the near box
    if (tid == 0 && fitN && !mbar_wait(barN)) {
        atomicAdd(stats, 1ull);
        near_lost = 1;
    }
    if (act) {
        trace_foot<TO, NI>(P, M, xa, ya, za, dt, us0, vs0, ws0, xd, yd, zd);  // half of 2 dt
        F = locate_foot<C, O>(P, xd, yd, zd, i0, j0, ncl);
    }
    block_minmax3(red + 6, act, F.rx, F.ry, F.k0);
    __syncthreads();
    const bool fitM = !near_lost && box_fits<O>(red + 6, i0, j0, P, X0, Y0, Z0, ox);
    if (tid == 0 && fitM) {
        atomicAdd(stats + 3, 1ull);
        mbar_expect_tx(barM, (unsigned)Box<O>::bytes);
        tma_load_3d(smem_u32(box), &tmM, X0, Y0, Z0, barM);
    }
    double val = 0.0;
    if (act) {
        double ubb;
        const bool staged = fitM && mbar_wait(barM);
        if (fitM && !staged) atomicAdd(stats, 1ull);
        if (staged)
            ubb = gather_box<C, O>(P, box, F, F.rx - red[6] + ox, F.ry - red[8], F.k0 - Z0);
        else
            ubb = gather_global<C, O>(P, VM, xd, yd, F);
        val = bdf2_combine(ubar, ubb, dt, xy_diffusion_bdf2<C>(P, VN, VM, i, j, k));
    }
    store_tile<C>(P, val, i0, j0, out);
    add_clamps(nclamp, ncl);
    if (tid == 0 && fitM && !mbar_wait(barM)) atomicAdd(stats, 1ull);
    overlap_end();
}

// The same through L1 alone, for order-6 flows whose feet spread wider than a
// box (where tma_pays says so): no barriers, and 128 registers for the weights.  Three instances of the
// 12-channel ensemble at 1.8 cells of mean displacement a step: 2.57 ms, against
// 3.5 ms with boxes (a third to three quarters of the far ones do not fit) and
// 3.03 ms with boxes and z along the lanes.  At order 4 k_sl is faster (256^3:
// 1.51 against 1.77 ms per component).
template <int C, int O, int TO, int NI>
__global__ void __launch_bounds__(kThreads, 2)
    k_sl_x(const __grid_constant__ SlcParams P, const __grid_constant__ Vel3X M, const __grid_constant__ NodeViewX VN,
           const __grid_constant__ NodeViewX VM, double dt, double *__restrict__ out, unsigned long long *nclamp)
{
    const int tid = threadIdx.x;
    const int i0 = blockIdx.x * kTI, j0 = blockIdx.y * kTJ;
    const int i = i0 + (tid & 31), j = j0 + ((tid >> 5) & (kTJ - 1)), k = blockIdx.z * kTK + (tid >> 6);
    overlap_begin();
    unsigned ncl = 0;
    double val = 0.0;
    if (k < ((C == 2) ? P.nz - 1 : P.nz) && j < P.ny && i < P.nx) {
        double xa, ya, za, us0, vs0, ws0, xn, yn, zn, xm, ym, zm;
        arrival_point<C>(P, i, j, k, xa, ya, za);
        first_sample<C, TO>(P, M, i, j, k, xa, ya, za, us0, vs0, ws0);
        trace_foot<TO, NI>(P, M, xa, ya, za, 0.5 * dt, us0, vs0, ws0, xn, yn, zn);
        trace_foot<TO, NI>(P, M, xa, ya, za, dt, us0, vs0, ws0, xm, ym, zm);  // half of 2 dt
        ncl = (zn < P.z_lo || zn > P.z_hi) + (zm < P.z_lo || zm > P.z_hi);
        Foot F{};
        F.z = clampz(P, zn);
        const double ubar = gather_global<C, O>(P, VN, xn, yn, F);
        F.z = clampz(P, zm);
        const double ubb = gather_global<C, O>(P, VM, xm, ym, F);
        val = bdf2_combine(ubar, ubb, dt, xy_diffusion_bdf2<C>(P, VN, VM, i, j, k));
    }
    store_tile<C>(P, val, i0, j0, out);
    add_clamps(nclamp, ncl);
    overlap_end();
}

// U* = 2 V^n - V^{n-1} at every node and the halo-padded node copies of V^n and
// V^{n-1}, all with x fastest: 32 (x) x 32 (z) tiles of one padded y row through
// shared memory, loads along z, stores along x.
struct MidPack {
    const double *a[3], *b[3];   // ghost-shaped V^n, V^{n-1}
    double *mid[3], *pad[6];
};

__global__ void __launch_bounds__(256) k_mid_pack(const __grid_constant__ SlcParams P,
                                                  const __grid_constant__ MidPack A, int ztiles)
{
    __shared__ double ta[32][33], tb[32][33];  // [x][z]
    const int PX = padded_nx(P.nx), PY = padded_ny(P.ny);
    const int c = blockIdx.z / ztiles, zt = blockIdx.z - c * ztiles;
    const int NZ = c < 2 ? P.nz + 2 : P.nz + 1;
    const int x0 = blockIdx.x * 32, y = blockIdx.y, z0 = zt * 32;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const NodeView<double> Va = ghost_view<double>(c, A.a[c], P.nx, P.ny, P.nz);
    const NodeView<double> Vb = ghost_view<double>(c, A.b[c], P.nx, P.ny, P.nz);
    const int yj = y % P.ny;
    double va[4], vb[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // all four rows' loads in flight together
        const int x = x0 + w + 8 * q, z = z0 + lane;
        const bool in = x < PX && z < NZ;
        const size_t g = (size_t)(x % P.nx) * Va.sx + (size_t)yj * Va.sy + z;
        va[q] = in ? Va.p[g] : 0.0;
        vb[q] = in ? Vb.p[g] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        ta[w + 8 * q][lane] = va[q];
        tb[w + 8 * q][lane] = vb[q];
    }
    __syncthreads();
    const int x = x0 + lane;
    if (x >= PX) return;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int z = z0 + w + 8 * q;
        if (z >= NZ) continue;
        const double a = ta[lane][w + 8 * q], b = tb[lane][w + 8 * q];
        const size_t o = ((size_t)z * PY + y) * PX + x;
        A.pad[c][o] = a;
        A.pad[c + 3][o] = b;
        if (x < P.nx && y < P.ny) A.mid[c][((size_t)z * P.ny + y) * P.nx + x] = fma(2.0, a, -b);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                  CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                  CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static std::once_flag once;
    static EncodeTiledFn fn = nullptr;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    });
    return fn;
}

template <int O, int TO, int NI>
cudaError_t launch_tma_t(const SlcParams &P, const Vel3X &M, double dt, TriMut out, unsigned long long *ncl,
                         unsigned long long *stats, const TmaSL &T, bool staged, cudaStream_t s)
{
    NodeViewX v[6];
    for (int q = 0; q < 6; ++q) v[q] = NodeViewX{T.pad[q], padded_nx(P.nx), padded_nx(P.nx) * padded_ny(P.ny)};
    const dim3 gc((P.nx + kTI - 1) / kTI, (P.ny + kTJ - 1) / kTJ, (P.nz + kTK - 1) / kTK);
    const dim3 gw(gc.x, gc.y, (P.nz - 1 + kTK - 1) / kTK);
    if constexpr (O == 6) if (!staged) {
        launch_chained(k_sl_x<0, O, TO, NI>, gc, kThreads, 0, s, false, P, M, v[0], v[3], dt, out.u, ncl);
        launch_chained(k_sl_x<1, O, TO, NI>, gc, kThreads, 0, s, true, P, M, v[1], v[4], dt, out.v, ncl);
        if (P.nz > 1) launch_chained(k_sl_x<2, O, TO, NI>, gw, kThreads, 0, s, true, P, M, v[2], v[5], dt, out.w, ncl);
        count_launches(P.nz > 1 ? 3 : 2);
        return cudaGetLastError();
    }
    // the attributes are per device context, so set on every launch (a
    // host-side attribute write)
    const size_t sm = Box<O>::bytes + 128;
    cudaError_t e = cudaFuncSetAttribute(k_sl_tma<0, O, TO, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sl_tma<1, O, TO, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_sl_tma<2, O, TO, NI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    const CUtensorMap *tq = (const CUtensorMap *)T.maps;
    launch_chained(k_sl_tma<0, O, TO, NI>, gc, kThreads, sm, s, false, P, M, v[0], v[3], dt, out.u, ncl, stats, tq[0],
                   tq[3]);
    launch_chained(k_sl_tma<1, O, TO, NI>, gc, kThreads, sm, s, true, P, M, v[1], v[4], dt, out.v, ncl, stats, tq[1],
                   tq[4]);
    if (P.nz > 1)
        launch_chained(k_sl_tma<2, O, TO, NI>, gw, kThreads, sm, s, true, P, M, v[2], v[5], dt, out.w, ncl, stats, tq[2],
                       tq[5]);
    count_launches(P.nz > 1 ? 3 : 2);
    return cudaGetLastError();
}

}  // namespace

// Boxes fit inside the padded arrays in every dimension; shallow and narrow
// grids (nz < 47 and nx < 32) have none, nor do grids whose padded copies exceed
// 32-bit indices or a launch grid's y extent.
bool tma_supported(const SlcParams &P)
{
    if (P.ny > 60000 || (double)(P.nx + kBX + 1) * padded_ny(P.ny) * (P.nz + 2) >= 2147483647.0) return false;
    return P.nz + 1 >= kBZ && (P.nz + 1 >= 48 || P.nx >= 32) && encode_fn() != nullptr;
}

// Whether a triquintic step is faster with x along the lanes than with k_sl
// (z along the lanes): from boxes, or through L1 where the feet spread too far.
// Whole steps, x lanes / k_sl, on a B200:
// - Lanes past the last x are idle and the copies are 48 nodes wider than the
//   grid.  Boxes, ny = nz = 128: 1.50 at nx 16, 1.29 at 24, 1.04 at 32, 1.33 at 33,
//   1.14 at 40, 0.98 at 48, 0.82 at 64, 1.06 at 65, 0.97 at 72; 256x128x128 0.75.
//   So three quarters of the lanes, from nx = 32.  A launch of less than one
//   wave hardly feels idle lanes (24x16x48 1.08, and 0.66 of what it took from
//   boxes with z along the lanes): there from nx = 24.
// - Through L1, k_sl's lanes spread with the profile over 32 levels, a whole
//   channel at nz = 32: 0.88 on 64x64x32, 0.85 on 128x96x64, 0.96 on 96x96x96, but
//   1.04 on 52x64x32, 1.09 on 64x128x128, 1.31 on 97x128x128, 1.02 on 120x120x120,
//   0.97 on 128x128x128.
// - Tricubic trajectories read 64 nodes per sample through L1, so the same line:
//   0.91 on 64x64x32, 0.79 on 160x64x48, 0.97 on 96x96x96, 0.96 on 256x192x192, but
//   1.05 on 80x64x32, 1.17 on 48x64x32; two iterations (unrolled, else 1.09 on 128x128x128).
bool tma_pays(const SlcParams &P, bool staged)
{
    const int tiles = (P.nx + kTI - 1) / kTI;
    const double lanes = (double)P.nx / (kTI * tiles);
    const bool cubic = P.traj_order != 2;
    if (cubic && P.n_iters != 2) return false;
    if (!staged || cubic) return P.nx >= kTI && (P.nz <= 96 ? lanes >= 0.875 : P.nx >= 96 && lanes >= 0.96);
    const long long blocks = 3LL * tiles * ((P.ny + kTJ - 1) / kTJ) * ((P.nz + kTK - 1) / kTK);
    return lanes >= 0.75 && (P.nx >= kTI || blocks <= 148 * Box<6>::min_blocks);
}

size_t tma_padded_elems(const SlcParams &P, int comp)
{
    const int NZ = comp < 2 ? P.nz + 2 : P.nz + 1;
    return (size_t)padded_nx(P.nx) * padded_ny(P.ny) * NZ;
}

// Tensor maps of the six padded node copies (slot comp + 3 * which).
cudaError_t tma_encode(const SlcParams &P, TmaSL &T)
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    static_assert(sizeof(CUtensorMap) * 6 <= sizeof(T.maps), "tensor-map storage");
    CUtensorMap *tm = (CUtensorMap *)T.maps;
    for (int q = 0; q < 6; ++q) {
        const int comp = q % 3;
        const int NZ = comp < 2 ? P.nz + 2 : P.nz + 1;
        const cuuint64_t px = (cuuint64_t)padded_nx(P.nx), py = (cuuint64_t)padded_ny(P.ny);
        const cuuint64_t dims[3] = {px, py, (cuuint64_t)NZ};
        const cuuint64_t strides[2] = {px * 8, px * py * 8};
        const bool o4 = P.order == 4;
        const cuuint32_t box[3] = {(cuuint32_t)Box<6>::X, (cuuint32_t)(o4 ? Box<4>::Y : Box<6>::Y),
                                   (cuuint32_t)(o4 ? Box<4>::Z : Box<6>::Z)};
        const cuuint32_t estr[3] = {1, 1, 1};
        CUresult r = enc(&tm[q], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 3, (void *)T.pad[q], dims, strides, box,
                         estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
    }
    return cudaSuccess;
}

cudaError_t launch_mid_pack(const SlcParams &P, Tri cur, Tri prev, TriMut mid, const TmaSL &T,
                            cudaStream_t s)
{
    const MidPack a{{cur.u, cur.v, cur.w}, {prev.u, prev.v, prev.w}, {mid.u, mid.v, mid.w},
                    {T.pad[0], T.pad[1], T.pad[2], T.pad[3], T.pad[4], T.pad[5]}};
    const int ztiles = (P.nz + 2 + 31) / 32;
    const dim3 grid((padded_nx(P.nx) + 31) / 32, padded_ny(P.ny), 3 * ztiles);
    k_mid_pack<<<grid, 256, 0, s>>>(P, a, ztiles);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_sl_tma(const SlcParams &P, Tri mid, double dt, TriMut out, unsigned long long *nclamp,
                          unsigned long long *stats, const TmaSL &T, bool staged, cudaStream_t s)
{
    Vel3X M;
    M.u = NodeViewX{mid.u, P.nx, P.nx * P.ny};
    M.v = NodeViewX{mid.v, P.nx, P.nx * P.ny};
    M.w = NodeViewX{mid.w, P.nx, P.nx * P.ny};
    const bool usual = P.traj_order == 2 && P.n_iters == 2;
    if (P.order == 4)
        return usual ? launch_tma_t<4, 2, 2>(P, M, dt, out, nclamp, stats, T, staged, s)
                     : launch_tma_t<4, 0, 0>(P, M, dt, out, nclamp, stats, T, staged, s);
    if (usual) return launch_tma_t<6, 2, 2>(P, M, dt, out, nclamp, stats, T, staged, s);
    if (P.n_iters == 2) return launch_tma_t<6, 4, 2>(P, M, dt, out, nclamp, stats, T, staged, s);
    return launch_tma_t<6, 0, 0>(P, M, dt, out, nclamp, stats, T, staged, s);
}

// One 3-D tiled tensor map (z innermost, no swizzle, zero fill) over a node
// array: FP32 or FP64 elements, dims (z, y, x), the y and x strides in
// bytes, and the box (z, y, x) in elements.
cudaError_t tma_encode_3d(void *map128, bool fp32, const void *base, const unsigned long long dims[3],
                          const unsigned long long strides[2], const unsigned box[3])
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return cudaErrorNotSupported;
    const cuuint64_t d[3] = {dims[0], dims[1], dims[2]};
    const cuuint64_t st[2] = {strides[0], strides[1]};
    const cuuint32_t bx[3] = {box[0], box[1], box[2]};
    const cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = enc((CUtensorMap *)map128, fp32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT64,
                     3, const_cast<void *>(base), d, st, bx, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}
