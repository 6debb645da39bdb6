// Light kernels of the explicit path: ghost fill (FillBoundary + physical
// boundary conditions), pack/unpack of valid cells, the stand-alone max
// wave speed reduction, per-box conserved sums, device time-step
// bookkeeping, and the per-box left/right flux and update kernels of the
// Fluxes.H / Update.H surface.  Level kernels are templated on the storage
// type (double, or float for the FP32-storage variant).
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "euler.cuh"
#include "launch.h"

namespace bamrex {

namespace {

constexpr int kThreads = 256;

int grid_for(long long work, int per_thread = 1)
{
    const long long want = (work + (long long)kThreads * per_thread - 1) / ((long long)kThreads * per_thread);
    const long long cap = (long long)device_sm_count() * 8;
    return (int)std::max(1LL, std::min(want, cap));
}

__device__ __forceinline__ long long fab_index(const FabDev& f, int i, int j, int k)
{
    return (long long)(i - f.b0) + (long long)(j - f.b1) * f.js + (long long)(k - f.b2) * f.ks;
}

template <typename V>
__device__ __forceinline__ int find_by_begin(const V* v, int n, long long idx)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (v[mid].cell_begin <= idx) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------- ghosts
// bamrexBCData::fill_consv_boundary (Source/BoundaryConditions/BCs.cpp:429-442)
// expressed as a table of region copies built on the host.
template <typename T>
__global__ void ghost_fill_kernel(int NC, const GhostOp* __restrict__ ops, int nops, int nchunks,
                                  const FabDev* __restrict__ fabs, const StepScalars* scal)
{
    static_assert(kGhostChunk == 32, "one ghost chunk per warp");
    if (scal && scal->done) return;
    const int* __restrict__ chunk_op = reinterpret_cast<const int*>(ops + nops);
    const int lane = threadIdx.x & 31;
    const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int nw = (int)((gridDim.x * blockDim.x) >> 5);
    for (int q = w; q < nchunks; q += nw) {
        const GhostOp& op = ops[chunk_op[q]];
        // 32-bit index arithmetic: a copy op is a ghost slab, far below 2^31 cells
        const int local = (q - op.chunk_begin) * kGhostChunk + lane;
        const int nx = op.hi[0] - op.lo[0] + 1, ny = op.hi[1] - op.lo[1] + 1;
        if (local < (int)ghost_op_cells(op)) {
            const int row = local / nx;
            const int ci = op.lo[0] + (local - row * nx);
            const int kk = row / ny;
            const int cj = op.lo[1] + (row - kk * ny);
            const int ck = op.lo[2] + kk;
            const int si = op.off[0] + op.mul[0] * ci;
            const int sj = op.off[1] + op.mul[1] * cj;
            const int sk = op.off[2] + op.mul[2] * ck;
            const FabDev& d = fabs[op.dst];
            const FabDev& s = fabs[op.src];
            const T* ps = s.ptr<T>() + fab_index(s, si, sj, sk);
            T* pd = d.ptr<T>() + fab_index(d, ci, cj, ck);
            // every load issued before the first store (the compiler cannot
            // tell that source and destination do not alias)
            T v[kMaxComp];
#pragma unroll
            for (int n = 0; n < kMaxComp; ++n)
                if (n < NC) v[n] = ps[n * s.ns];
#pragma unroll
            for (int n = 0; n < kMaxComp; ++n)
                if (n < NC) pd[n * d.ns] = ((op.negmask >> n) & 1) ? -v[n] : v[n];
        }
    }
}

// ---------------------------------------------------------------- cell walk
// A warp's walk over consecutive cells of the packed order (box after box,
// x fastest inside a box): lane t visits cells first + t, first + t + 32, ...
// and knows each one's box, position in the box and fab offset.  The box is
// searched for once per walk and then only advanced, and the position moves
// by carrying 32 cells into the rows, so a visit costs a few integer
// operations; one 64-bit division by the row length and two by the box per
// element had made the pack kernel instruction bound (4096^2 FP64: 470 us
// for 1.07 GB, 2.3 TB/s, against 164 us at the copy rate).
struct CellWalk {
    const PackBox* boxes;
    const FabDev* fabs;
    int nboxes, b, nx, ny, i, j, k;
    long long begin, end;  // this box's cells in the packed order
    long long off, js, ks, ns;

    __device__ __forceinline__ CellWalk(const PackBox* bx, const FabDev* fb, int nb, long long c)
        : boxes(bx), fabs(fb), nboxes(nb), b(find_by_begin(bx, nb, c))
    {
        enter(c);
    }
    __device__ __forceinline__ void enter(long long c)
    {
        const PackBox& B = boxes[b];
        nx = B.hi[0] - B.lo[0] + 1;
        ny = B.hi[1] - B.lo[1] + 1;
        begin = B.cell_begin;
        end = begin + (long long)nx * ny * (B.hi[2] - B.lo[2] + 1);
        const long long local = c - begin;
        long long row;
        if (local >> 31) {
            row = local / nx;
            i = (int)(local - row * nx);
        } else {
            const unsigned r = (unsigned)local / (unsigned)nx;
            i = (int)((unsigned)local - r * (unsigned)nx);
            row = r;
        }
        k = (int)(row / ny);
        j = (int)(row - (long long)k * ny);
        const FabDev& f = fabs[b];
        js = f.js;
        ks = f.ks;
        ns = f.ns;
        off = fab_index(f, B.lo[0], B.lo[1], B.lo[2]);
    }
    // to cell c, 32 further than the one before
    __device__ __forceinline__ void next(long long c)
    {
        if (c >= end) {
            while (b + 1 < nboxes && c >= boxes[b + 1].cell_begin) ++b;
            enter(c);
            return;
        }
        i += 32;
        while (i >= nx) {
            i -= nx;
            if (++j == ny) {
                j = 0;
                ++k;
            }
        }
    }
    __device__ __forceinline__ long long cell() const { return off + i + j * js + k * ks; }
    template <typename T>
    __device__ __forceinline__ T* ptr() const { return fabs[b].ptr<T>(); }
};

constexpr int kWalkUnroll = 4;  // cells a lane holds at once

// The consecutive cells [first, last) of this warp: the packed order cut
// into equal runs of whole 32 x kWalkUnroll groups.
__device__ __forceinline__ void walk_range(long long total, long long& first, long long& last)
{
    constexpr long long G = 32 * kWalkUnroll;
    const long long w = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long groups = (total + G - 1) / G;
    const long long lo = groups * w / nw, hi = groups * (w + 1) / nw;
    first = lo * G;
    last = hi * G < total ? hi * G : total;
}

// ---------------------------------------------------------------- pack
// packed element e = cell_begin*NC + n*ncells_box + cell (always double).
// HBM bound: every value of kWalkUnroll cells is loaded before the first
// store, 8-byte accesses of 32 consecutive cells.
template <typename T, int NC, bool OUT>
__global__ void __launch_bounds__(kThreads) pack_kernel(const FabDev* __restrict__ fabs, const PackBox* __restrict__ boxes, int nboxes,
                                                        long long total, double* __restrict__ packed)
{
    const int lane = threadIdx.x & 31;
    long long first, last;
    walk_range(total, first, last);
    if (first + lane >= last) return;
    CellWalk w(boxes, fabs, nboxes, first + lane);
    for (long long c0 = first + lane; c0 < last; c0 += 32 * kWalkUnroll) {
        T v[kWalkUnroll][NC];
        double* to_p[kWalkUnroll];
        T* to_f[kWalkUnroll];
        long long step[kWalkUnroll];
#pragma unroll
        for (int u = 0; u < kWalkUnroll; ++u) {
            const long long c = c0 + 32 * u;
            if (c >= last) break;
            if (c != first + lane) w.next(c);
            T* f = w.ptr<T>() + w.cell();
            const long long ncell = w.end - w.begin;
            double* p = packed + w.begin * NC + (c - w.begin);
#pragma unroll
            for (int n = 0; n < NC; ++n) v[u][n] = OUT ? f[n * w.ns] : (T)p[n * ncell];
            to_p[u] = p;
            to_f[u] = f;
            step[u] = OUT ? ncell : w.ns;
        }
#pragma unroll
        for (int u = 0; u < kWalkUnroll; ++u) {
            if (c0 + 32 * u >= last) break;
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                if (OUT) to_p[u][n * step[u]] = (double)v[u][n];
                else to_f[u][n * step[u]] = v[u][n];
            }
        }
    }
}

// One slab of one box (full extent in the other directions) between the fab
// and the packed layout of the whole box ([n][cells of the box], x fastest).
template <typename T>
__global__ void pack_slab_kernel(int NC, const FabDev f, const PackBox box, const PackBox slab, double* __restrict__ packed,
                                 int to_packed)
{
    const int bx = box.hi[0] - box.lo[0] + 1, by = box.hi[1] - box.lo[1] + 1, bz = box.hi[2] - box.lo[2] + 1;
    const long long ncells = (long long)bx * by * bz;
    const int sx = slab.hi[0] - slab.lo[0] + 1, sy = slab.hi[1] - slab.lo[1] + 1, sz = slab.hi[2] - slab.lo[2] + 1;
    const long long scells = (long long)sx * sy * sz;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < scells * NC;
         e += (long long)gridDim.x * blockDim.x) {
        const int n = (int)(e / scells);
        const long long c = e - n * scells;
        const int i = slab.lo[0] + (int)(c % sx);
        const int j = slab.lo[1] + (int)((c / sx) % sy);
        const int k = slab.lo[2] + (int)(c / ((long long)sx * sy));
        const long long q = n * ncells + (i - box.lo[0]) + (long long)bx * ((j - box.lo[1]) + (long long)by * (k - box.lo[2]));
        T* pf = f.ptr<T>() + fab_index(f, i, j, k) + n * f.ns;
        if (to_packed) packed[q] = (double)*pf;
        else *pf = (T)packed[q];
    }
}

// ---------------------------------------------------------------- max speed
// max_wave_speed (Source/System/Euler/Euler.cpp:46-74) over valid cells.
template <typename T, int D, bool FAST>
__global__ void max_ws_kernel(const FabDev* __restrict__ fabs, const PackBox* __restrict__ boxes, int nboxes,
                              long long total, const Consts kc, unsigned long long* ws_bits, const StepScalars* scal)
{
    if (scal && scal->done) return;
    constexpr int NC = D + 2;
    const K<T> k(kc);
    double wmax = 0.0;
    bool nan_seen = false;
    const int lane = threadIdx.x & 31;
    long long first, last;
    walk_range(total, first, last);
    if (first + lane < last) {
        CellWalk w(boxes, fabs, nboxes, first + lane);
        for (long long c0 = first + lane; c0 < last; c0 += 32 * kWalkUnroll) {
            T U[kWalkUnroll][NC];
#pragma unroll
            for (int u = 0; u < kWalkUnroll; ++u) {
                const long long c = c0 + 32 * u;
                if (c >= last) break;
                if (c != first + lane) w.next(c);
                const T* p = w.ptr<T>() + w.cell();
#pragma unroll
                for (int n = 0; n < NC; ++n) U[u][n] = p[n * w.ns];
            }
#pragma unroll
            for (int u = 0; u < kWalkUnroll; ++u) {
                if (c0 + 32 * u >= last) break;
                double s;
                if constexpr (FAST) s = wave_speed_f64<D>(U[u], k);
                else s = (double)wave_speed<T, D>(U[u], k);
                wmax = fmax(wmax, s);
                nan_seen = nan_seen || (s != s);
            }
        }
    }
    __syncwarp();
    for (int off = 16; off > 0; off >>= 1) wmax = fmax(wmax, __shfl_xor_sync(0xffffffffu, wmax, off));
    const bool any_nan = __any_sync(0xffffffffu, nan_seen);
    if (FAST && wmax < 1e-140) wmax = 0.0;  // wave_speed_f64's offset of a state without pressure and motion
    if ((threadIdx.x & 31) == 0) {
        if (any_nan) atomicMax(ws_bits, 0x7ff8000000000000ull);
        else if (wmax > 0.0) atomicMax(ws_bits, (unsigned long long)__double_as_longlong(wmax));
    }
}

// ---------------------------------------------------------------- box sums
// One block per box; each thread sums a fixed strided subset of cells in
// double, then a fixed-shape tree reduction: the result does not depend on
// scheduling, so repeated runs give identical totals.
template <typename T>
__global__ void box_sums_kernel(int NC, const FabDev* __restrict__ fabs, const PackBox* __restrict__ boxes,
                                double* __restrict__ sums)
{
    __shared__ double red[256];
    const int b = blockIdx.x;
    const PackBox& B = boxes[b];
    const FabDev& f = fabs[b];
    const int nx = B.hi[0] - B.lo[0] + 1, ny = B.hi[1] - B.lo[1] + 1, nz = B.hi[2] - B.lo[2] + 1;
    const long long ncell = (long long)nx * ny * nz;
    for (int n = 0; n < NC; ++n) {
        double acc = 0.0;
        for (long long c = threadIdx.x; c < ncell; c += blockDim.x) {
            const int i = B.lo[0] + (int)(c % nx);
            const int j = B.lo[1] + (int)((c / nx) % ny);
            const int k = B.lo[2] + (int)(c / ((long long)nx * ny));
            acc += (double)f.ptr<T>()[fab_index(f, i, j, k) + n * f.ns];
        }
        red[threadIdx.x] = acc;
        __syncthreads();
        for (int w = blockDim.x / 2; w > 0; w >>= 1) {
            if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
            __syncthreads();
        }
        if (threadIdx.x == 0) sums[(long long)b * NC + n] = red[0];
        __syncthreads();
    }
}

// ---------------------------------------------------------------- dt
// estTimeStep (Source/AmrLevelAdv.cpp:395-477 -> FluidSystem.cpp:194-206) by
// next_step_scalars (common.cuh): mode 0 of a run's start, 1 of a step's end.
__global__ void step_dt_kernel(StepScalars* s, int D, double dx0, double dx1, double dx2, double cfl, int mode)
{
    if (s->done) return;
    const double dxs[3] = { dx0, dx1, dx2 };
    next_step_scalars(*s, D, dxs, cfl, mode == 1);
}

// ---------------------------------------------------------------- LR flux
// compute_HLLC_flux_LR / compute_force_flux_LR on a box: one thread per face.
template <int D, int DIR, int KIND>
__global__ void flux_lr_kernel(int lo0, int lo1, int lo2, int hi0, int hi1, int hi2, const FabDev flux,
                               const FabDev cL, const FabDev cR, const Consts kc, double half_dx_dt, double dt_2dx)
{
    constexpr int NC = D + 2;
    const K<double> k(kc);
    const int fhi[3] = { hi0 + (DIR == 0), hi1 + (DIR == 1), hi2 + (DIR == 2) };
    const int nx = fhi[0] - lo0 + 1, ny = fhi[1] - lo1 + 1, nz = fhi[2] - lo2 + 1;
    const long long total = (long long)nx * ny * nz;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = lo0 + (int)(idx % nx);
        const int j = lo1 + (int)((idx / nx) % ny);
        const int kk = lo2 + (int)(idx / ((long long)nx * ny));
        double L[NC], R[NC], F[NC];
        const double* pl = cL.ptr<double>() + fab_index(cL, i - (DIR == 0), j - (DIR == 1), kk - (DIR == 2));
        const double* pr = cR.ptr<double>() + fab_index(cR, i, j, kk);
        for (int n = 0; n < NC; ++n) {
            L[n] = pl[n * cL.ns];
            R[n] = pr[n * cR.ns];
        }
        if (KIND == M_HLLC) hllc_face_f64<D, DIR, true>(L, R, k, F);
        else force_face<double, D, DIR>(L, R, k, half_dx_dt, dt_2dx, F);
        double* pf = flux.ptr<double>() + fab_index(flux, i, j, kk);
        for (int n = 0; n < NC; ++n) pf[n * flux.ns] = F[n];
    }
}

// ---------------------------------------------------------------- updates
// AmrLevelAdv_advance.cpp:330-341 (sweep, dt/dx division form)
template <int D, int DIR>
__global__ void sweep_update_kernel(const UpdateArgs u)
{
    constexpr int NC = D + 2;
    const int nx = u.hi[0] - u.lo[0] + 1, ny = u.hi[1] - u.lo[1] + 1, nz = u.hi[2] - u.lo[2] + 1;
    const long long total = (long long)nx * ny * nz;
    const FabDev& fl = u.flux[0];
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = u.lo[0] + (int)(idx % nx);
        const int j = u.lo[1] + (int)((idx / nx) % ny);
        const int k = u.lo[2] + (int)(idx / ((long long)nx * ny));
        const double* pin = u.in.ptr<double>() + fab_index(u.in, i, j, k);
        const double* pf0 = fl.ptr<double>() + fab_index(fl, i, j, k);
        const double* pf1 = fl.ptr<double>() + fab_index(fl, i + (DIR == 0), j + (DIR == 1), k + (DIR == 2));
        double* po = u.out.ptr<double>() + fab_index(u.out, i, j, k);
        // explicit rounding of the product: no FMA contraction, so the
        // stand-alone update rounds exactly as the scalar reference does
        for (int n = 0; n < NC; ++n)
            po[n * u.out.ns] = pin[n * u.in.ns] - __dmul_rn(u.dtdx[0], pf1[n * fl.ns] - pf0[n * fl.ns]);
    }
}

// conservative_update(bx, ...) (Source/Fluxes/Update.H:99-130, dt*idx form)
template <int D>
__global__ void cons_update_kernel(const UpdateArgs u)
{
    constexpr int NC = D + 2;
    const int nx = u.hi[0] - u.lo[0] + 1, ny = u.hi[1] - u.lo[1] + 1, nz = u.hi[2] - u.lo[2] + 1;
    const long long total = (long long)nx * ny * nz;
    for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (long long)gridDim.x * blockDim.x) {
        const int i = u.lo[0] + (int)(idx % nx);
        const int j = u.lo[1] + (int)((idx / nx) % ny);
        const int k = u.lo[2] + (int)(idx / ((long long)nx * ny));
        const double* pin = u.in.ptr<double>() + fab_index(u.in, i, j, k);
        double* po = u.out.ptr<double>() + fab_index(u.out, i, j, k);
        for (int n = 0; n < NC; ++n) {
            double v = pin[n * u.in.ns];
#pragma unroll
            for (int d = 0; d < D; ++d) {
                const FabDev& f = u.flux[d];
                const double a = f.ptr<double>()[fab_index(f, i + (d == 0), j + (d == 1), k + (d == 2)) + n * f.ns];
                const double b = f.ptr<double>()[fab_index(f, i, j, k) + n * f.ns];
                v = v - __dmul_rn(u.dtdx[d], a - b);
            }
            po[n * u.out.ns] = v;
        }
    }
}

}  // namespace

int device_sm_count()
{
    static int cache[64] = { 0 };
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) return 148;
    if (!cache[dev]) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cache[dev] = n > 0 ? n : 148;
    }
    return cache[dev];
}

cudaError_t launch_ghost_fill(int NC, bool fp32, const GhostOp* ops, int nops, int nchunks, const FabDev* fabs,
                              const StepScalars* scal, cudaStream_t s)
{
    if (nops == 0 || nchunks == 0) return cudaSuccess;
    const long long warps = kThreads / 32;
    const int g = (int)std::min<long long>((nchunks + warps - 1) / warps, (long long)device_sm_count() * 8);
    if (fp32) ghost_fill_kernel<float><<<g, kThreads, 0, s>>>(NC, ops, nops, nchunks, fabs, scal);
    else ghost_fill_kernel<double><<<g, kThreads, 0, s>>>(NC, ops, nops, nchunks, fabs, scal);
    return cudaGetLastError();
}

cudaError_t launch_pack_slab(int NC, bool fp32, const FabDev& fab, const PackBox& box, const PackBox& slab,
                             double* packed, int to_packed, cudaStream_t s)
{
    const long long cells = (long long)(slab.hi[0] - slab.lo[0] + 1) * (slab.hi[1] - slab.lo[1] + 1) * (slab.hi[2] - slab.lo[2] + 1);
    if (cells <= 0) return cudaSuccess;
    const int g = grid_for(cells * NC, 4);
    if (fp32) pack_slab_kernel<float><<<g, kThreads, 0, s>>>(NC, fab, box, slab, packed, to_packed);
    else pack_slab_kernel<double><<<g, kThreads, 0, s>>>(NC, fab, box, slab, packed, to_packed);
    return cudaGetLastError();
}

template <int NC>
static cudaError_t pack_dispatch(bool fp32, const FabDev* fabs, const PackBox* boxes, int nboxes, long long total,
                                 double* packed, int to_packed, cudaStream_t s)
{
    const int g = grid_for(total, kWalkUnroll);
    if (fp32) {
        if (to_packed) pack_kernel<float, NC, true><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total, packed);
        else pack_kernel<float, NC, false><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total, packed);
    } else {
        if (to_packed) pack_kernel<double, NC, true><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total, packed);
        else pack_kernel<double, NC, false><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total, packed);
    }
    return cudaGetLastError();
}

cudaError_t launch_pack(int NC, bool fp32, const FabDev* fabs, const PackBox* boxes, int nboxes,
                        long long total_cells, double* packed, int to_packed, cudaStream_t s)
{
    if (total_cells == 0) return cudaSuccess;
    switch (NC) {
    case 3: return pack_dispatch<3>(fp32, fabs, boxes, nboxes, total_cells, packed, to_packed, s);
    case 4: return pack_dispatch<4>(fp32, fabs, boxes, nboxes, total_cells, packed, to_packed, s);
    case 5: return pack_dispatch<5>(fp32, fabs, boxes, nboxes, total_cells, packed, to_packed, s);
    default: return cudaErrorInvalidValue;
    }
}

template <typename T, bool FAST>
static cudaError_t max_ws_dispatch(int D, const FabDev* fabs, const PackBox* boxes, int nboxes, long long total_cells,
                                   const Consts& k, unsigned long long* ws_bits, const StepScalars* scal,
                                   cudaStream_t s)
{
    const int g = grid_for(total_cells, 4);
    switch (D) {
    case 1: max_ws_kernel<T, 1, FAST><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total_cells, k, ws_bits, scal); break;
    case 2: max_ws_kernel<T, 2, FAST><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total_cells, k, ws_bits, scal); break;
    case 3: max_ws_kernel<T, 3, FAST><<<g, kThreads, 0, s>>>(fabs, boxes, nboxes, total_cells, k, ws_bits, scal); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_max_wave_speed(int D, bool fp32, bool fast, const FabDev* fabs, const PackBox* boxes, int nboxes,
                                  long long total_cells, const Consts& k, unsigned long long* ws_bits,
                                  const StepScalars* scal, cudaStream_t s)
{
    if (fp32) return max_ws_dispatch<float, false>(D, fabs, boxes, nboxes, total_cells, k, ws_bits, scal, s);
    return fast ? max_ws_dispatch<double, true>(D, fabs, boxes, nboxes, total_cells, k, ws_bits, scal, s)
                : max_ws_dispatch<double, false>(D, fabs, boxes, nboxes, total_cells, k, ws_bits, scal, s);
}

cudaError_t launch_box_sums(int NC, bool fp32, const FabDev* fabs, const PackBox* boxes, int nboxes, double* sums,
                            cudaStream_t s)
{
    if (nboxes == 0) return cudaSuccess;
    if (fp32) box_sums_kernel<float><<<nboxes, 256, 0, s>>>(NC, fabs, boxes, sums);
    else box_sums_kernel<double><<<nboxes, 256, 0, s>>>(NC, fabs, boxes, sums);
    return cudaGetLastError();
}

cudaError_t launch_step_dt(StepScalars* scal, int D, double dx0, double dx1, double dx2, double cfl, int mode,
                           cudaStream_t s)
{
    step_dt_kernel<<<1, 1, 0, s>>>(scal, D, dx0, dx1, dx2, cfl, mode);
    return cudaGetLastError();
}

template <int D, int DIR>
static cudaError_t flux_lr_dispatch(int kind, const int* lo, const int* hi, const FabDev& flux, const FabDev& cL,
                                    const FabDev& cR, const Consts& k, double half_dx_dt, double dt_2dx,
                                    cudaStream_t s)
{
    long long faces = 1;
    for (int d = 0; d < 3; ++d) faces *= (long long)(hi[d] - lo[d] + 1 + (d == DIR));
    const int g = grid_for(faces);
    if (kind == M_HLLC)
        flux_lr_kernel<D, DIR, M_HLLC><<<g, 128, 0, s>>>(lo[0], lo[1], lo[2], hi[0], hi[1], hi[2], flux, cL, cR, k,
                                                         half_dx_dt, dt_2dx);
    else
        flux_lr_kernel<D, DIR, M_FORCE><<<g, 128, 0, s>>>(lo[0], lo[1], lo[2], hi[0], hi[1], hi[2], flux, cL, cR, k,
                                                          half_dx_dt, dt_2dx);
    return cudaGetLastError();
}

cudaError_t launch_flux_LR(int D, int dir, int kind, const int* lo, const int* hi, const FabDev& flux,
                           const FabDev& cL, const FabDev& cR, const Consts& k, double dx, double dt,
                           cudaStream_t s)
{
    const double half_dx_dt = 0.5 * dx / dt, dt_2dx = dt / (2 * dx);
#define BAMREX_LR(DD, DR) \
    if (D == DD && dir == DR) return flux_lr_dispatch<DD, DR>(kind, lo, hi, flux, cL, cR, k, half_dx_dt, dt_2dx, s);
    BAMREX_LR(1, 0)
    BAMREX_LR(2, 0)
    BAMREX_LR(2, 1)
    BAMREX_LR(3, 0)
    BAMREX_LR(3, 1)
    BAMREX_LR(3, 2)
#undef BAMREX_LR
    return cudaErrorInvalidValue;
}

cudaError_t launch_sweep_update(int D, int dir, const UpdateArgs& u, cudaStream_t s)
{
    long long cells = 1;
    for (int d = 0; d < 3; ++d) cells *= (long long)(u.hi[d] - u.lo[d] + 1);
    const int g = grid_for(cells);
#define BAMREX_UP(DD, DR) \
    if (D == DD && dir == DR) { sweep_update_kernel<DD, DR><<<g, kThreads, 0, s>>>(u); return cudaGetLastError(); }
    BAMREX_UP(1, 0)
    BAMREX_UP(2, 0)
    BAMREX_UP(2, 1)
    BAMREX_UP(3, 0)
    BAMREX_UP(3, 1)
    BAMREX_UP(3, 2)
#undef BAMREX_UP
    return cudaErrorInvalidValue;
}

cudaError_t launch_conservative_update(int D, const UpdateArgs& u, cudaStream_t s)
{
    long long cells = 1;
    for (int d = 0; d < 3; ++d) cells *= (long long)(u.hi[d] - u.lo[d] + 1);
    const int g = grid_for(cells);
    switch (D) {
    case 1: cons_update_kernel<1><<<g, kThreads, 0, s>>>(u); break;
    case 2: cons_update_kernel<2><<<g, kThreads, 0, s>>>(u); break;
    case 3: cons_update_kernel<3><<<g, kThreads, 0, s>>>(u); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

}  // namespace bamrex
