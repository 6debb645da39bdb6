// The x sweep by row groups: the fused flux + conservative update of the
// contiguous direction (compute_*_flux + the update lambda of
// AmrLevelAdv::advance_explicit, Source/AmrLevelAdv_advance.cpp:290-341), for
// every method, dimension and storage type, over every box of a level or one
// box given by value.
//
// Work decomposition.  A row's positions lo-2 .. hi+2 are cut into groups of
// kP (row_group: 4 or 2) and the groups of a box's rows are numbered
// one row after the other.  A chunk is 32 consecutive groups, one per lane;
// lanes 1 .. 30 store their cells, lanes 0 and 31 are the halo of the chunk
// (the neighbouring chunks own them).  A row carries its own halo positions,
// so nothing crosses from one row into the next, and rows of any width fill
// the warp: a 64-cell row is 17 groups, an 8-cell one is 3.  Each warp takes
// an equal run of consecutive chunks of the level.
//
// Inside a chunk a lane computes its group's kP cell stages, kP faces and kP
// updates in registers; the neighbours' edge cells, edge states and edge face
// come by warp shuffle.  The kP cells are independent instruction streams
// without a branch between them, which is what fills the FP64 pipe (two
// cycles per warp instruction, eight to the result).
//
// Input: the lane's own positions, two at a time (cp.async of 16 bytes, or 8
// in FP32), into a buffer of its own in shared memory, one chunk ahead.
// Updates leave as pairs too.
//
// Measured on the B200 (x sweep, before -> now; before: the wavefront, a row
// kernel with a carried pipeline or the marching kernel, whichever was
// fastest): 4096^2 FP64 377 -> 359 us, in 64^2 boxes 482 -> 388, 256^3 in
// 64^3 boxes 651 -> 466, in 32^3 674 -> 491; FP32 storage 4096^2 206 -> 174,
// in 64^2 boxes 403 -> 213, 256^3 in 64^3 boxes 574 -> 241.  Bound by the
// FP64 pipe (185 instructions per cell, 388 in all, half of the issue slots)
// and the waits of two warps per scheduler.
//
// LEVEL: a level's own fabs (in and out laid out
// alike, rows aligned to pairs, x halos possibly in a neighbouring box's
// fab).  Otherwise one caller's box, with the optional flux output; VEC =
// false there (rows not aligned to pairs) copies and stores single elements.
#pragma once

#include "common.cuh"
#include "euler.cuh"
#include "sweep.cuh"
#include "tma.cuh"

namespace bamrex {

#ifndef BAMREX_ROW_MIN_BLOCKS
#define BAMREX_ROW_MIN_BLOCKS 2
#endif
#ifndef BAMREX_ROW_MIN_BLOCKS_F32
#define BAMREX_ROW_MIN_BLOCKS_F32 3
#endif
template <typename T>
constexpr int row_min_blocks() { return sizeof(T) == 4 ? BAMREX_ROW_MIN_BLOCKS_F32 : BAMREX_ROW_MIN_BLOCKS; }

template <typename T>
struct alignas(2 * sizeof(T)) Pair {
    T a, b;
};

__device__ __forceinline__ void cp_async_pair(Pair<double>* dst, const double* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_pair(Pair<float>* dst, const float* src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_one() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

__device__ __forceinline__ void st_pair_if(double* p, double a, double b, bool pred)
{
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %3, 0;\n @q st.global.v2.f64 [%0], {%1, %2};\n}\n" ::"l"(p), "d"(a),
                 "d"(b), "r"((int)pred)
                 : "memory");
}
__device__ __forceinline__ void st_pair_if(float* p, float a, float b, bool pred)
{
    asm volatile("{\n .reg .pred q;\n setp.ne.b32 q, %3, 0;\n @q st.global.v2.f32 [%0], {%1, %2};\n}\n" ::"l"(p), "f"(a),
                 "f"(b), "r"((int)pred)
                 : "memory");
}

template <typename T, int N>
__device__ __forceinline__ void shfl_up1(const T (&s)[N], T (&d)[N])
{
#pragma unroll
    for (int n = 0; n < N; ++n) d[n] = __shfl_up_sync(0xffffffffu, s[n], 1);
}
template <typename T, int N>
__device__ __forceinline__ void shfl_down1(const T (&s)[N], T (&d)[N])
{
#pragma unroll
    for (int n = 0; n < N; ++n) d[n] = __shfl_down_sync(0xffffffffu, s[n], 1);
}

// A neighbouring fab that holds one side's x halo, in shared memory (read by
// the few lanes at a row's end).
struct RowHalo {
    const void* p;  // cell (0, lo[1], lo[2]) of the box, in the neighbour's fab; null: none
    long long js, ks, ns;
};

template <typename T, int D, int METHOD, int LIM, bool LEVEL, bool VEC>
__global__ void __launch_bounds__(kSweepThreads, row_min_blocks<T>()) sweep_row_kernel(const SweepArgs a)
{
    using S = Scheme<T, D, 0, METHOD, LIM>;
    constexpr int NC = D + 2;
    constexpr int H = S::kHalo;
    constexpr int kP = row_group(METHOD, LIM);
    constexpr int kPairs = kP / 2;
    static_assert(VEC || !LEVEL, "a level's rows are aligned to pairs");
    __shared__ Pair<T> stage[kSweepThreads / 32][2][NC][kPairs][32];
    __shared__ RowHalo halos[kSweepThreads / 32][2];
    StepFactors<T> f;
    if (!step_factors(a, f)) return;
    const K<T> k(a.k);
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
    auto& st = stage[threadIdx.x >> 5];
    auto& halo = halos[threadIdx.x >> 5];
    const bool owner = lane >= 1 && lane <= kRowOwned;
    const bool do_update = LEVEL || a.do_update != 0, ws_on = a.ws_max != nullptr;
    WsMax<T> wsmax;

    // this warp's chunks, split over the boxes they fall in
    long long c = a.total_items * gw / nw;
    const long long c_end = a.total_items * (gw + 1) / nw;
    int b = (a.boxes && c < c_end) ? find_box(a.boxes, a.nboxes, c) : 0;
    for (; c < c_end; ++b) {
        const SweepBox& B = a.boxes ? a.boxes[b] : a.one;
        const long long box_end = (a.boxes && b + 1 < a.nboxes) ? a.boxes[b + 1].item_begin : a.total_items;
        const int lo = B.lo[0], hi = B.hi[0];
        const int ny = B.hi[1] - B.lo[1] + 1, nrow = ny * (B.hi[2] - B.lo[2] + 1);
        const int G = B.ngroup;
        const int ngroups = G * nrow;
        const long long ijs = B.in.js, iks = B.in.ks, ins = B.in.ns;
        const long long ojs = LEVEL ? ijs : B.out.js, oks = LEVEL ? iks : B.out.ks, ons = LEVEL ? ins : B.out.ns;
        // cell (x, lo[1] + j, lo[2] + kz) at in + j js + kz ks + x
        const T* __restrict__ in = B.in.ptr<T>() + (long long)(B.lo[1] - B.in.b1) * ijs + (long long)(B.lo[2] - B.in.b2) * iks - B.in.b0;
        T* __restrict__ out = B.out.ptr<T>() + (long long)(B.lo[1] - B.out.b1) * ojs + (long long)(B.lo[2] - B.out.b2) * oks - B.out.b0;
        // x halos read from the neighbouring boxes' fabs (else from this
        // box's ghost cells)
        bool xlo = false, xhi = false;
        if constexpr (LEVEL) {
            xlo = a.xnb_on && B.xnb[0].p;
            xhi = a.xnb_on && B.xnb[1].p;
            __syncwarp();
            if (lane < 2) {
                const FabDev& N = B.xnb[lane];
                halo[lane] = { N.ptr<T>() + (long long)(B.lo[1] - N.b1) * N.js + (long long)(B.lo[2] - N.b2) * N.ks - N.b0,
                               N.js, N.ks, N.ns };
            }
            __syncwarp();
        }
        T* __restrict__ fl = nullptr;
        long long fns = 0;
        if constexpr (!LEVEL) {
            if (B.flux.p)
                fl = B.flux.ptr<T>() + (long long)(B.lo[1] - B.flux.b1) * B.flux.js + (long long)(B.lo[2] - B.flux.b2) * B.flux.ks - B.flux.b0;
            fns = B.flux.ns;
        }

        // the lane's group: gi-th of row (j, kz)
        int g = kRowOwned * (int)(c - B.item_begin) - 1 + lane;
        int gi, j, kz;
        bool active;
        auto place = [&]() {
            active = g >= 0 && g < ngroups;
            const int row = active ? g / G : 0;
            gi = active ? g - row * G : 0;
            kz = D == 3 ? row / ny : 0;
            j = D == 1 ? 0 : (D == 3 ? row - kz * ny : row);
        };
        place();
        // start the copies of the lane's group into buffer q; positions
        // outside lo - H .. hi + H get a benign state
        auto issue = [&](int q) {
            const T* row = in + j * ijs + kz * iks;
            const int p0 = lo - 2 + kP * gi;
#pragma unroll
            for (int h = 0; h < kPairs; ++h) {
                const int x = p0 + 2 * h;
                const T* src = row + x;
                long long ns = ins;
                if constexpr (LEVEL) {
                    if ((xlo && x < lo) || (xhi && x > hi)) {
                        const RowHalo& N = halo[x > hi];
                        src = static_cast<const T*>(N.p) + j * N.js + kz * N.ks + x;
                        ns = N.ns;
                    }
                }
                const bool ok0 = active && x >= lo - H && x <= hi + H;
                const bool ok1 = active && x + 1 >= lo - H && x + 1 <= hi + H;
                if (VEC && ok0 && ok1) {
#pragma unroll
                    for (int n = 0; n < NC; ++n) cp_async_pair(&st[q][n][h][lane], src + n * ns);
                } else {
                    T u[NC];
                    benign(u);
#pragma unroll
                    for (int n = 0; n < NC; ++n) {
                        Pair<T>& d = st[q][n][h][lane];
                        if (ok0) cp_async_elem(&d.a, src + n * ns);
                        else d.a = u[n];
                        if (ok1) cp_async_elem(&d.b, src + n * ns + 1);
                        else d.b = u[n];
                    }
                }
            }
            cp_async_commit();
        };
        issue(0);
        int q = 0;
        const long long e = c_end < box_end ? c_end : box_end;
        for (; c < e; ++c, q ^= 1) {
            // this chunk's group, then on to the next one's copies
            const int x0 = lo - 2 + kP * gi;
            const bool own = owner && active;
            T* __restrict__ po = out + j * ojs + kz * oks + x0;
            T* __restrict__ pf = nullptr;
            if constexpr (!LEVEL)
                if (fl) pf = fl + j * B.flux.js + kz * B.flux.ks + x0;
            g += kRowOwned;
            gi += kRowOwned;
            if (gi >= G || !active) place();
            else active = g < ngroups;
            if (c + 1 < e) issue(q ^ 1);
            else cp_async_commit();
            cp_async_wait_one();

            T U[kP + 2][NC];  // positions x0 - 1 .. x0 + kP
#pragma unroll
            for (int h = 0; h < kPairs; ++h)
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    const Pair<T> v = st[q][n][h][lane];
                    U[1 + 2 * h][n] = v.a;
                    U[2 + 2 * h][n] = v.b;
                }
            shfl_up1(U[kP], U[0]);
            shfl_down1(U[1], U[kP + 1]);
            T UL[kP][NC], UR[kP][NC], URm[NC];
            T F[kP + 1][NC];  // faces x0 .. x0 + kP
            // cell after cell, each face as soon as its states are there and
            // the exchanged one last: the order the compiler overlaps best
            // (4096^2 FP64 357 us when tried; all cells first 409, the exchange early 404)
#pragma unroll
            for (int i = 0; i < kP; ++i) {
                S::cell(U[i], U[i + 1], U[i + 2], k, f.hdtdx, UL[i], UR[i]);
                if (i) S::face(UR[i - 1], UL[i], k, f.half_dx_dt, f.dt_2dx, F[i]);
            }
            if constexpr (S::kReconstruct) {
                shfl_up1(UR[kP - 1], URm);
            } else {  // the state itself, exchanged above
#pragma unroll
                for (int n = 0; n < NC; ++n) URm[n] = U[0][n];
            }
            S::face(URm, UL[0], k, f.half_dx_dt, f.dt_2dx, F[0]);
            shfl_down1(F[0], F[kP]);
            T Un[kP][NC];
#pragma unroll
            for (int i = 0; i < kP; ++i)
#pragma unroll
                for (int n = 0; n < NC; ++n) Un[i][n] = U[i + 1][n] - f.dtdx * (F[i + 1][n] - F[i][n]);
#pragma unroll
            for (int h = 0; h < kPairs; ++h) {
                // pairs start at an even distance from lo: a pair is inside
                // the row, outside it, or half inside at its end
                const int x = x0 + 2 * h;
                const bool in0 = own && do_update && x >= lo && x <= hi, in1 = in0 && x + 1 <= hi;
#pragma unroll
                for (int n = 0; n < NC; ++n) {
                    T* p = po + 2 * h + n * ons;
                    if (VEC) {
                        st_pair_if(p, Un[2 * h][n], Un[2 * h + 1][n], in1);
                        st_global_if(p, Un[2 * h][n], in0 && !in1);
                    } else {
                        st_global_if(p, Un[2 * h][n], in0);
                        st_global_if(p + 1, Un[2 * h + 1][n], in1);
                    }
                }
            }
            if (ws_on) {
#pragma unroll
                for (int i = 0; i < kP; ++i) wsmax.add(S::speed(Un[i], k), own && x0 + i >= lo && x0 + i <= hi);
            }
            if constexpr (!LEVEL) {
                if (fl) {
#pragma unroll
                    for (int i = 0; i < kP; ++i) {
                        const bool face = own && x0 + i >= lo && x0 + i <= hi + 1;
#pragma unroll
                        for (int n = 0; n < NC; ++n) st_global_if(pf + i + n * fns, F[i][n], face);
                    }
                }
            }
        }
        cp_async_wait_all();
    }
    if (ws_on) reduce_ws(wsmax, a.ws_max);
}

}  // namespace bamrex
