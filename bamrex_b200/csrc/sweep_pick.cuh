// Kernel selection for the sweep launches; instantiated once per storage
// type (sweep_f64.cu, sweep_f32.cu) so the two compile in parallel.
#pragma once

#include "sweep.cuh"
#include "sweep_row.cuh"

namespace bamrex {

// march: the x sweep as one thread per row (D >= 2); ignored for y / z.
// rows: whose fabs the x sweep by row groups works on (kRows*; FP32 only on
// levels).
template <typename T>
const void* pick_sweep_kernel(int D, int dir, int method, int fast_lim, bool march, int rows);

namespace detail {

template <typename T, int D, int DIR, bool MARCH, int M, int LIM>
const void* kernel_ptr(int rows)
{
    if constexpr (DIR == 0 && !MARCH) {
        if constexpr (sizeof(T) == 8) {
            if (rows == kRowsBoxPaired) return (const void*)sweep_row_kernel<T, D, M, LIM, false, true>;
            if (rows == kRowsBox) return (const void*)sweep_row_kernel<T, D, M, LIM, false, false>;
        }
        return (const void*)sweep_row_kernel<T, D, M, LIM, true, true>;
    } else return (const void*)sweep_s_kernel<T, D, DIR, M, LIM>;
}

// fast_lim >= 0: the fast MUSCL-Hancock path with that limiter; -1: general
template <typename T, int D, int DIR, bool MARCH>
const void* pick_method(int method, int fast_lim, int rows)
{
    if (method == M_MUSCL && fast_lim >= 0) {
        switch (fast_lim) {
        case LIM_MINBEE: return kernel_ptr<T, D, DIR, MARCH, M_MUSCL, LIM_MINBEE>(rows);
        case LIM_VAN_LEER: return kernel_ptr<T, D, DIR, MARCH, M_MUSCL, LIM_VAN_LEER>(rows);
        case LIM_VAN_ALBADA: return kernel_ptr<T, D, DIR, MARCH, M_MUSCL, LIM_VAN_ALBADA>(rows);
        case LIM_SUPERBEE: return kernel_ptr<T, D, DIR, MARCH, M_MUSCL, LIM_SUPERBEE>(rows);
        default: return nullptr;
        }
    }
    switch (method) {
    case M_MUSCL: return kernel_ptr<T, D, DIR, MARCH, M_MUSCL, -1>(rows);
    case M_HLLC: return kernel_ptr<T, D, DIR, MARCH, M_HLLC, -1>(rows);
    case M_SLIC: return kernel_ptr<T, D, DIR, MARCH, M_SLIC, -1>(rows);
    case M_FORCE: return kernel_ptr<T, D, DIR, MARCH, M_FORCE, -1>(rows);
    case M_LF: return kernel_ptr<T, D, DIR, MARCH, M_LF, -1>(rows);
    default: return nullptr;
    }
}

}  // namespace detail

template <typename T>
const void* pick_sweep_kernel(int D, int dir, int method, int fast_lim, bool march, int rows)
{
    using namespace detail;
    if (D == 1 && dir == 0) return pick_method<T, 1, 0, false>(method, fast_lim, rows);
    if (D == 2 && dir == 0)
        return march ? pick_method<T, 2, 0, true>(method, fast_lim, rows) : pick_method<T, 2, 0, false>(method, fast_lim, rows);
    if (D == 2 && dir == 1) return pick_method<T, 2, 1, false>(method, fast_lim, rows);
    if (D == 3 && dir == 0)
        return march ? pick_method<T, 3, 0, true>(method, fast_lim, rows) : pick_method<T, 3, 0, false>(method, fast_lim, rows);
    if (D == 3 && dir == 1) return pick_method<T, 3, 1, false>(method, fast_lim, rows);
    if (D == 3 && dir == 2) return pick_method<T, 3, 2, false>(method, fast_lim, rows);
    return nullptr;
}

}  // namespace bamrex
