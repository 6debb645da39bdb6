// A run of steps of a 1D level that is one short box (AmrLevelAdv::advance in
// a loop, Source/AmrLevelAdv_advance.cpp:60-260, with computeNewDt between),
// in one block: both state buffers stay in shared memory, and ghost cells,
// sweep, wave-speed maximum and next dt of a step are one pass over the line
// with one barrier.
//
// A step of a short line does no work to speak of: as three launches (ghost
// fill, sweep, dt) it takes 10.3 - 12.3 us whatever its length, all of it
// launch and drain.  In here (FP64 MUSCL-Hancock) 1.25 us up to 90 cells, the
// chain of one cell's arithmetic, 1.95 at 480 and 1.2 more per further 480,
// the FP64 pipe of one SM; 50 steps of 400 cells 630 -> 133 us with the call.  Here a chunk is 32 consecutive cells, one per lane,
// of which lanes 1 .. 30 store theirs; the neighbours' states come by
// shuffle.  The owner of a cell next to an end writes the ghost cells it
// determines.  Every thread forms the step's dt for itself from the warps'
// maxima, so nothing waits for one thread's result.
#include <cuda_runtime.h>

#include <algorithm>

#include "bamrex_cuda.h"
#include "common.cuh"
#include "euler.cuh"
#include "launch.h"
#include "sweep.cuh"

namespace bamrex {

namespace {

constexpr int kLineThreads = 512;  // 16 warps of at most 128 registers a thread
constexpr int kLineOwned = 30;
constexpr int kLineGhost = 2;
constexpr int kLineMaxCells = 4 * kLineOwned * kLineThreads / 32;  // 1920: four passes (the rule of line_run, abi.cu)

// Largest of the lanes' values; non-negative doubles order like their bits.
__device__ __forceinline__ unsigned long long warp_max_bits(unsigned long long v)
{
    const unsigned hi = (unsigned)(v >> 32);
    const unsigned top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned low = __reduce_max_sync(0xffffffffu, hi == top ? (unsigned)v : 0u);
    return ((unsigned long long)top << 32) | low;
}

// A NaN as the NaN pattern, above every other value.
template <typename T>
__device__ __forceinline__ unsigned long long speed_bits(const WsMax<T>& w)
{
    if (w.nan()) return 0x7ff8000000000000ull;
    const double v = (double)w.v;
    return v < 1e-140 ? 0ull : (unsigned long long)__double_as_longlong(v);  // wave_speed_f64's offset
}

template <typename T>
struct Line {
    T* u;   // NC rows of w = n + 2 kLineGhost cells
    int n, w;
    __device__ __forceinline__ T& at(int c, int x) const { return u[c * w + x + kLineGhost]; }
    __device__ __forceinline__ void put3(int x, const T (&v)[3], bool mirror) const
    {
        at(0, x) = v[0];
        at(1, x) = mirror ? -v[1] : v[1];
        at(2, x) = v[2];
    }
    // cell x and the ghost cells that copy it
    __device__ __forceinline__ void put(int x, const T (&v)[3], int bc_lo, int bc_hi) const
    {
        put3(x, v, false);
        if (x < kLineGhost) {
            if (bc_lo == BAMREX_BC_PERIODIC) put3(n + x, v, false);
            else if (bc_lo == BAMREX_BC_REFLECTIVE) put3(-1 - x, v, true);
            else if (x == 0)
                for (int g = 1; g <= kLineGhost; ++g) put3(-g, v, false);
        }
        if (x >= n - kLineGhost) {
            if (bc_hi == BAMREX_BC_PERIODIC) put3(x - n, v, false);
            else if (bc_hi == BAMREX_BC_REFLECTIVE) put3(2 * n - 1 - x, v, true);
            else if (x == n - 1)
                for (int g = 0; g < kLineGhost; ++g) put3(n + g, v, false);
        }
    }
};

template <typename T, int METHOD, int LIM>
__global__ void __launch_bounds__(kLineThreads, 1) line_run_kernel(const LineArgs a)
{
    using S = Scheme<T, 1, 0, METHOD, LIM>;
    constexpr int NC = 3;
    extern __shared__ double line_smem[];
    __shared__ unsigned long long warp_ws[2][kLineThreads / 32];
    StepScalars s;
    if (a.init) {
        s = StepScalars{};
        s.time = a.time;
        s.stop_time = a.stop_time;
    } else {
        s = *a.scal;
        if (s.done) return;
    }
    const K<T> k(a.k);
    const double dxs[3] = { a.dx, a.dx, a.dx };
    const int n = a.n, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nchunks = (n + kLineOwned - 1) / kLineOwned;
    T* const mem = reinterpret_cast<T*>(line_smem);
    const int w = n + 2 * kLineGhost;
    auto line = [&](int q) { return Line<T>{ mem + (q ? NC * w : 0), n, w }; };
    auto reduce = [&](unsigned long long bits, int q) {
        const unsigned long long m = warp_max_bits(bits);
        if (lane == 0) warp_ws[q][warp] = m;
        __syncthreads();
        return warp_max_bits(lane < nwarps ? warp_ws[q][lane] : 0ull);
    };

    {
        const T* in = static_cast<const T*>(a.in);
        double v = 0.0;
        bool nan = false;
        for (int x = threadIdx.x; x < n; x += blockDim.x) {
            const T U[NC] = { in[x], in[x + a.in_ns], in[x + 2 * a.in_ns] };
            line(0).put(x, U, a.bc_lo, a.bc_hi);
            // the stand-alone maximum's formula, and like it an infinite
            // speed stays one (launch_max_wave_speed)
            double ws;
            if constexpr (sizeof(T) == 8 && LIM >= 0) ws = wave_speed_f64<1>(U, k);
            else ws = (double)wave_speed<T, 1>(U, k);
            v = fmax(v, ws);
            nan = nan || ws != ws;
        }
        if (sizeof(T) == 8 && LIM >= 0 && v < 1e-140) v = 0.0;
        const unsigned long long m = reduce(nan ? 0x7ff8000000000000ull : (unsigned long long)__double_as_longlong(v), 0);
        if (a.init) {
            s.ws_bits = m;
            next_step_scalars(s, 1, dxs, a.cfl, false);
        }
    }
    int q = 0;
    for (int step = 0; step < a.nsteps && !s.done; ++step, q ^= 1) {
        StepFactors<T> f;
        step_factors(s.dt, a.dx, f);
        WsMax<T> v;
        for (int c = warp; c < nchunks; c += nwarps) {
            const int x = kLineOwned * c - 1 + lane;
            const int xr = min(x, n);  // lanes past the end repeat the ghost cell
            T U[3][NC], UL[NC], UR[NC], URm[NC], F[NC], Fp[NC], Un[NC];
#pragma unroll
            for (int i = 0; i < 3; ++i)
#pragma unroll
                for (int m = 0; m < NC; ++m) U[i][m] = line(q).at(m, xr - 1 + i);
            S::cell(U[0], U[1], U[2], k, f.hdtdx, UL, UR);
#pragma unroll
            for (int m = 0; m < NC; ++m) URm[m] = __shfl_up_sync(0xffffffffu, UR[m], 1);
            S::face(URm, UL, k, f.half_dx_dt, f.dt_2dx, F);
#pragma unroll
            for (int m = 0; m < NC; ++m) Fp[m] = __shfl_down_sync(0xffffffffu, F[m], 1);
#pragma unroll
            for (int m = 0; m < NC; ++m) Un[m] = U[1][m] - f.dtdx * (Fp[m] - F[m]);
            const bool own = lane >= 1 && lane <= kLineOwned && x < n;
            v.add(S::speed(Un, k), own);
            if (own) line(q ^ 1).put(x, Un, a.bc_lo, a.bc_hi);
        }
        s.ws_bits = reduce(speed_bits(v), (step + 1) & 1);
        next_step_scalars(s, 1, dxs, a.cfl, true);
    }
    const int taken = s.steps - (a.init ? 0 : a.scal->steps);
    if (taken > 0) {
        // both buffers as the steps leave them: the state and the one before
        T* now = static_cast<T*>(taken & 1 ? a.out : a.in);
        T* old = static_cast<T*>(taken & 1 ? a.in : a.out);
        const long long nns = taken & 1 ? a.out_ns : a.in_ns, ons = taken & 1 ? a.in_ns : a.out_ns;
        for (int x = threadIdx.x; x < n; x += blockDim.x)
#pragma unroll
            for (int m = 0; m < NC; ++m) {
                now[x + m * nns] = line(q).at(m, x);
                old[x + m * ons] = line(q ^ 1).at(m, x);
            }
    }
    __syncthreads();  // everyone has read scal
    if (threadIdx.x == 0) *a.scal = s;
}

template <typename T>
const void* pick_line_kernel(int method, int fast_lim)
{
    if (method == M_MUSCL && fast_lim >= 0) {
        switch (fast_lim) {
        case LIM_MINBEE: return (const void*)line_run_kernel<T, M_MUSCL, LIM_MINBEE>;
        case LIM_VAN_LEER: return (const void*)line_run_kernel<T, M_MUSCL, LIM_VAN_LEER>;
        case LIM_VAN_ALBADA: return (const void*)line_run_kernel<T, M_MUSCL, LIM_VAN_ALBADA>;
        case LIM_SUPERBEE: return (const void*)line_run_kernel<T, M_MUSCL, LIM_SUPERBEE>;
        default: return nullptr;
        }
    }
    switch (method) {
    case M_MUSCL: return (const void*)line_run_kernel<T, M_MUSCL, -1>;
    case M_HLLC: return (const void*)line_run_kernel<T, M_HLLC, -1>;
    case M_SLIC: return (const void*)line_run_kernel<T, M_SLIC, -1>;
    case M_FORCE: return (const void*)line_run_kernel<T, M_FORCE, -1>;
    case M_LF: return (const void*)line_run_kernel<T, M_LF, -1>;
    default: return nullptr;
    }
}

}  // namespace

// At least four cells, so that a ghost cell copies a cell of the other half.
bool line_run_supported(int n) { return n >= 2 * kLineGhost && n <= kLineMaxCells; }

cudaError_t launch_line_run(int method, bool fp32, const LineArgs& a, cudaStream_t s)
{
    const int lim = fast_limiter(1, method, fp32, a.k);
    const void* fn = fp32 ? pick_line_kernel<float>(method, lim) : pick_line_kernel<double>(method, lim);
    if (!fn) return cudaErrorInvalidValue;
    const auto line_bytes = [fp32](int n) { return 2 * 3 * (size_t)(n + 2 * kLineGhost) * (fp32 ? sizeof(float) : sizeof(double)); };
    const size_t smem = line_bytes(a.n);
    if (smem > 40 * 1024) {
        // the limit is the kernel's, shared by every level and thread that
        // uses it: always the longest line's, so that no launch lowers it
        // under another's
        const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)line_bytes(kLineMaxCells));
        if (e != cudaSuccess) return e;
    }
    const int chunks = (a.n + kLineOwned - 1) / kLineOwned;
    void* args[] = { (void*)&a };
    return cudaLaunchKernel(fn, dim3(1), dim3(32 * std::min(chunks, kLineThreads / 32)), args, smem, s);
}

}  // namespace bamrex
