// The coarse end of a 2D V-cycle without a gradient term, in one block
// (included by helmholtz.cu, inside its namespace): vcycle_small_kernel's
// phases with everything a phase can do without taken out of it.  A thread
// finds its cells of both colours, their neighbours and the boundary sides
// once per visit of a level and keeps them in registers; gamma and 1 / gamma
// are formed once per cycle (the quotient by Markstein's correction has the
// rounding of the IEEE division); residual and restriction are one phase;
// levels of at most 64 cells run in one warp without block barriers.  The
// cycle is a chain of about 80 phases, so a phase's latency is its cost: from
// 32 x 32 cells down, 16 bottom sweeps, 97 -> 39 us.
#pragma once

constexpr int kSmall2Threads = 512;
constexpr int kSmall2Cells = (int)(kSmallCells / kSmall2Threads);  // cells of a colour per thread, at most

struct SmallLev {
    int n0, n1, ncell;
    double *phi, *rhs, *a, *bx, *by, *g, *gi;
    GsCoef gc;
    ApplyCoef ac;
};

__host__ __device__ __forceinline__ long long small2_level_doubles(const HLev& L)
{
    return 5 * L.ncell + face_count(L, 0) + face_count(L, 1);
}

// Red-black sweeps of one level; every thread of the block calls it.  BND: a
// side of the domain is not periodic.
template <bool BND>
__device__ __forceinline__ void small2_sweeps(const SmallLev& L, const HOp& op, int sweeps)
{
    const int n0 = L.n0, n1 = L.n1, nxh = (n0 + 1) / 2, half = nxh * n1;
    const bool px = !BND || op.bc_lo[0] == BAMREX_LINOP_PERIODIC, py = !BND || op.bc_lo[1] == BAMREX_LINOP_PERIODIC;
    const bool one_warp = half <= 32;
    if (one_warp && threadIdx.x >= 32) {
        __syncthreads();
        return;
    }
    // per cell of each colour: its index (-1: none), its neighbours', its low
    // x face's, and the non-periodic sides it touches
    struct Cell {
        int c, w, e, s, n, f, side;
    } cell[2][kSmall2Cells];
#pragma unroll
    for (int m = 0; m < kSmall2Cells; ++m) {
        const int t = threadIdx.x + m * kSmall2Threads;
        const int j = t / nxh;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            Cell& x = cell[k][m];
            const int i = 2 * (t - j * nxh) + ((j + k) & 1);
            const int q = j * n0 + i;
            x.c = t < half && i < n0 ? q : -1;
            x.w = i > 0 ? q - 1 : q + n0 - 1;
            x.e = i + 1 < n0 ? q + 1 : q + 1 - n0;
            x.s = j > 0 ? q - n0 : q + (n1 - 1) * n0;
            x.n = j + 1 < n1 ? q + n0 : q - (n1 - 1) * n0;
            x.f = q + j;  // (rows of x faces are one longer)
            x.side = (!px && i == 0 ? kMgXlo : 0) | (!px && i + 1 == n0 ? kMgXhi : 0) | (!py && j == 0 ? kMgYlo : 0) |
                     (!py && j + 1 == n1 ? kMgYhi : 0);
        }
    }
    const double dh0 = L.gc.dh[0], dh1 = L.gc.dh[1];
    double* const phi = L.phi;
    auto update = [&](const Cell& x) {
        const int q = x.c;
        if (q < 0) return;
        const double pm0 = phi[x.w], pp0 = phi[x.e], pm1 = phi[x.s], pp1 = phi[x.n];
        const double bl0 = L.bx[x.f], bh0 = L.bx[x.f + 1], bl1 = L.by[q], bh1 = L.by[q + n0];
        double rho = dh0 * (bl0 * pm0 + bh0 * pp0);
        rho = rho + dh1 * (bl1 * pm1 + bh1 * pp1);
        const double num = L.rhs[q] + rho, gam = L.g[q], inv = L.gi[q];
        const double q0 = num * inv;
        double v = fma(fma(-gam, q0, num), inv, q0);
        if (BND && x.side) {
            const double pc = phi[q];
            const double pmv[3] = { pm0, pm1, 0.0 }, ppv[3] = { pp0, pp1, 0.0 };
            double pm[3], pp[3], cfm[3] = { 0, 0, 0 }, cfp[3] = { 0, 0, 0 };
            for (int d = 0; d < 2; ++d) {
                const bool lo = x.side & (d == 0 ? kMgXlo : kMgYlo), hi = x.side & (d == 0 ? kMgXhi : kMgYhi);
                cfm[d] = lo ? (op.bc_lo[d] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) : 0.0;
                cfp[d] = hi ? (op.bc_hi[d] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) : 0.0;
                pm[d] = lo ? cfm[d] * pc : pmv[d];
                pp[d] = hi ? cfp[d] * pc : ppv[d];
            }
            const double bl[3] = { bl0, bl1, 0.0 }, bh[3] = { bh0, bh1, 0.0 }, cc[3] = { 0.0, 0.0, 0.0 };
            v = gsrb_core<2>(op, L.gc, L.a[q], bl, bh, cc, pc, pm, pp, cfm, cfp, L.rhs[q]);
        }
        phi[q] = v;
    };
    const bool more = half > kSmall2Threads;
#pragma unroll 1
    for (int it = 0; it < sweeps; ++it) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            update(cell[k][0]);
            if (more)
                for (int m = 1; m < kSmall2Cells; ++m) update(cell[k][m]);
            if (one_warp) __syncwarp();
            else __syncthreads();
        }
    }
    if (one_warp) __syncthreads();
}

template <bool BND>
__global__ void __launch_bounds__(kSmall2Threads) vcycle_small2_kernel(const HLevs lv, const HOp op, int nu1, int nu2,
                                                                       int bottom)
{
    extern __shared__ double small_sm2[];
    __shared__ SmallLev S[kSmallLevels];
    const int nl = lv.n;
    // a thread per level lays it out and forms its coefficients
    if (threadIdx.x < nl) {
        double* p = small_sm2;
        for (int l = 0; l < (int)threadIdx.x; ++l) p += small2_level_doubles(lv.lev[l]);
        {
            const int l = threadIdx.x;
            const HLev& G = lv.lev[l];
            SmallLev& L = S[l];
            L.n0 = G.n[0];
            L.n1 = G.n[1];
            L.ncell = (int)G.ncell;
            L.gc = gs_coef(G, op);
            L.ac = apply_coef(G, op);
            double** f[] = { &L.phi, &L.rhs, &L.a, &L.g, &L.gi };
            for (double** v : f) {
                *v = p;
                p += G.ncell;
            }
            L.bx = p;
            p += face_count(G, 0);
            L.by = p;
            p += face_count(G, 1);
        }
    }
    __syncthreads();
    for (int l = 0; l < nl; ++l) {
        const HLev& G = lv.lev[l];
        const SmallLev& L = S[l];
        const GsCoef gc = L.gc;
        for (int q = threadIdx.x; q < (int)face_count(G, 0); q += kSmall2Threads) L.bx[q] = G.b[0][q];
        for (int q = threadIdx.x; q < (int)face_count(G, 1); q += kSmall2Threads) L.by[q] = G.b[1][q];
        for (int q = threadIdx.x; q < L.ncell; q += kSmall2Threads) {
            const double a = G.a[q];
            L.a[q] = a;
            const int j = q / L.n0;
            double g = op.ascal * a;
            g = g + gc.dh[0] * (G.b[0][q + j] + G.b[0][q + j + 1]);
            g = g + gc.dh[1] * (G.b[1][q] + G.b[1][q + L.n0]);
            L.g[q] = g;
            L.gi[q] = 1.0 / g;
            L.phi[q] = l == 0 ? G.phi[q] : 0.0;
            if (l == 0) L.rhs[q] = G.rhs[q];
        }
    }
    __syncthreads();
    for (int l = 0; l + 1 < nl; ++l) {
        const SmallLev &F = S[l], &C = S[l + 1];
        small2_sweeps<BND>(F, op, nu1);
        // residual of the four children and their mean (apply_value,
        // restrict_cell)
        const ApplyCoef ac = F.ac;
        for (int q = threadIdx.x; q < C.ncell; q += kSmall2Threads) {
            const int J = q / C.n0, I = q - J * C.n0;
            double sum = 0.0;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
                const int i = 2 * I + (t & 1), j = 2 * J + (t >> 1), f = j * F.n0 + i;
                const double xc = F.phi[f];
                auto at = [&](int d, int st, int pos, int len, int stride) {
                    const int x = pos + st;
                    if (x >= 0 && x < len) return F.phi[f + st * stride];
                    const int bc = st < 0 ? op.bc_lo[d] : op.bc_hi[d];
                    if (!BND || bc == BAMREX_LINOP_PERIODIC) return F.phi[f - st * (len - 1) * stride];
                    return (bc == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) * xc;
                };
                const double xm0 = at(0, -1, i, F.n0, 1), xp0 = at(0, 1, i, F.n0, 1);
                const double xm1 = at(1, -1, j, F.n1, F.n0), xp1 = at(1, 1, j, F.n1, F.n0);
                double v = op.ascal * F.a[f] * xc;
                v = v - ac.dh[0] * (F.bx[f + j + 1] * (xp0 - xc) - F.bx[f + j] * (xc - xm0));
                v = v - ac.dh[1] * (F.by[f + F.n0] * (xp1 - xc) - F.by[f] * (xc - xm1));
                sum = sum + (F.rhs[f] - v);
            }
            C.rhs[q] = sum * 0.25;
        }
        __syncthreads();
    }
    small2_sweeps<BND>(S[nl - 1], op, bottom);
    for (int l = nl - 2; l >= 0; --l) {
        const SmallLev &F = S[l], &C = S[l + 1];
        for (int q = threadIdx.x; q < F.ncell; q += kSmall2Threads) {
            const int j = q / F.n0, i = q - j * F.n0;
            F.phi[q] = F.phi[q] + C.phi[(j >> 1) * C.n0 + (i >> 1)];
        }
        __syncthreads();
        small2_sweeps<BND>(F, op, nu2);
    }
    for (int q = threadIdx.x; q < S[0].ncell; q += kSmall2Threads) lv.lev[0].phi[q] = S[0].phi[q];
}
