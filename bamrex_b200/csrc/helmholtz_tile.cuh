// Half a 2D V-cycle level in one launch (included by helmholtz.cu, inside its
// namespace): a block owns a tile of 32 x 32 cells and works on a window
// around it, wide enough that every value of the tile is the one the
// grid-wide phases give.
//  * PRE: two red-black sweeps from a zero guess, the residual, and its
//    restriction to the next level's right-hand side.
//  * POST: the coarse correction added, then two red-black sweeps.
// A colour's cells never read each other, so the order of the updates does
// not matter; the window's edge cells are updated from incomplete neighbours
// and spoil one ring per colour phase, which the halo (3 pairs of columns; 4
// rows, 5 with the residual) absorbs.  Each cell's arithmetic is gsrb_core's
// and apply_value's, term by term (without a gradient term the boundary
// factor sums vanish away from a non-periodic boundary), so the V-cycle is
// the grid-wide one bit for bit.
//
// A thread owns pairs of cells (one red, one black) and keeps their face
// coefficients and 1 / gamma in registers, their rhs and gamma in shared
// memory of its own; phi is shared, the two colours apart, so that 32 lanes
// read consecutive words.  The quotient by gamma is Markstein's: 1 / gamma
// once per cell, then two corrections' worth of multiply-adds with the
// rounding of the IEEE division.  Per cell a level reads a, b, rhs (and phi)
// once for two sweeps instead of once per sweep.
//
// 2048^2, before -> now: two sweeps, residual and restriction, four launches
// of 190 us in all -> 118 us; prolongation and two sweeps, three launches of
// 170 us -> 120 us (a floor of about 32 us of HBM traffic; the window is 1.8
// times the tile, and instruction issue bounds it).  Solve to 1e-12: 16.4 ->
// 10.1 ms with the one-block coarse cycle of helmholtz_small.cuh.
#pragma once

constexpr int kMgTile = 32;
constexpr int kMgThreads = 320;  // 3 pairs a thread; two blocks per SM (one of 480: 10.6 ms a 2048^2 solve, two of 320: 10.1)

template <bool PRE>
struct MgWin {
    static constexpr int HX = 6, HY = PRE ? 5 : 4;
    static constexpr int WP = (kMgTile + 2 * HX) / 2;     // pairs per row
    static constexpr int WR = kMgTile + 2 * HY;           // rows
    static constexpr int SP = WP + 2;                     // stored pairs (one beyond each end)
    static constexpr int kPairs = (WP * WR + kMgThreads - 1) / kMgThreads;
    static constexpr int kSmem = (2 * (WR + 2) * SP + 4 * kPairs * kMgThreads + (PRE ? kMgTile * (kMgTile + 1) : 0)) * 8;
};

// bits of a pair: its window position is updated; the domain's non-periodic
// sides it touches
// and whether its second cell is the red one (odd rows; a periodic image keeps
// its row's parity: the sides are even).
enum { kMgOn = 1, kMgXlo = 2, kMgXhi = 4, kMgYlo = 8, kMgYhi = 16, kMgSwap = 32 };

// BND: a side of the domain is not periodic.
template <bool PRE, bool BND>
__global__ void __launch_bounds__(kMgThreads, 2) mg_tile_kernel(const HLev L, const HOp op, const double* __restrict__ rhs,
                                                                const double* __restrict__ phi,
                                                                const double* __restrict__ coarse, double* __restrict__ out,
                                                                const HLev C)
{
    using W = MgWin<PRE>;
    constexpr int NP = W::kPairs;
    extern __shared__ double mg_smem[];
    double* const sc[2] = { mg_smem, mg_smem + (W::WR + 2) * W::SP };  // a colour's cells, [row + 1][pair + 1]
    double* sf = mg_smem + 2 * (W::WR + 2) * W::SP;  // rhs and gamma of a thread's own cells: [2 m + colour][thread]
    double* sg = sf + 2 * NP * kMgThreads;
    double (*sres)[kMgTile + 1] = reinterpret_cast<double (*)[kMgTile + 1]>(sg + 2 * NP * kMgThreads);
    const GsCoef gc = gs_coef(L, op);
    const int nx = L.n[0], ny = L.n[1];
    const bool px = !BND || op.bc_lo[0] == BAMREX_LINOP_PERIODIC, py = !BND || op.bc_lo[1] == BAMREX_LINOP_PERIODIC;
    const int tx = (nx + kMgTile - 1) / kMgTile;
    const int i0 = (blockIdx.x % tx) * kMgTile, j0 = (blockIdx.x / tx) * kMgTile;
    const int tid = threadIdx.x;

    // the pair at window row wr, pair wp in the domain (a periodic image past
    // its sides); false outside a non-periodic side
    auto locate = [&](int wr, int wp, int& ci, int& cj) {
        ci = i0 - W::HX + 2 * wp;
        cj = j0 - W::HY + wr;
        bool in = true;
        if (ci < 0 || ci >= nx) {
            in = px;
            ci %= nx;
            ci = ci < 0 ? ci + nx : ci;
        }
        if (cj < 0 || cj >= ny) {
            in = in && py;
            cj %= ny;
            cj = cj < 0 ? cj + ny : cj;
        }
        return in;
    };
    // per pair, of the red (0) and black (1) cell: the x and y faces below and
    // above and 1 / gamma.  Every load is issued before the first
    // use (pairs outside the domain read cell 0).
    double xl[2][NP], xh[2][NP], yl[2][NP], yh[2][NP], gi[2][NP];
    int flags[NP], at[NP];  // at: the pair's place in a colour's array
    {
        double2 a2[NP], f2[NP], bl[NP], bh[NP], p2[NP];
        double pc[NP], x0[NP], x1[NP], x2[NP];
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            const int q = tid + m * kMgThreads;
            const int wr = q / W::WP, wp = q - wr * W::WP;
            int ci, cj;
            const bool in = locate(wr, wp, ci, cj) && q < W::WP * W::WR;
            ci = in ? ci : 0;
            cj = in ? cj : 0;
            const long long c = (long long)cj * nx + ci;
            const double* bx = L.b[0] + (long long)cj * (nx + 1) + ci;
            a2[m] = *reinterpret_cast<const double2*>(L.a + c);
            f2[m] = *reinterpret_cast<const double2*>(rhs + c);
            bl[m] = *reinterpret_cast<const double2*>(L.b[1] + c);
            bh[m] = *reinterpret_cast<const double2*>(L.b[1] + c + nx);
            x0[m] = bx[0];
            x1[m] = bx[1];
            x2[m] = bx[2];
            if constexpr (!PRE) {
                p2[m] = *reinterpret_cast<const double2*>(phi + c);
                pc[m] = coarse[(long long)(cj >> 1) * (nx >> 1) + (ci >> 1)];
            }
            // edge rows and pairs of the window are not updated, except
            // where the window ends with the domain
            int fl = 0;
            if (!px) fl |= (ci == 0 ? kMgXlo : 0) | (ci + 2 == nx ? kMgXhi : 0);
            if (!py) fl |= (cj == 0 ? kMgYlo : 0) | (cj + 1 == ny ? kMgYhi : 0);
            const bool edge = (wr == 0 && !(fl & kMgYlo)) || (wr == W::WR - 1 && !(fl & kMgYhi)) ||
                              (wp == 0 && !(fl & kMgXlo)) || (wp == W::WP - 1 && !(fl & kMgXhi));
            flags[m] = (in ? (fl | (edge ? 0 : kMgOn)) : 0) | (((j0 - W::HY + wr) & 1) ? kMgSwap : 0);
            at[m] = q < W::WP * W::WR ? (wr + 1) * W::SP + wp + 1 : W::SP + 1;
        }
#pragma unroll
        for (int m = 0; m < NP; ++m) {
            const int q = tid + m * kMgThreads;
            const bool swap = flags[m] & kMgSwap;
            // gamma of the pair's first and second cell
            double ga = op.ascal * a2[m].x, gb = op.ascal * a2[m].y;
            ga = ga + gc.dh[0] * (x0[m] + x1[m]);
            gb = gb + gc.dh[0] * (x1[m] + x2[m]);
            ga = ga + gc.dh[1] * (bl[m].x + bh[m].x);
            gb = gb + gc.dh[1] * (bl[m].y + bh[m].y);
            const double gr = swap ? gb : ga, gk = swap ? ga : gb;
            gi[0][m] = 1.0 / gr;
            gi[1][m] = 1.0 / gk;
            sg[(2 * m) * kMgThreads + tid] = gr;
            sg[(2 * m + 1) * kMgThreads + tid] = gk;
            sf[(2 * m) * kMgThreads + tid] = swap ? f2[m].y : f2[m].x;
            sf[(2 * m + 1) * kMgThreads + tid] = swap ? f2[m].x : f2[m].y;
            xl[0][m] = swap ? x1[m] : x0[m];
            xh[0][m] = swap ? x2[m] : x1[m];
            xl[1][m] = swap ? x0[m] : x1[m];
            xh[1][m] = swap ? x1[m] : x2[m];
            yl[0][m] = swap ? bl[m].y : bl[m].x;
            yl[1][m] = swap ? bl[m].x : bl[m].y;
            yh[0][m] = swap ? bh[m].y : bh[m].x;
            yh[1][m] = swap ? bh[m].x : bh[m].y;
            if (q < W::WP * W::WR) {
                double p0 = 0.0, p1 = 0.0;
                if constexpr (!PRE) {
                    p0 = p2[m].x + pc[m];
                    p1 = p2[m].y + pc[m];
                }
                sc[swap][at[m]] = p0;
                sc[!swap][at[m]] = p1;
            }
        }
    }
    __syncthreads();

#pragma unroll 1
    for (int sweep = 0; sweep < 2; ++sweep) {
#pragma unroll
        for (int k = 0; k < 2; ++k) {  // red, black
            const double* o = sc[k ^ 1];
            double v[NP];
#pragma unroll
            for (int m = 0; m < NP; ++m) {
                // 1 when this colour's cell is the pair's second
                const int second = (k == 0) == ((flags[m] & kMgSwap) != 0);
                const double* c = o + at[m] + second;
                const double pm0 = c[-1], pp0 = c[0], pm1 = o[at[m] - W::SP], pp1 = o[at[m] + W::SP];
                double rho = gc.dh[0] * (xl[k][m] * pm0 + xh[k][m] * pp0);
                rho = rho + gc.dh[1] * (yl[k][m] * pm1 + yh[k][m] * pp1);
                // the quotient by 1/gamma and Markstein's correction: the
                // rounding of the IEEE division (Markstein 2000)
                const double rh = sf[(2 * m + k) * kMgThreads + tid], gam = sg[(2 * m + k) * kMgThreads + tid];
                const double num = rh + rho;
                const double q0 = num * gi[k][m];
                v[m] = fma(fma(-gam, q0, num), gi[k][m], q0);
                if (BND && (flags[m] & (kMgXlo | kMgXhi | kMgYlo | kMgYhi))) {
                    const double pcv = sc[k][at[m]];
                    const double pmv[3] = { pm0, pm1, 0.0 }, ppv[3] = { pp0, pp1, 0.0 };
                    double pm[3], pp[3], cfm[3] = { 0, 0, 0 }, cfp[3] = { 0, 0, 0 };
                    const bool lo[2] = { (flags[m] & kMgXlo) && !second, (flags[m] & kMgYlo) != 0 };
                    const bool hi[2] = { (flags[m] & kMgXhi) && second, (flags[m] & kMgYhi) != 0 };
                    for (int d = 0; d < 2; ++d) {
                        cfm[d] = lo[d] ? (op.bc_lo[d] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) : 0.0;
                        cfp[d] = hi[d] ? (op.bc_hi[d] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) : 0.0;
                        pm[d] = lo[d] ? cfm[d] * pcv : pmv[d];
                        pp[d] = hi[d] ? cfp[d] * pcv : ppv[d];
                    }
                    const double bl[3] = { xl[k][m], yl[k][m], 0.0 }, bh[3] = { xh[k][m], yh[k][m], 0.0 };
                    const double cc[3] = { 0.0, 0.0, 0.0 };
                    const int r = at[m] / W::SP - 1, p = at[m] % W::SP - 1;
                    int ci, cj;
                    locate(r, p, ci, cj);
                    const double a = L.a[(long long)cj * nx + ci + second];
                    v[m] = gsrb_core<2>(op, gc, a, bl, bh, cc, pcv, pm, pp, cfm, cfp, rh);
                }
            }
#pragma unroll
            for (int m = 0; m < NP; ++m)
                if (flags[m] & kMgOn) sc[k][at[m]] = v[m];
            __syncthreads();
        }
    }

    // the tile's cells
    const ApplyCoef ac = apply_coef(L, op);
#pragma unroll
    for (int m = 0; m < NP; ++m) {
        const int q = threadIdx.x + m * kMgThreads;
        const int wr = q / W::WP, wp = q - wr * W::WP;
        const int li = 2 * wp - W::HX, lj = wr - W::HY;
        if (q >= W::WP * W::WR || li < 0 || li >= kMgTile || lj < 0 || lj >= kMgTile || i0 + li >= nx || j0 + lj >= ny) continue;
        const int swap = (j0 + lj) & 1;
        double2 u;
        u.x = sc[swap][at[m]];
        u.y = sc[swap ^ 1][at[m]];
        const long long c = (long long)(j0 + lj) * nx + i0 + li;
        *reinterpret_cast<double2*>(out + c) = u;
        if constexpr (PRE) {
            const double2 a2 = *reinterpret_cast<const double2*>(L.a + c);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int second = (k == 0) == (swap != 0);  // the colour's cell in the pair
                const double* o = sc[k ^ 1] + at[m];
                const double xc = second ? u.y : u.x;
                double xm0 = o[second - 1], xp0 = o[second], xm1 = o[-W::SP], xp1 = o[W::SP];
                if (BND && (flags[m] & (kMgXlo | kMgXhi | kMgYlo | kMgYhi))) {
                    if ((flags[m] & kMgXlo) && !second) xm0 = (op.bc_lo[0] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) * xc;
                    if ((flags[m] & kMgXhi) && second) xp0 = (op.bc_hi[0] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) * xc;
                    if (flags[m] & kMgYlo) xm1 = (op.bc_lo[1] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) * xc;
                    if (flags[m] & kMgYhi) xp1 = (op.bc_hi[1] == BAMREX_LINOP_NEUMANN ? 1.0 : -1.0) * xc;
                }
                double v = op.ascal * (second ? a2.y : a2.x) * xc;
                v = v - ac.dh[0] * (xh[k][m] * (xp0 - xc) - xl[k][m] * (xc - xm0));
                v = v - ac.dh[1] * (yh[k][m] * (xp1 - xc) - yl[k][m] * (xc - xm1));
                sres[lj][li + second] = sf[(2 * m + k) * kMgThreads + tid] - v;
            }
        }
    }
    if constexpr (PRE) {
        __syncthreads();
        // restrict_cell on the tile's 16 x 16 coarse cells
        const int I = threadIdx.x % (kMgTile / 2), J = threadIdx.x / (kMgTile / 2);
        const int gI = i0 / 2 + I, gJ = j0 / 2 + J;
        if (J < kMgTile / 2 && gI < C.n[0] && gJ < C.n[1]) {
            double s = 0.0;
            s = s + sres[2 * J][2 * I];
            s = s + sres[2 * J][2 * I + 1];
            s = s + sres[2 * J + 1][2 * I];
            s = s + sres[2 * J + 1][2 * I + 1];
            const long long c = (long long)gJ * C.n[0] + gI;
            C.rhs[c] = s * 0.25;
            C.phi[c] = 0.0;
        }
    }
}
