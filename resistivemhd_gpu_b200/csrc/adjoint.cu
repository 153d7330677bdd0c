// adjoint.cu -- discrete adjoint of the RK2 step (dt of each step held
// fixed): the reverse of one stage, and the transpose of the periodic
// boundary.
//
// Forward stage (resistiveMHD_2D.cu:133-195), W the stage input:
//   Wc  = W with cell-centred bX, bY            (shiftUToCenterForCT)
//   F,G = HLLD(MUSCL(prim(Wc))) + eta*J terms   (flux_solver.cu, hlld.cu,
//                                                main_plasmoid.cu:175-290)
//   Ez  = (G4 + G4[i+1] - F5 - F5[j+1]) / 4     (stage 1 only, ct.cu:22-41)
//   hydro out = s_in*U0 + s*(W - dt div(F,G))   (s = 1 stage 1, 1/2 stage 2)
//   bX, bY out = CT of the step input's faces with the stage-1 Ez
// Reverse, given Ub = adjoint of the stage output after the boundary
// transpose (so every ghost entry is 0), four launches:
//   adj_prep_kernel   (adjoint_prep.cu) per cell: interface primitives of
//                     both sweeps; reverse of the eta*J terms
//   adj_iface_kernel  per interface (grid.y = sweep): F-bar or G-bar, the
//                     MUSCL states and the HLLD reverse -> adjoints of the
//                     left and right states + the minmod branches
//   adj_gather_kernel per cell: MUSCL and primitive-recovery transposes over
//                     the four interfaces of each sweep that read the cell
//                     -> adjoint of Wc (hydro part written out, centred B
//                     parked for the next kernel)
//   adj_center_kernel per cell: transpose of the face->centre averaging and
//                     of the CT copy of the step input's faces
// Compiled with fused multiply-add: the branch-deciding forward values are
// formed with explicitly rounded operations (adjoint_core.cuh).
#include <cuda_runtime.h>

#include "adjoint.h"
#include "adjoint_common.cuh"
#include "adjoint_core.cuh"
#include "cell_block.cuh"

namespace rmhd2d {

void launch_adjoint_prep(const AdjStageArgs &a, cudaStream_t st);

namespace {

using namespace adjk;
using adj::recon_comp;

using IfaceCells = CellBlock<4>;
using GatherCells = CellBlock<8>;
using CenterCells = CellBlock<8>;

__global__ void __launch_bounds__(IfaceCells::THREADS, 3) adj_iface_kernel(AdjStageArgs a)
{
    const Grid &g = a.g;
    const int dir = blockIdx.y;
    int i, j;
    if (!IfaceCells::cell(g, i, j)) return;
    const long long k = at(g, i, j), P = g.plane;
    double *out = a.IF + (long long)dir * IF_PLANES * P + k;
    if (!iface_live(g, dir, i, j)) {
#pragma unroll
        for (int p = 0; p < IF_PLANES; ++p) out[p * P] = 0.0;
        return;
    }
    // flux adjoint in sweep order
    double nat[8], fb[8];
    if (dir == 0) f_bar(a, i, j, nat); else g_bar(a, i, j, nat);
#pragma unroll
    for (int s = 0; s < 8; ++s) fb[s] = nat[sweep_field(dir, s)];
    // interface primitives of cells m-1 .. m+2 along the sweep
    const double *Q = a.Q + (long long)dir * Q_PLANES * P + k;
    const long long step = dir == 0 ? g.pitch : 1;
    double q[4][8];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int s = 0; s < 8; ++s) q[m][s] = Q[s * P + (m - 1) * step];
    double L[8], R[8], Lb[8], Rb[8];
    const unsigned bits = adj::muscl_states(q[0], q[1], q[2], q[3], g.eps, L, R);
#pragma unroll
    for (int c = 0; c < 8; ++c) { Lb[c] = 0.0; Rb[c] = 0.0; }
    adj::hlld_flux_adj(L, R, g.gamma, g.eps, fb, Lb, Rb);
#pragma unroll
    for (int n = 0; n < 7; ++n) {
        out[n * P] = Lb[recon_comp(n)];
        out[(8 + n) * P] = Rb[recon_comp(n)];
    }
    out[7 * P] = Lb[adj::QBX] + Rb[adj::QBX];
    out[15 * P] = __longlong_as_double((long long)bits);
}

// MUSCL transpose of one sweep at cell c: the adjoint of dQ[c] from
// interfaces m = c+1 (left state, qm), c (left q, right q), c-1 (left qp,
// right qp) and c-2 (right qpp), then the primitive-recovery transpose.
// Every load is issued unconditionally (indices clamped into the grid,
// contributions from outside it masked to 0).
__device__ __forceinline__ void gather_sweep(const AdjStageArgs &a, int dir, int i, int j, double *nat_bar)
{
    const Grid &g = a.g;
    const long long P = g.plane, k = at(g, i, j);
    const int n_along = dir == 0 ? g.nx : g.ny;
    const int c = dir == 0 ? i : j;
    const long long step = dir == 0 ? g.pitch : 1;
    const double *IFd = a.IF + (long long)dir * IF_PLANES * P + k;
    const double mp1 = c + 1 < n_along ? 1.0 : 0.0, mm1 = c >= 1 ? 1.0 : 0.0, mm2 = c >= 2 ? 1.0 : 0.0;
    const double *s1 = IFd + (c + 1 < n_along ? step : 0);
    const double *s0 = IFd;
    const double *sm1 = IFd - (c >= 1 ? step : 0);
    const double *sm2 = IFd - (c >= 2 ? 2 * step : 0);
    const unsigned b1 = (unsigned)__double_as_longlong(s1[15 * P]);
    const unsigned b0 = (unsigned)__double_as_longlong(s0[15 * P]);
    const unsigned bm1 = (unsigned)__double_as_longlong(sm1[15 * P]);
    const unsigned bm2 = (unsigned)__double_as_longlong(sm2[15 * P]);
    double qb[8];
#pragma unroll
    for (int n = 0; n < 7; ++n) {
        const double L1 = s1[n * P], L0 = s0[n * P], R0 = s0[(8 + n) * P];
        const double Lm1 = sm1[n * P], Rm1 = sm1[(8 + n) * P], Rm2 = sm2[(8 + n) * P];
        auto sel = [n](unsigned bits, int right) -> unsigned { return (bits >> (2 * n + (right ? 14 : 0))) & 3u; };
        const unsigned l1 = sel(b1, 0), l0 = sel(b0, 0), r0 = sel(b0, 1), lm1 = sel(bm1, 0), rm1 = sel(bm1, 1),
                       rm2 = sel(bm2, 1);
        double v = mp1 * (l1 == 1 ? -0.5 * L1 : 0.0);
        v += L0 * (l0 == 1 ? 1.5 : (l0 == 2 ? 0.5 : 1.0)) + (r0 == 1 ? 0.5 * R0 : 0.0);
        v += mm1 * ((lm1 == 2 ? 0.5 * Lm1 : 0.0) + Rm1 * (rm1 == 1 ? 0.5 : (rm1 == 2 ? 1.5 : 1.0)));
        v += mm2 * (rm2 == 2 ? -0.5 * Rm2 : 0.0);
        qb[recon_comp(n)] = v;
    }
    qb[adj::QBX] = s0[7 * P];
    const double *Q = a.Q + (long long)dir * Q_PLANES * P + k;
    double q[8], cb[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) { q[s] = Q[s * P]; cb[s] = 0.0; }
    adj::basic_param_adj(q, Q[8 * P], g.gamma, qb, cb);
    // b_n of dQ[c - 1] is the average of cells c-1 and c
    cb[4] += mm1 * 0.5 * sm1[7 * P];
#pragma unroll
    for (int s = 0; s < 8; ++s) nat_bar[sweep_field(dir, s)] += cb[s];
}

// Bound by the latency of its 120 loads per cell: at 128 registers (two blocks
// per SM) more of them are in flight than at 80 (three): 130 x 96 x 36 steps and
// their reverse 4.77 -> 4.57 ms, 150 x 90 4.96 -> 4.82, 512 x 512 22.7 -> 22.5.
__global__ void __launch_bounds__(GatherCells::THREADS, 2) adj_gather_kernel(AdjStageArgs a)
{
    const Grid &g = a.g;
    int i, j;
    if (!GatherCells::cell(g, i, j)) return;
    const long long k = at(g, i, j), P = g.plane;
    double wb[8];
#pragma unroll
    for (int f = 0; f < 8; ++f) wb[f] = 0.0;
    if (i >= 1 && i <= g.nx - 2 && j >= 1 && j <= g.ny - 2) {
        gather_sweep(a, 0, i, j, wb);
        gather_sweep(a, 1, i, j, wb);
        // eta*J: direct B terms, and J of the neighbours (centred differences)
        const double *RJ = a.RJ;
        auto rj = [&](int p, int ii, int jj) -> double {
            if (ii < 0 || jj < 0 || ii >= g.nx || jj >= g.ny) return 0.0;
            return RJ[p * P + at(g, ii, jj)];
        };
        wb[BXF] += RJ[3 * P + k] + (rj(2, i, j + 1) - rj(2, i, j - 1)) / (2.0 * g.dy);
        wb[BYF] += RJ[4 * P + k] + (rj(2, i - 1, j) - rj(2, i + 1, j)) / (2.0 * g.dx);
        wb[BZF] += RJ[5 * P + k] + (rj(1, i + 1, j) - rj(1, i - 1, j)) / (2.0 * g.dx)
                 + (rj(0, i, j - 1) - rj(0, i, j + 1)) / (2.0 * g.dy);
    }
#pragma unroll
    for (int f = 0; f < 8; ++f) {
        if (!hydro_field(f)) continue;
        const long long kf = f * P + k;
        if (a.stage == 2) {
            a.Ustage[kf] = 0.5 * a.Ub[kf] + wb[f];   // adjoint of the stage-1 state
            a.Uin[kf] = 0.5 * a.Ub[kf];              // adjoint of the step input (U^n term)
        } else {
            a.Uin[kf] += a.Ub[kf] + wb[f];
        }
    }
    a.tmp[k] = wb[BXF];
    a.tmp[P + k] = wb[BYF];
}

__global__ void __launch_bounds__(256) adj_center_kernel(AdjStageArgs a)
{
    const Grid &g = a.g;
    int i, j;
    if (!CenterCells::cell(g, i, j)) return;
    const long long k = at(g, i, j), P = g.plane;
    const double *tx = a.tmp, *ty = a.tmp + P;
    const double cbx = (i >= 1 ? 0.5 : 1.0) * tx[k] + (i + 1 < g.nx ? 0.5 * tx[at(g, i + 1, j)] : 0.0);
    const double cby = (j >= 1 ? 0.5 : 1.0) * ty[k] + (j + 1 < g.ny ? 0.5 * ty[at(g, i, j + 1)] : 0.0);
    const long long kx = BXF * P + k, ky = BYF * P + k;
    if (a.stage == 2) {
        a.Ustage[kx] = cbx;
        a.Ustage[ky] = cby;
        a.Uin[kx] = a.Ub[kx];      // CT copies the step input's faces
        a.Uin[ky] = a.Ub[ky];
    } else {
        a.Uin[kx] += a.Ub[kx] + cbx;
        a.Uin[ky] += a.Ub[ky] + cby;
    }
}

// Transpose of the periodic boundary (periodicBoundaryX2nd then
// periodicBoundaryY2nd, boundary.cu:4-141).  After both passes every ghost
// cell holds the interior cell (wrap(i), wrap(j)), so its adjoint moves onto
// that cell and the ghost's becomes 0.  One thread per interior cell of the
// 3-wide bands along the walls and per field gathers its images -- the
// y-wall image Jg, the x-wall image Ig and the corner (Ig, Jg) -- and zeroes
// them, summing in the order the two passes' transposes (y first, then x)
// would: (U(I,J) + U(I,Jg)) + (U(Ig,J) + U(Ig,Jg)).  Each ghost has one
// image, so no two threads touch the same entry.
__global__ void periodic_transpose_kernel(Grid g, double *Ub)
{
    const unsigned nrow = 6u * (unsigned)(g.nx - 6);    // rows 3..5 and ny-6..ny-4, interior columns
    const unsigned ncol = 6u * (unsigned)(g.ny - 12);   // columns 3..5 and nx-6..nx-4, rows 6..ny-7
    unsigned u = blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= nrow + ncol) return;
    const int f = (int)blockIdx.y;
    int I, J;
    if (u < nrow) {
        const unsigned r = u / (unsigned)(g.nx - 6);
        I = 3 + (int)(u - r * (unsigned)(g.nx - 6));
        J = (int)r + (r < 3 ? 3 : g.ny - 9);
    } else {
        u -= nrow;
        const unsigned c = u / (unsigned)(g.ny - 12);
        J = 6 + (int)(u - c * (unsigned)(g.ny - 12));
        I = (int)c + (c < 3 ? 3 : g.nx - 9);
    }
    const int Ig = I < 6 ? I + g.nx - 6 : (I >= g.nx - 6 ? I - (g.nx - 6) : -1);
    const int Jg = J < 6 ? J + g.ny - 6 : (J >= g.ny - 6 ? J - (g.ny - 6) : -1);
    double *p = Ub + (long long)f * g.plane;
    double v = p[at(g, I, J)];
    if (Jg >= 0) {
        v = v + p[at(g, I, Jg)];
        p[at(g, I, Jg)] = 0.0;
    }
    if (Ig >= 0) {
        double w = p[at(g, Ig, J)];
        if (Jg >= 0) {
            w = w + p[at(g, Ig, Jg)];
            p[at(g, Ig, Jg)] = 0.0;
        }
        p[at(g, Ig, J)] = 0.0;
        v = v + w;
    }
    p[at(g, I, J)] = v;
}

// Transpose of the symmetric walls and of mixed periodic / symmetric walls.
// The forward (TS boundary.cu:4-205, as the oracle's tangent restates it)
// runs the x pass over every row, then the y pass over every column.  Each
// pass copies every field but the wall-normal B from the mirror cells
// (ghost 2 <- 3, 1 <- 4, 0 <- 5 and their upper twins) and integrates the
// normal B into the wall from its neighbours' tangential B, e.g. at the
// lower y wall, for column i > 0,
//   bY(i,2) = bY(i,3) + (bX(i,3) - bX(i-1,3)) dy/dx
//   bY(i,1) = bY(i,2) + (bX(i,2) - bX(i-1,2)) dy/dx      (bX(.,2) a copy of row 3)
//   bY(i,0) = bY(i,1) + (bX(i,1) - bX(i-1,1)) dy/dx      (bX(.,1) a copy of row 4)
// The transposes run in the opposite order, y then x, in gather form: a
// thread owns one field of one column (y) or one row (x), takes the chain
// adjoints of its own and of the next column or row, writes only its own
// entries, and clears the ghost entries that only it reads.  Those that a
// neighbour's chain reads too -- BYF in the y pass, BXF in the x pass -- are
// cleared by the launch after it.  Every value is loaded before the first
// store: with one thread per line and all fields' read-modify-writes in a
// row, each waited for the one before it (150 x 90: 27 + 18 us per transpose,
// now 4.5 + 3.3 and 2.3 for the last clear).  The x pass at row 3 reads the lower wall face bY(c,2)
// before the y pass replaces it -- in the step, the stage-1 CT result (row2)
// -- so the x transpose leaves that adjoint in the ghost entry (c,2) of the
// interior columns, where the stage-1 reverse takes it as the CT'd face's.

// Running sums of a lower and an upper chain's output adjoints: t1 = the
// sum of all three, t2 = the outer two, t3 = the outermost.
struct ChainAdj {
    double t1, t2, t3;
};

__device__ __forceinline__ ChainAdj chain_adj(double inner, double middle, double outer)
{
    return ChainAdj{inner + middle + outer, middle + outer, outer};
}

// The twelve entries of one field along a line of n cells that a wall's
// transpose touches: ghosts 0..2 and n-3..n-1 (g), interior 3..5 and n-6..n-4
// (v), `st` doubles apart from p on.
struct WallLine {
    double g[6], v[6];
    __device__ __forceinline__ WallLine(const double *p, int n, long long st)
    {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            g[q] = p[q * st];
            v[q] = p[(3 + q) * st];
            v[3 + q] = p[(n - 6 + q) * st];
            g[3 + q] = p[(n - 3 + q) * st];
        }
    }
    // Adds what the ghosts were copied from: periodic (ghost q <- n-6+q,
    // n-3+q <- 3+q) or mirror (2 <- 3, 1 <- 4, 0 <- 5 and their twins).
    __device__ __forceinline__ void add_copies(bool periodic)
    {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            v[3 + q] += periodic ? g[q] : g[5 - q];
            v[q] += periodic ? g[3 + q] : g[2 - q];
        }
    }
    __device__ __forceinline__ void store(double *p, int n, long long st, bool clear_ghosts) const
    {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            p[(3 + q) * st] = v[q];
            p[(n - 6 + q) * st] = v[3 + q];
            if (clear_ghosts) {
                p[q * st] = 0.0;
                p[(n - 3 + q) * st] = 0.0;
            }
        }
    }
};

// One thread per column and field (blockIdx.y).
template <int BY> __global__ void ytrans_kernel(Grid g, double *Ub)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, f = (int)blockIdx.y;
    if (i >= g.nx) return;
    const long long P = g.plane;
    const int ny = g.ny;
    double *p = Ub + f * P + at(g, i, 0);
    WallLine w(p, ny, 1);
    if (BY == BC_PERIODIC || (f != BXF && f != BYF)) {
        w.add_copies(BY == BC_PERIODIC);
        w.store(p, ny, 1, true);
        return;
    }
    auto B = [&](int col, int j) -> double { return Ub[BYF * P + at(g, col, j)]; };
    auto lower = [&](int col) { return chain_adj(B(col, 2), B(col, 1), B(col, 0)); };
    auto upper = [&](int col) { return chain_adj(B(col, ny - 3), B(col, ny - 2), B(col, ny - 1)); };
    const ChainAdj lo = lower(i), up = upper(i);
    if (f == BYF) {
        w.v[0] += lo.t1;
        w.v[5] += up.t1;
        w.store(p, ny, 1, false);
        return;
    }
    // chain terms on bX: this column's (i > 0) and the next column's
    const double c = g.dy / g.dx;
    const ChainAdj z{0.0, 0.0, 0.0};
    const ChainAdj lo_own = i > 0 ? lo : z, up_own = i > 0 ? up : z;
    const ChainAdj lo_nxt = i + 1 < g.nx ? lower(i + 1) : z, up_nxt = i + 1 < g.nx ? upper(i + 1) : z;
    w.v[0] += w.g[2] + c * (lo_own.t1 - lo_nxt.t1) + c * (lo_own.t2 - lo_nxt.t2);
    w.v[1] += w.g[1] + c * (lo_own.t3 - lo_nxt.t3);
    w.v[2] += w.g[0];
    w.v[5] += w.g[3] - c * (up_own.t1 - up_nxt.t1);
    w.v[4] += w.g[4] - c * (up_own.t2 - up_nxt.t2);
    w.v[3] += w.g[5] - c * (up_own.t3 - up_nxt.t3);
    w.store(p, ny, 1, true);
}

// One thread per row 2 .. ny-4 and field (blockIdx.y); row 2 only gathers the
// lower wall face's adjoint from row 3's chains.  blockIdx.y = NFIELD: with
// mirror y walls, clears what the y pass left of the ghost rows' BYF (except
// row 2's gathered entries).
template <int BX> __global__ void xtrans_kernel(Grid g, double *Ub, int clear_rows)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x, f = (int)blockIdx.y;
    const long long P = g.plane;
    const int nx = g.nx;
    if (f == NFIELD) {
        if (!clear_rows || t >= nx) return;
        double *p = Ub + BYF * P + at(g, t, 0);
        const bool gathered = BX != BC_PERIODIC && (t == 3 || t == 4 || (t >= nx - 6 && t <= nx - 4));
        p[0] = p[1] = p[g.ny - 3] = p[g.ny - 2] = p[g.ny - 1] = 0.0;
        if (!gathered) p[2] = 0.0;
        return;
    }
    const int j = 2 + t;
    if (j > g.ny - 4) return;
    double *p = Ub + f * P + at(g, 0, j);
    const long long st = g.pitch;
    if (BX == BC_PERIODIC) {
        if (j < 3) return;
        WallLine w(p, nx, st);
        w.add_copies(true);
        w.store(p, nx, st, true);
        return;
    }
    if (j < 3 && f != BYF) return;
    auto B = [&](int i, int row) -> double { return Ub[BXF * P + at(g, i, row)]; };
    auto lower = [&](int row) { return chain_adj(B(2, row), B(1, row), B(0, row)); };
    auto upper = [&](int row) { return chain_adj(B(nx - 3, row), B(nx - 2, row), B(nx - 1, row)); };
    WallLine w(p, nx, st);
    if (f == BXF) {
        w.v[0] += chain_adj(w.g[2], w.g[1], w.g[0]).t1;
        w.v[5] += chain_adj(w.g[3], w.g[4], w.g[5]).t1;
        w.store(p, nx, st, false);
        return;
    }
    if (f == BYF) {
        const double c = g.dx / g.dy;
        const ChainAdj z{0.0, 0.0, 0.0};
        const ChainAdj lo = j >= 3 ? lower(j) : z, up = j >= 3 ? upper(j) : z;
        const ChainAdj lo_nxt = lower(j + 1), up_nxt = upper(j + 1);
        if (j < 3) {
            // the ghost row's own entries are cleared, not read
#pragma unroll
            for (int q = 0; q < 6; ++q) w.v[q] = 0.0;
        }
        // the chains' bY terms at this row: + from its own chain, - from the next
        // row's (its j-1), through the copies 2 <- 3 and 1 <- 4
        w.v[0] += c * (lo.t1 - lo_nxt.t1) + c * (lo.t2 - lo_nxt.t2);
        w.v[1] += c * (lo.t3 - lo_nxt.t3);
        w.v[5] -= c * (up.t1 - up_nxt.t1);
        w.v[4] -= c * (up.t2 - up_nxt.t2);
        w.v[3] -= c * (up.t3 - up_nxt.t3);
        if (j < 3) {
            p[3 * st] = w.v[0];
            p[4 * st] = w.v[1];
            p[(nx - 4) * st] = w.v[5];
            p[(nx - 5) * st] = w.v[4];
            p[(nx - 6) * st] = w.v[3];
            return;
        }
    }
    w.add_copies(false);
    w.store(p, nx, st, true);
}

// Clears BXF's ghost columns in the interior rows (blockIdx.y: column).
__global__ void clear_bx_columns_kernel(Grid g, double *Ub)
{
    const int j = 3 + blockIdx.x * blockDim.x + threadIdx.x, q = (int)blockIdx.y;
    if (j > g.ny - 4) return;
    Ub[BXF * g.plane + at(g, q < 3 ? q : g.nx - 6 + q, j)] = 0.0;
}

// Pitched plane -> dense (nx, ny) table.
__global__ void plane_to_table_kernel(Grid g, const double *plane, double *tab)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (long long)g.nx * g.ny) return;
    const int i = (int)(t / g.ny), j = (int)(t - (long long)i * g.ny);
    tab[t] = plane[at(g, i, j)];
}

int blocks_for(long long n, int threads) { return (int)((n + threads - 1) / threads); }

}  // namespace

void launch_adjoint_stage(const AdjStageArgs &a, cudaStream_t st)
{
    launch_adjoint_prep(a, st);
    adj_iface_kernel<<<dim3(IfaceCells::blocks(a.g), 2), IfaceCells::THREADS, 0, st>>>(a);
    adj_gather_kernel<<<GatherCells::blocks(a.g), GatherCells::THREADS, 0, st>>>(a);
    adj_center_kernel<<<CenterCells::blocks(a.g), CenterCells::THREADS, 0, st>>>(a);
}

void launch_boundary_transpose(const Grid &g, double *Ub, cudaStream_t st)
{
    if (g.bc_x == BC_PERIODIC && g.bc_y == BC_PERIODIC) {
        const long long n = 6LL * (g.nx - 6) + 6LL * (g.ny - 12);
        periodic_transpose_kernel<<<dim3(blocks_for(n, 128), NFIELD), 128, 0, st>>>(g, Ub);
        return;
    }
    const dim3 ycols(blocks_for(g.nx, 64), NFIELD);
    const int along = g.nx > g.ny - 5 ? g.nx : g.ny - 5;
    const dim3 xrows(blocks_for(along, 64), NFIELD + 1);
    const int mirror_y = g.bc_y != BC_PERIODIC;
    if (mirror_y)
        ytrans_kernel<BC_SYMMETRIC><<<ycols, 64, 0, st>>>(g, Ub);
    else
        ytrans_kernel<BC_PERIODIC><<<ycols, 64, 0, st>>>(g, Ub);
    if (g.bc_x == BC_PERIODIC) {
        xtrans_kernel<BC_PERIODIC><<<xrows, 64, 0, st>>>(g, Ub, mirror_y);
    } else {
        xtrans_kernel<BC_SYMMETRIC><<<xrows, 64, 0, st>>>(g, Ub, mirror_y);
        clear_bx_columns_kernel<<<dim3(blocks_for(g.ny - 6, 128), 6), 128, 0, st>>>(g, Ub);
    }
}

void launch_plane_to_table(const Grid &g, const double *plane, double *tab, cudaStream_t st)
{
    plane_to_table_kernel<<<blocks_for((long long)g.nx * g.ny, 256), 256, 0, st>>>(g, plane, tab);
}

}  // namespace rmhd2d
