// Transport stage kernels of a general (logically rectangular) quad mesh:
// perturbed-quadrilateral and stretched meshes, where every cell has its own
// stencil geometry (src/core/mesh.cpp:27-55; src/mlweno/reconstruction.cpp:
// 109-210). Same stage as the uniform kernels (src/couple/evolve.cpp:279-384),
// with
//   * per-cell candidate matrices and cell moments read from HBM
//     (quad_tables.hpp) instead of one table set in the kernel parameters;
//   * every evaluation point mapped from the cell's corners (bilinear map,
//     edge interpolation, normal-line samples with per-edge spacing) into the
//     cell's frame, and the limited polynomial evaluated as a full Q2 form;
//   * physical edge lengths, normals and cell areas of each cell and edge.
// The per-point physics (phase, porosity, velocities, fluxes, rate) is the
// uniform kernels' own device code.
#ifndef MP_QUAD_KERNELS_CUH
#define MP_QUAD_KERNELS_CUH

#include "common.hpp"
#include "phase_math.cuh"
#include "stage_device.cuh"
#include "stage_kernels.cuh"
#include "quad_device.cuh"

namespace mp {
namespace {

// Adiabatic-source inputs and per-cell outputs (null when alpha0 = 0).
struct SourcePtrs {
    const double* cvs_y = nullptr;
    const double* cud_y = nullptr;
    double* srcH = nullptr;
    double* srcR = nullptr;
    double* srcS = nullptr;
};

// Deviation coefficients beyond this: a limiter value could overflow.
constexpr double kQuadGuard = 1e100;

// Everything one stage of one quad mesh reads and writes (the single-mesh
// launch passes it by value; the batched launch reads one per instance).
struct QuadStageArgs {
    int nx = 0, ny = 0, gj0 = 0, gny = 0;   // local rows; local row 0 is global row gj0 of gny
    const double* H = nullptr;              // stage input
    const double* C = nullptr;
    double* rec = nullptr;                  // deviation coefficients (rec_at)
    unsigned char* flags = nullptr;
    double* T = nullptr;
    double* phi = nullptr;
    const double* vsn = nullptr;            // [edge*5 + q], canonical
    const double* udn = nullptr;
    double* face = nullptr;                 // 4 * nedge: fluxH, fluxC, rate, fluxMixture
    unsigned long long* status = nullptr;
    double* theta = nullptr;                // optional limiter factors (2 * ncell)
    QuadDev q{};
    SourcePtrs src{};
};

// ------------------------------------------------------------------ kernels

// Reconstruction (Reconstruction::Update, src/mlweno/reconstruction.cpp:
// 275-355) of H and C with the cell's own tables, each table entry read once
// for both fields: the unlimited deviation polynomials into rec. The limiter runs in the next kernel, so that neither
// kernel holds both the table-driven weights and the point scan in
// registers (the table reads need many warps in flight).
__device__ __forceinline__ void quad_weno_cell(const QuadStageArgs& a, int i, int j) {
    const int nx = a.nx, ny = a.ny, gj0 = a.gj0, gny = a.gny;
    const double* H = a.H;
    const double* C = a.C;
    unsigned long long* status = a.status;
    const QuadDev& q = a.q;
    double* rec = a.rec;
    const long long cell = (long long)j * nx + i;
    const size_t N = (size_t)nx * ny;
    MP_CHECK_INDEX(status, cell, N);
    const int gj = gj0 + j;
    const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = gj == 0 ? 0 : (gj == gny - 1 ? 2 : 1);
    const double eA = 1e-2 * __ldg(q.geo + 3 * N + cell);
    double u[2][3][3];
#pragma unroll
    for (int dj = 0; dj < 3; ++dj)
#pragma unroll
        for (int di = 0; di < 3; ++di) {
            const int ii = min(max(i + di - 1, 0), nx - 1), jj = min(max(j + dj - 1, 0), ny - 1);
            MP_CHECK_INDEX(status, (long long)jj * nx + ii, N);
            u[0][dj][di] = MP_LD(H + (size_t)jj * nx + ii);
            u[1][dj][di] = MP_LD(C + (size_t)jj * nx + ii);
        }
    double D[2][9];
    const int st = reconstruct_quad<2>(q, N, cell, ci, cj, eA, u, D);
    double* r = rec + rec_at(cell);
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        r[m * kRecStride] = D[0][m];
        r[(m + 9) * kRecStride] = D[1][m];
    }
    if (st) record_error(status, PART_UPDATE, cell + (long long)gj0 * nx, st);
}
__global__ void __launch_bounds__(128, 2) quad_weno_kernel(const __grid_constant__ QuadStageArgs a, unsigned c0, unsigned c1,
                                                           const int* gate) {
    if (gated_off(gate)) return;
    const unsigned cell = c0 + blockIdx.x * blockDim.x + threadIdx.x, nx = (unsigned)a.nx;
    if (cell < c1) quad_weno_cell(a, (int)(cell % nx), (int)(cell / nx));
}

// Extremes of both deviation polynomials over the cell's limiter points, in
// physical coordinates and with the finiteness check of every value. Out of
// line: coefficients so large that a value could overflow.
__device__ __noinline__ void quad_scan_exact(const QuadStageArgs& a, long long cell, const double* DH, const double* DC,
                                             double* ext, bool* bad_out) {
    const int nx = a.nx, ny = a.ny;
    const QuadDev& q = a.q;
    const CellFrame f = cell_frame(q, nx, (size_t)nx * ny, cell);
    double hmx = -INFINITY, hmn = INFINITY, cmx = -INFINITY, cmn = INFINITY;
    bool bad = false;
    auto visit = [&](P2 p) {
        const double x = (p.x - f.cx) * f.inv_h, y = (p.y - f.cy) * f.inv_h;
        const double vh = q2v(DH, x, y), vc = q2v(DC, x, y);
        bad = bad || !isfinite(vh) || !isfinite(vc);
        hmx = fmax(hmx, vh); hmn = fmin(hmn, vh);
        cmx = fmax(cmx, vc); cmn = fmin(cmn, vc);
    };
    visit(bilinear(0.0, 0.0, f.c));
    for (int i = 0; i < kNQ; ++i)
        for (int j = 0; j < kNQ; ++j) visit(bilinear(q.gq[i], q.gq[j], f.c));
    for (int e = 0; e < 4; ++e)
        for (int k = 0; k < kNQ; ++k) visit(lerp_edge(q.gq[k], f.c[e], f.c[(e + 1) & 3]));
    visit_samples(q, nx, ny, a.gj0, a.gny, (int)(cell % nx), (int)(cell / nx), f, visit);
    ext[0] = hmx; ext[1] = hmn; ext[2] = cmx; ext[3] = cmn;
    *bad_out = bad;
}

// Extremes of both deviation polynomials over the cell's limiter points
// (state_reconstruction.cpp:152-168): centre, 5x5 Gauss points, 5 points per
// edge, the normal-line samples on this side; mq: the largest H value at the
// centre and the Gauss points. The points are formed in the
// cell's frame from its normalised corners (two FMAs each), so that a point
// costs little beside its two Q2 values (16 FMAs): 2461 FP64 instructions per
// warp and 225 us at 640x1280, against 3135 and 310 us with the points mapped
// in physical coordinates and every value tested. Bound by the FP64 pipe; 3
// resident blocks instead of 4 took 248 us, 5 (96 registers) 231.
__device__ __forceinline__ void quad_scan(const QuadStageArgs& a, int i, int j, const NormalCell& k, double inv_h,
                                          const double (&DH)[9], const double (&DC)[9], Extremes& eh, Extremes& ec,
                                          double& mq) {
    const QuadDev& q = a.q;
    auto visit = [&](double x, double y) {
        const double vh = q2v(DH, x, y), vc = q2v(DC, x, y);
        eh.up(vh); eh.down(vh);
        ec.up(vc); ec.down(vc);
    };
    eh.mx = eh.mn = q2v(DH, k.m.x, k.m.y);
    ec.mx = ec.mn = q2v(DC, k.m.x, k.m.y);
#pragma unroll 1
    for (int b = 0; b < kNQ; ++b) {
        const double s = q.gq[b];
        const double x0 = fma(k.c.x, s, k.m.x), y0 = fma(k.c.y, s, k.m.y);
        const double x1 = fma(k.d.x, s, k.b.x), y1 = fma(k.d.y, s, k.b.y);
#pragma unroll
        for (int r = 0; r < kNQ; ++r) visit(fma(x1, q.gq[r], x0), fma(y1, q.gq[r], y0));
    }
    mq = eh.mx;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        long long id;
        bool wall, rev;
        cell_edge(a.nx, a.ny, i, j, a.gj0, a.gny, e, id, wall, rev);
        const P2 u = k.n[e], v = k.n[(e + 1) & 3];
        const P2 mid = P2{0.5 * (u.x + v.x), 0.5 * (u.y + v.y)}, half = P2{0.5 * (v.x - u.x), 0.5 * (v.y - u.y)};
        P2 n;
        double len;
        edge_geometry(u, v, len, n);
#pragma unroll 1
        for (int g = 0; g < kNQ; ++g) {
            const double x = fma(half.x, q.gq[g], mid.x), y = fma(half.y, q.gq[g], mid.y);
            const double sp = __ldg(q.sp + id * kNQ + (rev ? kNQ - 1 - g : g)) * inv_h;
            const double sx = sp * n.x, sy = sp * n.y;
            visit(x, y);
            if (wall) {
#pragma unroll 1
                for (int m = 1; m <= 4; ++m) visit(fma(-m, sx, x), fma(-m, sy, y));
            } else {
                visit(fma(-1.5, sx, x), fma(-1.5, sy, y));
                visit(fma(-0.5, sx, x), fma(-0.5, sy, y));
            }
        }
    }
}

// Limiter over the cell's own limiter points (state_reconstruction.cpp:
// 136-192): theta of H and C from the unlimited polynomials in rec, which
// are scaled in place.
__device__ __forceinline__ void quad_limit_cell(const QuadStageArgs& a, const Physics& ph, int i, int j) {
    const int nx = a.nx, ny = a.ny, gj0 = a.gj0, gny = a.gny;
    const double* H = a.H;
    const double* C = a.C;
    unsigned long long* status = a.status;
    const QuadDev& q = a.q;
    double* rec = a.rec;
    unsigned char* flags = a.flags;
    double* theta = a.theta;
    const long long cell = (long long)j * nx + i;
    const size_t N = (size_t)nx * ny;
    MP_CHECK_INDEX(status, cell, N);
    const CellFrame f = cell_frame(q, nx, N, cell);
    double DH[9], DC[9];
    load_rec(rec, cell, DH, DC);
    // 3x3 neighbour bounds of the averages (state_reconstruction.cpp:189-196).
    double lo[2], hi[2], m[2];
#pragma unroll
    for (int fi = 0; fi < 2; ++fi) {
        const double* F = fi ? C : H;
        m[fi] = MP_LD(F + cell);
        lo[fi] = m[fi]; hi[fi] = m[fi];
#pragma unroll
        for (int dj = -1; dj <= 1; ++dj)
#pragma unroll
            for (int di = -1; di <= 1; ++di) {
                const int ii = min(max(i + di, 0), nx - 1), jj = min(max(j + dj, 0), ny - 1);
                MP_CHECK_INDEX(status, (long long)jj * nx + ii, N);
                const double v = MP_LD(F + (size_t)jj * nx + ii);
                lo[fi] = fmin(lo[fi], v); hi[fi] = fmax(hi[fi], v);
            }
    }
    const double mH = m[0], mC = m[1];
    const double loH = fmax(0.0, lo[0]), hiH = hi[0], loC = fmax(0.0, lo[1]), hiC = fmin(ph.k.Xe, hi[1]);
    int st_lim = 0;
    if (!(isfinite(mH) && mH >= 0.0 && isfinite(mC) && mC >= 0.0 && mC <= ph.k.Xe)) st_lim = E_OUTOFRANGE;
    Extremes eh, ec;
    double size = 0.0, mq;
#pragma unroll
    for (int k = 0; k < 9; ++k) size += fabs(DH[k]) + fabs(DC[k]);
    if (size < kQuadGuard) {
        quad_scan(a, i, j, normal_cell(f), f.inv_h, DH, DC, eh, ec, mq);
    } else {
        double D0[9], D1[9], ext[4];
        bool bad;
#pragma unroll
        for (int k = 0; k < 9; ++k) { D0[k] = DH[k]; D1[k] = DC[k]; }
        quad_scan_exact(a, cell, D0, D1, ext, &bad);
        eh = Extremes{ext[0], ext[1]};
        mq = ext[0];
        ec = Extremes{ext[2], ext[3]};
        if (bad) st_lim = st_lim ? st_lim : E_FP;
    }
    const double thH = theta_of(mH, loH, hiH, eh.mx, eh.mn);
    const double thC = theta_of(mC, loC, hiC, ec.mx, ec.mn);
    if (theta) { theta[cell] = thH; theta[N + cell] = thC; }
    // The eutectic temperature is monotone over the cell's height range.
    double ylo = f.c[0].y, yhi = f.c[0].y;
#pragma unroll
    for (int k = 1; k < 4; ++k) { ylo = fmin(ylo, f.c[k].y); yhi = fmax(yhi, f.c[k].y); }
    const double t0 = ph.litho ? tep_at(ph, ylo) : ph.Tep, t1 = ph.litho ? tep_at(ph, yhi) : ph.Tep;
    double* r = rec + rec_at(cell);
#pragma unroll
    for (int k = 0; k < 9; ++k) {
        r[k * kRecStride] = DH[k] * thH;
        r[(k + 9) * kRecStride] = DC[k] * thC;
    }
    flags[cell] = st_lim ? (unsigned char)FLAG_CHECK
                         : cell_flags(ph, fmin(t0, t1), fmax(t0, t1), loH, hiH, loC, hiC, fma(thH, mq, mH));
    if (st_lim) record_error(status, PART_LIMIT, cell + (long long)gj0 * nx, st_lim);
}
__global__ void __launch_bounds__(128, 4) quad_limit_kernel(const __grid_constant__ QuadStageArgs a,
                                                            const __grid_constant__ Physics ph, unsigned c0, unsigned c1,
                                                            const int* gate) {
    if (gated_off(gate)) return;
    const unsigned cell = c0 + blockIdx.x * blockDim.x + threadIdx.x, nx = (unsigned)a.nx;
    if (cell < c1) quad_limit_cell(a, ph, (int)(cell % nx), (int)(cell / nx));
}


// 5x5 cell quadrature of T and phi on the bilinear map, wet flag, adiabatic
// source, and the exact check of the diffusion samples when flagged, every
// point with its admissibility test: cells that are not plain. Inlined for
// the same reason as cellphase_general (44 us against 55 at 320x640 where no
// cell is plain).
__device__ __forceinline__ void quad_cellphase_general(const QuadStageArgs& a, const Physics& ph, long long cell) {
    const int nx = a.nx, ny = a.ny, gj0 = a.gj0, gny = a.gny;
    const double* H = a.H;
    const double* C = a.C;
    unsigned long long* status = a.status;
    const QuadDev& q = a.q;
    const double* rec = a.rec;
    unsigned char* flags = a.flags;
    double* T = a.T;
    double* phi = a.phi;
    const SourcePtrs& src = a.src;
    const long long N = (long long)nx * ny;
    MP_CHECK_INDEX(status, cell, N);
    const int i = (int)(cell % nx), j = (int)(cell / nx);
    const CellFrame f = cell_frame(q, nx, (size_t)N, cell);
    const double mH = MP_LD(H + cell), mC = MP_LD(C + cell);
    double DH[9], DC[9];
    load_rec(rec, cell, DH, DC);
    int st_por = 0, st_cell = 0, st_face = 0;
    double Tsum = 0.0, Psum = 0.0, Ssum = 0.0, Rsum = 0.0, Wsum = 0.0;
    bool wet = false;
    for (int b = 0; b < kNQ; ++b)
        for (int a = 0; a < kNQ; ++a) {
            const P2 p = bilinear(q.gq[a], q.gq[b], f.c);
            const double wj = q.gw[a] * q.gw[b] * jacobian(q.gq[a], q.gq[b], f.c);
            const double x = (p.x - f.cx) * f.inv_h, y = (p.y - f.cy) * f.inv_h;
            const double tep = ph.litho ? tep_at(ph, p.y) : ph.Tep;
            PhaseLean pl;
            const int s = phase_stage_lean(ph.sk, mH + q2v(DH, x, y), mC + q2v(DC, x, y), tep, pl);
            if (s) { st_por = st_por ? st_por : s; continue; }
            if (!(pl.T >= 0.0 && pl.phil < 1.0)) st_cell = st_cell ? st_cell : E_OUTOFRANGE;
            const double w = wj / f.area;
            Tsum += w * pl.T;
            Psum += w * pl.phil;
            wet = wet || pl.phil > 0.0;
            if (ph.source) {
                const long long at = cell * (kNQ * kNQ) + b * kNQ + a;
                const double factor = pl.phil == 0.0 ? 0.0 : (ph.theta == 0.0 ? pl.phil : pow(pl.phil, 1.0 + ph.theta));
                const double vy = __ldg(src.cvs_y + at) + factor * __ldg(src.cud_y + at);
                const double s_ = -ph.cooling * pl.T * vy;
                Ssum += w * s_;
                Rsum += w * ph.cooling * fabs(vy);
                Wsum += wj * s_;
            }
        }
    const unsigned char fl = flags[cell];
    if (fl & FLAG_CHECK) {
        visit_samples(q, nx, ny, gj0, gny, i, j, f, [&](P2 p) {
            const double x = (p.x - f.cx) * f.inv_h, y = (p.y - f.cy) * f.inv_h;
            const double tep = ph.litho ? tep_at(ph, p.y) : ph.Tep;
            PhaseLean pl;
            const int s = phase_stage_lean(ph.sk, mH + q2v(DH, x, y), mC + q2v(DC, x, y), tep, pl);
            if (s) { st_face = st_face ? st_face : s; return; }
            if (!(pl.T >= 0.0 && pl.phil < 1.0)) st_face = st_face ? st_face : E_OUTOFRANGE;
        });
    }
    const long long key = cell + (long long)gj0 * nx;
    if (st_por) record_error(status, PART_POROSITY, key, st_por);
    if (st_face) record_error(status, PART_FACES, key, st_face);
    if (st_cell) record_error(status, PART_CELLS, key, st_cell);
    flags[cell] = (unsigned char)((fl & FLAG_CHECK) | (wet ? FLAG_WET : 0));
    T[cell] = Tsum;
    phi[cell] = Psum;
    if (ph.source) { src.srcH[cell] = Ssum; src.srcR[cell] = Rsum; src.srcS[cell] = Wsum; }
}

// The same quadrature of a plain cell (phase_plain): the points in the
// cell's frame, and the Jacobian, which is linear in (r, s), per unit area;
// averages as for cellphase_cell.
// 101 us at 640x1280 (217 with every point tested and mapped in physical
// coordinates); 5 and 6 resident blocks took an eighth and two fifths more.
__device__ __forceinline__ void quad_cellphase_cell(const QuadStageArgs& a, const Physics& ph, long long cell,
                                                    bool averages) {
    const int nx = a.nx;
    const size_t N = (size_t)nx * a.ny;
    MP_CHECK_INDEX(a.status, cell, N);
    const unsigned char fl = a.flags[cell];
    if (__builtin_expect(!(fl & FLAG_PLAIN), 0)) { quad_cellphase_general(a, ph, cell); return; }
    if (!averages && !ph.litho && !ph.source) return;
    const QuadDev& q = a.q;
    const CellFrame f = cell_frame(q, nx, N, cell);
    const NormalCell k = normal_cell(f);
    double DH[9], DC[9];
    load_rec(a.rec, cell, DH, DC);
    DH[0] += MP_LD(a.H + cell);
    DC[0] += MP_LD(a.C + cell);
    double j0, jr, js;
    k.mean_jacobian(j0, jr, js);
    double Tsum = 0.0, Psum = 0.0, Ssum = 0.0, Rsum = 0.0;
#pragma unroll 1
    for (int b = 0; b < kNQ; ++b) {
        const double s = q.gq[b], ws = q.gw[b], js0 = fma(js, s, j0);
        const double x0 = fma(k.c.x, s, k.m.x), y0 = fma(k.c.y, s, k.m.y);
        const double x1 = fma(k.d.x, s, k.b.x), y1 = fma(k.d.y, s, k.b.y);
        double Trow = 0.0, Prow = 0.0;   // by row, as the split form adds them
#pragma unroll
        for (int r = 0; r < kNQ; ++r) {
            const double x = fma(x1, q.gq[r], x0), y = fma(y1, q.gq[r], y0);
            const double w = ws * q.gw[r] * fma(jr, q.gq[r], js0);
            const double tep = ph.litho ? tep_at(ph, fma(y, 1.0 / f.inv_h, f.cy)) : ph.Tep;
            PhaseLean pl;
            phase_plain<false>(ph.sk, q2v(DH, x, y), q2v(DC, x, y), tep, pl);
            Trow = fma(w, pl.T, Trow);
            Prow = fma(w, pl.phil, Prow);
            if (ph.source) {
                const long long at = cell * (kNQ * kNQ) + b * kNQ + r;
                const double factor = pl.phil == 0.0 ? 0.0 : (ph.theta == 0.0 ? pl.phil : pow(pl.phil, 1.0 + ph.theta));
                const double vy = __ldg(a.src.cvs_y + at) + factor * __ldg(a.src.cud_y + at);
                Ssum += w * (-ph.cooling * pl.T * vy);
                Rsum += w * ph.cooling * fabs(vy);
            }
        }
        Tsum += Trow;
        Psum += Prow;
    }
    // Porosities are not negative: the cell is wet where their mean is not 0.
    if (ph.litho) a.flags[cell] = (unsigned char)(fl | (Psum > 0.0 ? FLAG_WET : 0));
    a.T[cell] = Tsum;
    a.phi[cell] = Psum;
    if (ph.source) { a.src.srcH[cell] = Ssum; a.src.srcR[cell] = Rsum; a.src.srcS[cell] = Ssum * f.area; }
}
__global__ void __launch_bounds__(128, 4) quad_cellphase_kernel(const __grid_constant__ QuadStageArgs a, const __grid_constant__ Physics ph,
                                                             long long c0, long long c1, int averages,
                                                             const int* gate) {
    if (gated_off(gate)) return;
    const long long cell = c0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (cell >= c1) return;
    quad_cellphase_cell(a, ph, cell, averages != 0);
}


struct Side {
    double cx, cy, inv_h, mH, mC;
    double DH[9], DC[9];
};
__device__ __forceinline__ void load_side(const QuadDev& q, size_t N, const double* H, const double* C,
                                          const double* rec, long long cell, Side& s) {
    s.cx = __ldg(q.geo + cell);
    s.cy = __ldg(q.geo + N + cell);
    s.inv_h = 1.0 / __ldg(q.geo + 2 * N + cell);
    s.mH = MP_LD(H + cell);
    s.mC = MP_LD(C + cell);
    load_rec(rec, cell, s.DH, s.DC);
}
__device__ __forceinline__ void side_values(const Side& s, P2 p, double& h, double& c) {
    const double x = (p.x - s.cx) * s.inv_h, y = (p.y - s.cy) * s.inv_h;
    h = s.mH + q2v(s.DH, x, y);
    c = s.mC + q2v(s.DC, x, y);
}

// Face fluxes, edge porosity and rate of one edge at its 5 Gauss points,
// every point with its admissibility tests. Out of line: edges with a cell
// that is not plain (inlined, it takes the plain edges' registers: 52 us
// against 45 at 320x640). Both sides' values come first, so that only one
// side's coefficients are held at a time: 78 us at 320x640 where no cell is
// plain, against 110 with both sides' held.
__device__ __noinline__ void quad_face_general(const QuadStageArgs& a, const Physics& ph, long long e) {
    const int nx = a.nx, ny = a.ny, gj0 = a.gj0, gny = a.gny;
    const double* H = a.H;
    const double* C = a.C;
    unsigned long long* status = a.status;
    const QuadDev& q = a.q;
    const double* rec = a.rec;
    const unsigned char* flags = a.flags;
    const double* vsn = a.vsn;
    const double* udn = a.udn;
    double* face = a.face;
    const long long nE = (long long)nx * (ny + 1) + (long long)(nx + 1) * ny;
    const size_t N = (size_t)nx * ny;
    MP_CHECK_INDEX(status, e, nE);
    const QuadEdge g = quad_edge(q, nx, ny, gj0, gny, e);
    MP_CHECK_INDEX(status, g.L, N);
    if (!g.boundary) MP_CHECK_INDEX(status, g.R, N);
    double len;
    P2 nrm;
    edge_geometry(g.a, g.b, len, nrm);
    double hL[kNQ], cL[kNQ], hR[kNQ], cR[kNQ];
    auto values = [&](long long cell, double (&h)[kNQ], double (&c)[kNQ]) {
        Side s;
        load_side(q, N, H, C, rec, cell, s);
#pragma unroll
        for (int k = 0; k < kNQ; ++k) side_values(s, lerp_edge(q.gq[k], g.a, g.b), h[k], c[k]);
    };
    values(g.L, hL, cL);
    if (!g.boundary) values(g.R, hR, cR);
    const bool wetL = (flags[g.L] & FLAG_WET) != 0, wetR = g.boundary ? true : (flags[g.R] & FLAG_WET) != 0;
    const double sgn = g.reverse ? -1.0 : 1.0;
    double fluxH = 0.0, fluxC = 0.0, fluxMix = 0.0, rate = 0.0;
    int st = 0;
#pragma unroll 1
    for (int k = 0; k < kNQ; ++k) {
        const int cq = g.reverse ? kNQ - 1 - k : k;
        const P2 p = lerp_edge(q.gq[k], g.a, g.b);
        const double vs = sgn * __ldg(vsn + e * kNQ + cq);
        const double ud = sgn * __ldg(udn + e * kNQ + cq);
        const double tep = ph.litho ? tep_at(ph, p.y) : ph.Tep;
        PhaseLean A, B;
        int s = phase_stage(ph.sk, hL[k], cL[k], tep, A);
        if (!s && !(A.T >= 0.0 && A.phil < 1.0)) s = E_OUTOFRANGE;
        if (g.boundary) { B = A; hR[k] = hL[k]; cR[k] = cL[k]; }
        else {
            int s2 = phase_stage(ph.sk, hR[k], cR[k], tep, B);
            if (!s2 && !(B.T >= 0.0 && B.phil < 1.0)) s2 = E_OUTOFRANGE;
            s = s ? s : s2;
        }
        if (s) { st = st ? st : s; continue; }
        const PointFlux pf = face_point(ph, A, B, cL[k], cR[k], wetL, wetR, g.boundary, vs, ud, tep, ph.k.LD, st);
        const double w = 0.5 * len * q.gw[k];
        fluxH += w * pf.fh;
        fluxC += w * pf.fc;
        fluxMix += w * pf.vn;
        rate += w * pf.speed;
    }
    if (st) record_error(status, PART_FACES, g.L + (long long)gj0 * nx, st);
    face[e] = fluxH;
    face[nE + e] = fluxC;
    face[2 * nE + e] = rate;
    face[3 * nE + e] = fluxMix;
}

// Limited values of one side at the edge's Gauss points (oriented a -> b).
__device__ __forceinline__ void quad_edge_values(const QuadStageArgs& a, size_t N, long long cell, P2 ea, P2 eb,
                                                 double (&h)[kNQ], double (&c)[kNQ]) {
    const QuadDev& q = a.q;
    const double cx = __ldg(q.geo + cell), cy = __ldg(q.geo + N + cell), inv_h = 1.0 / __ldg(q.geo + 2 * N + cell);
    double DH[9], DC[9];
    load_rec(a.rec, cell, DH, DC);
    DH[0] += MP_LD(a.H + cell);
    DC[0] += MP_LD(a.C + cell);
    const P2 u = normalised(ea, cx, cy, inv_h), v = normalised(eb, cx, cy, inv_h);
    const P2 mid = P2{0.5 * (u.x + v.x), 0.5 * (u.y + v.y)}, half = P2{0.5 * (v.x - u.x), 0.5 * (v.y - u.y)};
#pragma unroll
    for (int k = 0; k < kNQ; ++k) {
        const double x = fma(half.x, q.gq[k], mid.x), y = fma(half.y, q.gq[k], mid.y);
        h[k] = q2v(DH, x, y);
        c[k] = q2v(DC, x, y);
    }
}

// The same edge between plain cells, or (kWall) at the wall of one: both
// sides' values first, so that only one side's coefficients are held at a
// time, then the points without tests or divisions. 152 us at 640x1280 (349
// with both sides' coefficients held and every point tested); 4 and 3
// resident blocks instead of 5 took 3 and 22 % more.
template <bool kWall>
__device__ __forceinline__ void quad_face_plain(const QuadStageArgs& a, const Physics& ph, const QuadEdge& g, bool wet) {
    const QuadDev& q = a.q;
    const size_t N = (size_t)a.nx * a.ny;
    double len;
    P2 nrm;
    edge_geometry(g.a, g.b, len, nrm);
    double hL[kNQ], cL[kNQ], hR[kNQ], cR[kNQ];
    quad_edge_values(a, N, g.L, g.a, g.b, hL, cL);
    if (!kWall) quad_edge_values(a, N, g.R, g.a, g.b, hR, cR);
    const double sgn = kWall && g.reverse ? -1.0 : 1.0;
    double fluxH = 0.0, fluxC = 0.0, fluxMix = 0.0, rate = 0.0;
    int st = 0;
#pragma unroll
    for (int k = 0; k < kNQ; ++k) {
        const int cq = kWall && g.reverse ? kNQ - 1 - k : k;
        const double vs = sgn * __ldg(a.vsn + g.e * kNQ + cq), ud = sgn * __ldg(a.udn + g.e * kNQ + cq);
        const double tep = ph.litho ? tep_at(ph, lerp_edge(q.gq[k], g.a, g.b).y) : ph.Tep;
        PhaseLean A, B;
        PointFlux pf;
        phase_plain<true>(ph.sk, hL[k], cL[k], tep, A);
        if (kWall) {
            pf = wall_point_plain(ph, A, cL[k], wet, vs, ud, tep, st);
        } else {
            phase_plain<true>(ph.sk, hR[k], cR[k], tep, B);
            pf = face_point_plain(ph, A, B, cL[k], cR[k], wet, vs, ud, st);
        }
        const double w = q.gw[k];
        fluxH = fma(w, pf.fh, fluxH);
        fluxC = fma(w, pf.fc, fluxC);
        fluxMix = fma(w, pf.vn, fluxMix);
        rate = fma(w, pf.speed, rate);
    }
    if (st) record_error(a.status, PART_FACES, g.L + (long long)a.gj0 * a.nx, st);
    const long long nE = (long long)a.nx * (a.ny + 1) + (long long)(a.nx + 1) * a.ny;
    const double hl = 0.5 * len;
    a.face[g.e] = hl * fluxH;
    a.face[nE + g.e] = hl * fluxC;
    a.face[2 * nE + g.e] = hl * rate;
    a.face[3 * nE + g.e] = hl * fluxMix;
}
__device__ __noinline__ void quad_face_wall(const QuadStageArgs& a, const Physics& ph, long long e, bool wet) {
    quad_face_plain<true>(a, ph, quad_edge(a.q, a.nx, a.ny, a.gj0, a.gny, e), wet);
}
__device__ __forceinline__ void quad_face_edge(const QuadStageArgs& a, const Physics& ph, const EdgeAt& at) {
    const size_t N = (size_t)a.nx * a.ny;
    const QuadEdge g = quad_edge(a.q, a.nx, a.ny, a.gj0, a.gny, at.horizontal, at.i, at.j);
    MP_CHECK_INDEX(a.status, g.L, N);
    if (!g.boundary) MP_CHECK_INDEX(a.status, g.R, N);
    const unsigned char fl = a.flags[g.L] & (g.boundary ? 0xff : a.flags[g.R]);
    const bool wet = (fl & FLAG_WET) != 0;
    if (!(fl & FLAG_PLAIN)) quad_face_general(a, ph, g.e);
    else if (g.boundary) quad_face_wall(a, ph, g.e, wet);
    else quad_face_plain<false>(a, ph, g, wet);
}
__global__ void __launch_bounds__(128, 5) quad_face_kernel(const __grid_constant__ QuadStageArgs a, const __grid_constant__ Physics ph,
                                                        long long h0, long long nh, long long v0, long long nv,
                                                        const int* gate) {
    if (gated_off(gate)) return;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nh + nv) return;
    // A whole mesh: walls last, in warps of their own (edge_by_kind).
    const bool all = nh == (long long)a.nx * (a.ny + 1) && nv == (long long)(a.nx + 1) * a.ny;
    quad_face_edge(a, ph, all ? edge_by_kind(a.nx, a.ny, k) : edge_by_id(a.nx, a.ny, k < nh ? h0 + k : v0 + (k - nh)));
}


// Diffusive H flux and rate of one edge (diffusiveflux.cpp:105-200 through
// evolve.cpp:330-347): temperatures of the limited states at the normal-line
// samples, spacing per edge point. By Gauss point, so that the lanes of
// small_steps.cu share an edge: quad_diffusion_gradient is the temperature
// gradient at point k (sample spacing sp) of an interior edge or a wall of
// prescribed temperature, quad_diffusion_add the sums over the points in their
// order.
__device__ __forceinline__ double quad_spacing(const QuadDev& q, const QuadEdge& g, int k) {
    return __ldg(q.sp + g.e * kNQ + (g.reverse ? kNQ - 1 - k : k));
}
__device__ __forceinline__ double quad_diffusion_gradient(const QuadDev& q, const Physics& ph, const QuadEdge& g,
                                                          const P2& nrm, const Side& sl, const Side& sr, int k, double sp,
                                                          int& st) {
    const P2 p = lerp_edge(q.gq[k], g.a, g.b);
    const int count = g.boundary ? 5 : 4;
    double v[5];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const bool left = g.boundary || s < 2;
        const double d = (g.boundary ? (double)(s - 4) : (double)s - 1.5) * sp;
        const P2 x = P2{p.x + d * nrm.x, p.y + d * nrm.y};
        double h, c;
        side_values(left ? sl : sr, x, h, c);
        const double tep = ph.litho ? tep_at(ph, x.y) : ph.Tep;
        PhaseLean pl;
        int s1 = phase_stage_lean(ph.sk, h, c, tep, pl);
        if (!s1 && !(pl.T >= 0.0 && pl.phil < 1.0)) s1 = E_OUTOFRANGE;
        if (s1) st = st ? st : s1;
        v[s] = s1 ? 0.0 : pl.T;
    }
    v[4] = g.boundary ? ph.wall_value[g.wall] : 0.0;
    const double* c = g.boundary ? q.dif_c_bnd : q.dif_c_int;
    const double last = v[count - 1];
    double grad = 0.0;
    for (int s = 0; s + 1 < count; ++s) grad += c[s] * (v[s] - last);
    grad /= sp;
    if (!isfinite(grad)) st = st ? st : E_FP;
    return grad;
}
// Adds the diffusive part to the edge's H flux and rate; gradient(k, sp): the
// gradient at point k (called for them in order).
template <class Gradient>
__device__ __forceinline__ void quad_diffusion_add(const QuadStageArgs& a, const Physics& ph, const QuadEdge& g, int type,
                                                   double len, Gradient&& gradient) {
    const QuadDev& q = a.q;
    const long long nE = (long long)a.nx * (a.ny + 1) + (long long)(a.nx + 1) * a.ny;
    const int count = g.boundary ? 5 : 4;
    const double* c = g.boundary ? q.dif_c_bnd : q.dif_c_int;
    double integral = 0.0, rate = a.face[2 * nE + g.e], clast = 0.0;
    for (int s = 0; s + 1 < count; ++s) clast -= c[s];
    for (int k = 0; k < kNQ; ++k) {
        const double w = len * q.gw[k] / 2;
        if (g.boundary && type == 2) { integral += w * ph.wall_value[g.wall]; continue; }
        const double sp = quad_spacing(q, g, k);
        integral = fma(-(w * ph.kappa), gradient(k, sp), integral);
        const double scale = -w * ph.kappa / sp;
        for (int s = 0; s < count; ++s) {
            if (g.boundary && s + 1 == count) continue;
            rate += fabs(scale * (s + 1 == count ? clast : c[s]));
        }
    }
    a.face[g.e] += integral;
    a.face[2 * nE + g.e] = rate;
}
__device__ __forceinline__ void quad_diffusion_edge(const QuadStageArgs& a, const Physics& ph, long long e) {
    const int nx = a.nx, ny = a.ny, gj0 = a.gj0, gny = a.gny;
    const QuadDev& q = a.q;
    const long long nE = (long long)nx * (ny + 1) + (long long)(nx + 1) * ny;
    const size_t N = (size_t)nx * ny;
    MP_CHECK_INDEX(a.status, e, nE);
    const QuadEdge g = quad_edge(q, nx, ny, gj0, gny, e);
    MP_CHECK_INDEX(a.status, g.L, N);
    if (!g.boundary) MP_CHECK_INDEX(a.status, g.R, N);
    const int type = g.boundary ? ph.wall_type[g.wall] : 1;
    if (g.boundary && type == 0) return;
    double len;
    P2 nrm;
    edge_geometry(g.a, g.b, len, nrm);
    Side sl, sr;
    if (type == 1) {
        load_side(q, N, a.H, a.C, a.rec, g.L, sl);
        if (!g.boundary) load_side(q, N, a.H, a.C, a.rec, g.R, sr);
    }
    int st = 0;
    quad_diffusion_add(a, ph, g, type, len,
                       [&](int k, double sp) { return quad_diffusion_gradient(q, ph, g, nrm, sl, sr, k, sp, st); });
    if (st) record_error(a.status, PART_FACES, g.L + (long long)gj0 * nx, st);
}
__global__ void __launch_bounds__(128) quad_diffusion_kernel(const __grid_constant__ QuadStageArgs a, const __grid_constant__ Physics ph,
                                                             long long h0, long long nh, long long v0, long long nv,
                                                             const int* gate) {
    if (gated_off(gate)) return;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nh + nv) return;
    quad_diffusion_edge(a, ph, k < nh ? h0 + k : v0 + (k - nh));
}


// Reconstruction, limiter, cell phase, faces (+ diffusion) of state (H, C)
// on a general quad mesh; the accumulation is the shared sum kernel. Local
// rows [rec0, rec1) are reconstructed, the edges [h0, h0+nh) and [v0, v0+nv)
// (those of the advanced rows) get fluxes; local row 0 is global row gj0 of
// gny (a whole mesh: gj0 = 0, gny = ny). averages: see cellphase_cell. gate: device flag, every kernel
// returns at once while it is 0 (the device-resident step graph).
void launch_quad_stage(const QuadDev& q, int nx, int ny, int gj0, int gny, int rec0, int rec1, long long h0,
                       long long nh, long long v0, long long nv, const Physics& ph, const double* H, const double* C,
                       double* rec, unsigned char* flags, double* T, double* phi, const double* vsn, const double* udn,
                       double* face, unsigned long long* status, double* theta, const SourcePtrs& src,
                       bool averages, cudaStream_t s, const int* gate = nullptr) {
    QuadStageArgs a;
    a.nx = nx; a.ny = ny; a.gj0 = gj0; a.gny = gny;
    a.H = H; a.C = C; a.rec = rec; a.flags = flags; a.T = T; a.phi = phi;
    a.vsn = vsn; a.udn = udn; a.face = face; a.status = status; a.theta = theta;
    a.q = q; a.src = src;
    const unsigned u0 = (unsigned)rec0 * nx, u1 = (unsigned)rec1 * nx, gc = (u1 - u0 + 127) / 128;
    quad_weno_kernel<<<gc, 128, 0, s>>>(a, u0, u1, gate);
    quad_limit_kernel<<<gc, 128, 0, s>>>(a, ph, u0, u1, gate);
    const long long c0 = (long long)rec0 * nx, c1 = (long long)rec1 * nx;
    quad_cellphase_kernel<<<(unsigned)((c1 - c0 + 127) / 128), 128, 0, s>>>(a, ph, c0, c1, averages, gate);
    const unsigned ge = (unsigned)((nh + nv + 127) / 128);
    quad_face_kernel<<<ge, 128, 0, s>>>(a, ph, h0, nh, v0, nv, gate);
    count_launch(4);
    if (ph.diffusion) {
        quad_diffusion_kernel<<<ge, 128, 0, s>>>(a, ph, h0, nh, v0, nv, gate);
        count_launch();
    }
}

}  // namespace
}  // namespace mp

#endif
