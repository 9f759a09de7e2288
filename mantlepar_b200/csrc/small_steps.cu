// Device-resident steps of a small mesh: every phase of every stage of up to
// 64 steps in ONE kernel of one thread-block cluster.
//
// A mesh of a few hundred to a few thousand cells is one wave of threads per
// phase: as a graph of kernels a step is 24 nodes, each of which takes its
// launch, its own cold start and the tail of its slowest thread, and most of
// the GPU idles. Here the blocks of one cluster (16 where the GPU offers that
// size, else 8) share the phases and meet at the cluster's hardware barrier,
// which the co-scheduling of a cluster guarantees to end; the step rule runs
// on one thread of the first block between phases (step_ctl.cuh, the same
// functions as the graph's controller kernels) and the others read its
// decisions from that block's shared memory. Every element runs the device
// functions of the stage kernels and every reduction their order, so results
// equal the graph's and the host loop's bit for bit. All loops are bounded:
// the requested steps, at most 41 attempts, a fixed sequence of phases.
//
// The arrays that a phase writes and a later one reads are loaded through the
// coherent path (MP_LD): the read-only path may keep a stale line.
#define MP_LD(p) (*(p))

#include "small_steps.hpp"

#include "common.hpp"
#include "quad_kernels.cuh"
#include "stage_kernels.cuh"
#include "step_ctl.cuh"

#include <cooperative_groups.h>

namespace mp {
namespace {

namespace cg = cooperative_groups;

enum : int { KIND_P = 0, KIND_B = 1, KIND_C = 2, NKIND = 3 };   // L(U^n), second and third stage

struct SmallArgs {
    StageHot tab;
    Physics ph;
    StepOpts opts;
    int nx, ny;
    ReconArgs recon[NKIND];
    CellPhaseArgs phase[NKIND];
    FaceArgs face[NKIND];
    QuadStageArgs quad[NKIND];
    SumArgs sum[NKIND];
    const double *H0, *C0, *LH, *LC;    // stage 1: U1 = U^n + dt L(U^n)
    double *H1, *C1;
    const double *newH, *newC;          // the accepted state, copied to H, C
    double *H, *C;
    const double* cell_area;
    Partial* partial;
    unsigned long long* status;
    InstCtl* ctl;
    CtlHeader* hdr;
    mp_step_report* reports;
};

// The first block's record, read by the whole cluster.
struct Board {
    InstCtl c;
    Totals tot;
    double dt;
    int go;                             // attempt / stage / commit goes ahead
};

constexpr int kSmallThreads = 512;

// Largest meshes (small_steps_blocks); kSmallCells is in stage_kernels.cuh.
constexpr long long kSmallCellsMore = 1024, kSmallQuadCells = 1024, kSmallQuadDiffusion = 640;

// A mesh this small leaves a cell's chain of dependent FP64 instructions as
// the length of a phase, so a group of eight lanes shares each element:
// reconstruction and limiter by field and quarter of the limiter's lines or
// points, the cell quadrature by row, a face by Gauss point. Extremes combine
// in any order and sums are added by one lane in the kernels' order, so the
// values are those of one thread per element. Cells and edges that are not
// plain, and the diffusion of a uniform mesh, take the kernels' own forms
// (each_of_warp).
constexpr int kGroup = 8;
constexpr unsigned kAll = 0xffffffffu;

__device__ __forceinline__ double group_get(double v, int lane) { return __shfl_sync(kAll, v, lane, kGroup); }

// Sum over the first kNQ lanes in lane order (valid in every lane).
__device__ __forceinline__ double rows_sum(double v) {
    double s = group_get(v, 0);
#pragma unroll
    for (int l = 1; l < kNQ; ++l) s += group_get(v, l);
    return s;
}
// sum_l w_l v_l as one FMA chain over the first kNQ lanes.
__device__ __forceinline__ double points_sum(const double (&w)[kNQ], double v) {
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < kNQ; ++l) s = fma(w[l], group_get(v, l), s);
    return s;
}

// Limiter factors, records and flag byte of the group's cell from each field's
// extremes (lanes 0-3 field H, 4-7 field C, quarter `part` of its scan; mq:
// the largest value of its share of the cell quadrature points). True in the
// group's first lane when the cell is not plain.
template <class TepRange>
__device__ __forceinline__ bool small_limit(const Physics& ph, bool active, int part, int f, long long cell, double mean,
                                            double lo, double hi, Extremes x, double mq, int st, bool bad,
                                            const double (&D)[9], double* rec, unsigned char* flags, unsigned long long* status,
                                            TepRange&& tep_range) {
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
        x.up(__shfl_xor_sync(kAll, x.mx, o));
        x.down(__shfl_xor_sync(kAll, x.mn, o));
        const double y = __shfl_xor_sync(kAll, mq, o);
        mq = y > mq ? y : mq;
    }
    const double th = theta_of(mean, lo, hi, x.mx, x.mn);
    const bool mean_ok = isfinite(mean) && mean >= 0.0 && (f == 0 || mean <= ph.k.Xe);
    const double loC = group_get(lo, 4), hiC = group_get(hi, 4);
    const int stH = __shfl_sync(kAll, st, 0, kGroup), stC = __shfl_sync(kAll, st, 4, kGroup);
    const int okH = __shfl_sync(kAll, (int)mean_ok, 0, kGroup), okC = __shfl_sync(kAll, (int)mean_ok, 4, kGroup);
    const int badH = __shfl_sync(kAll, (int)bad, 0, kGroup), badC = __shfl_sync(kAll, (int)bad, 4, kGroup);
    if (!active) return false;
    double* r = rec + rec_at(cell) + f * 9 * kRecStride;
#pragma unroll
    for (int m = 0; m < 9; ++m)
        if ((m & 3) == part) r[m * kRecStride] = D[m] * th;
    if (part != 0 || f != 0) return false;
    const int st_all = stH ? stH : stC;
    const int st_lim = !(okH && okC) ? (int)E_OUTOFRANGE : (badH || badC ? (int)E_FP : 0);
    double t0, t1;
    tep_range(t0, t1);
    const unsigned char fl = st_all || st_lim ? (unsigned char)FLAG_CHECK
                                              : cell_flags(ph, fmin(t0, t1), fmax(t0, t1), lo, hi, loC, hiC, fma(th, mq, mean));
    flags[cell] = fl;
    if (st_all) record_error(status, PART_UPDATE, cell, st_all);
    if (st_lim) record_error(status, PART_LIMIT, cell, st_lim);
    return !(fl & FLAG_PLAIN);
}

// What takes a whole element in one lane runs after the warp's rounds of four
// elements, each element in a lane of its own, and out of line. Done in every
// round by the first lane of each group, four steps of a 32x48 mesh of pure
// component took 980 us, with diffusion 1597; so 618 and 857 (the graph 537
// and 677).
template <class F>
__device__ __forceinline__ void each_of_warp(int group, int groups, int count, F&& f) {
    const int lane = threadIdx.x & 31, base = group - (lane >> 3);
    __syncwarp();
    for (int k = lane;; k += 32) {
        const int at = base + (k >> 2) * groups + (k & 3);
        if (at >= count) break;
        f(at);
    }
}
template <bool kQuad, bool kLitho>
__device__ __noinline__ void small_cells_rest(const SmallArgs& m, int kind, int group, int groups) {
    const CellPhaseArgs& a = m.phase[kind];
    each_of_warp(group, groups, m.nx * m.ny, [&](int cell) {
        if (a.flags[cell] & FLAG_PLAIN) return;
        if (kQuad) quad_cellphase_general(m.quad[kind], m.ph, cell);
        else cellphase_general<kLitho>(m.tab, a, m.ph, cell);
    });
}
template <bool kQuad, bool kLitho>
__device__ __noinline__ void small_edges_rest(const SmallArgs& m, int kind, int group, int groups) {
    const int nx = m.nx, ny = m.ny;
    const FaceArgs& a = m.face[kind];
    each_of_warp(group, groups, nx * (ny + 1) + (nx + 1) * ny, [&](int k) {
        const EdgeAt at = edge_by_kind(nx, ny, k);
        const EdgeCells g = edge_cells(a, at);
        MP_CHECK_INDEX(a.status, g.L, nx * ny);
        if (!g.boundary) MP_CHECK_INDEX(a.status, g.R, nx * ny);
        if (!(a.flags[g.L] & (g.boundary ? 0xff : a.flags[g.R]) & FLAG_PLAIN)) {
            if (kQuad) quad_face_general(m.quad[kind], m.ph, g.e);
            else face_general<kLitho>(m.tab, a, m.ph, g.e);
        }
        if (!kQuad && m.ph.diffusion) diffusion_edge<kLitho>(m.tab, a, m.ph, at);
    });
}

// Diffusion on a general quad mesh: lane p < 5 takes the p-th Gauss point's
// gradient, the first lane adds them up (four steps of a 20x24 mesh 807 us;
// with an edge per lane 1111, the graph 1240).
__device__ __noinline__ void small_quad_diffusion(const SmallArgs& m, int kind, int group, int groups) {
    const QuadStageArgs& a = m.quad[kind];
    const Physics& ph = m.ph;
    const int nx = m.nx, ny = m.ny, edges = nx * (ny + 1) + (nx + 1) * ny;
    const int l = threadIdx.x & 7, p = min(l, kNQ - 1);
    const size_t N = (size_t)nx * ny;
    __syncwarp();
    for (int base = group - ((threadIdx.x & 31) >> 3); base < edges; base += groups) {
        const int k0 = base + (int)((threadIdx.x & 31) >> 3);
        bool active = k0 < edges;
        const EdgeAt at = edge_by_kind(nx, ny, active ? k0 : edges - 1);
        QuadEdge g = quad_edge(a.q, nx, ny, 0, ny, at.horizontal, at.i, at.j);
        g.e = checked_index(a.status, g.e, edges, active);
        g.L = checked_index(a.status, g.L, N, active);
        if (!g.boundary) g.R = checked_index(a.status, g.R, N, active);
        const int type = g.boundary ? ph.wall_type[g.wall] : 1;
        double len, grad = 0.0, all[kNQ];
        P2 nrm;
        edge_geometry(g.a, g.b, len, nrm);
        int st = 0;
        if (type == 1) {
            Side sl, sr;
            load_side(a.q, N, a.H, a.C, a.rec, g.L, sl);
            if (!g.boundary) load_side(a.q, N, a.H, a.C, a.rec, g.R, sr);
            grad = quad_diffusion_gradient(a.q, ph, g, nrm, sl, sr, p, quad_spacing(a.q, g, p), st);
        }
        int first = 0;                      // failure of the first point that has one
#pragma unroll
        for (int n = 0; n < kNQ; ++n) {
            all[n] = group_get(grad, n);
            const int s = __shfl_sync(kAll, st, n, kGroup);
            first = first ? first : s;
        }
        if (!active || l != 0 || type == 0) continue;
        quad_diffusion_add(a, ph, g, type, len, [&](int k, double) { return all[k]; });
        if (first) record_error(a.status, PART_FACES, g.L, first);
    }
}

// Reconstruction and limiter of a uniform mesh, and the whole cell phase of
// the cells that are not plain. Each lane of a field scans
// two of the symmetric line pairs of scan_cell and one of the lines that
// depend on the walls (the centre row as a pair at 0).
template <bool kLitho>
__device__ __noinline__ void small_recon(const SmallArgs& m, int kind, int group, int groups) {
    const StageHot& t = m.tab;
    const ReconArgs& a = m.recon[kind];
    const int nx = m.nx, ny = m.ny, N = nx * ny;
    const int l = threadIdx.x & 7, f = l >> 2, part = l & 3;
    bool rest = false;
    for (int base = group - ((threadIdx.x & 31) >> 3); base < N; base += groups) {
        const int c0 = base + (int)((threadIdx.x & 31) >> 3);
        bool active = c0 < N;
        // Idle groups repeat the last cell and write nothing.
        const int cell = checked_index(a.status, active ? c0 : N - 1, N, active);
        const int i = cell % nx, j = cell / nx;
        const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = j == 0 ? 0 : (j == ny - 1 ? 2 : 1);
        const double* F = f ? a.C : a.H;
        double u[3][3];
#pragma unroll
        for (int dj = 0; dj < 3; ++dj)
#pragma unroll
            for (int di = 0; di < 3; ++di)
                u[dj][di] = MP_LD(F + checked_index(a.status, min(max(j + dj - 1, 0), ny - 1) * nx + min(max(i + di - 1, 0), nx - 1), N, active));
        double lo = u[1][1], hi = u[1][1];
        const double mean = u[1][1];
#pragma unroll
        for (int dj = 0; dj < 3; ++dj)
#pragma unroll
            for (int di = 0; di < 3; ++di) {
                const double v = u[dj][di];
                lo = v < lo ? v : lo;
                hi = v > hi ? v : hi;
            }
        const bool small = lo > -kScanGuard && hi < kScanGuard;
        lo = fmax(0.0, lo);
        const double top = f ? m.ph.k.Xe : INFINITY;
        hi = top < hi ? top : hi;
        double D[9];
        const int st = reconstruct(t, candidate_mask(ci, cj), u, D);
        Extremes x{D[0], D[0]};
        double mq;
        bool bad = false;
        if (small) {
            // Pairs: rows 0, g1 | g2, 0.8 | row 1, column 0.8 | column 1 (twice).
            const double ca = part == 0 ? 0.0 : part == 1 ? kG2 : 1.0, cb = part == 0 ? kG1 : part == 3 ? 1.0 : 0.8;
            auto pair = [&](bool col, double c) {
                const double p0[3] = {D[0], col ? D[3] : D[1], col ? D[6] : D[2]};
                const double p1[3] = {col ? D[1] : D[3], D[4], col ? D[7] : D[5]};
                const double p2[3] = {col ? D[2] : D[6], col ? D[5] : D[7], D[8]};
                x.line_pair(c, p0, p1, p2);
            };
            mq = D[0];
            pair(part == 3, ca);
            if (part == 1) mq = x.mx;
            pair(part >= 2, cb);
            if (part == 0) mq = x.mx;
            // The 0.3-size line of one side (parts 0, 1: bottom and top rows,
            // 2, 3: left and right columns), or the wall's three.
            const bool col = part >= 2;
            const int side = (part & 1) * 2, at = col ? ci : cj;
            auto line = [&](double c) {
                double a0, a1, a2, b0, b1, b2;
                q2_row(D, c, a0, a1, a2);
                q2_col(D, c, b0, b1, b2);
                x.line(col ? b0 : a0, col ? b1 : a1, col ? b2 : a2);
            };
            const double sgn = side ? -1.0 : 1.0;
            line(at == side ? 0.35 * sgn : -0.4 * sgn);
            if (at == side) { line(-0.1 * sgn); line(-0.55 * sgn); }
        } else {
            double Dc[9], mx, mn;
#pragma unroll
            for (int k = 0; k < 9; ++k) Dc[k] = D[k];
            scan_lines_exact(t, t.line_off[cj * 3 + ci], t.line_off[cj * 3 + ci + 1], Dc, mx, mn, bad);
            x = Extremes{mx, mn};
            mq = mx;
        }
        rest |= small_limit(m.ph, active, part, f, cell, mean, lo, hi, x, mq, st, bad, D, a.rec, a.flags, a.status,
                    [&](double& t0, double& t1) {
                        t0 = t1 = m.ph.Tep;
                        if (m.ph.litho) {
                            t0 = tep_at(m.ph, t.y0 + j * t.dy);
                            t1 = tep_at(m.ph, t.y0 + (j + 1) * t.dy);
                        }
                    });
    }
    if (__any_sync(kAll, rest)) small_cells_rest<false, kLitho>(m, kind, group, groups);
}

// The same on a general quad mesh: each lane of a field scans one edge's
// points and samples and a quarter of the cell's Gauss points.
__device__ __noinline__ void small_quad_recon(const SmallArgs& m, int kind, int group, int groups) {
    const QuadStageArgs& a = m.quad[kind];
    const QuadDev& q = a.q;
    const int nx = m.nx, ny = m.ny, N = nx * ny;
    const int l = threadIdx.x & 7, f = l >> 2, part = l & 3;
    bool rest = false;
    for (int base = group - ((threadIdx.x & 31) >> 3); base < N; base += groups) {
        const int c0 = base + (int)((threadIdx.x & 31) >> 3);
        bool active = c0 < N;
        const int cell = checked_index(a.status, active ? c0 : N - 1, N, active);
        const int i = cell % nx, j = cell / nx;
        const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = j == 0 ? 0 : (j == ny - 1 ? 2 : 1);
        const double* F = f ? a.C : a.H;
        double u[1][3][3];
#pragma unroll
        for (int dj = 0; dj < 3; ++dj)
#pragma unroll
            for (int di = 0; di < 3; ++di)
                u[0][dj][di] = MP_LD(F + checked_index(a.status, min(max(j + dj - 1, 0), ny - 1) * nx + min(max(i + di - 1, 0), nx - 1), N, active));
        const double mean = u[0][1][1];
        double lo = mean, hi = mean;
#pragma unroll
        for (int dj = 0; dj < 3; ++dj)
#pragma unroll
            for (int di = 0; di < 3; ++di) { lo = fmin(lo, u[0][dj][di]); hi = fmax(hi, u[0][dj][di]); }
        lo = fmax(0.0, lo);
        if (f) hi = fmin(m.ph.k.Xe, hi);
        double D[1][9];
        const int st = reconstruct_quad<1>(q, (size_t)N, cell, ci, cj, 1e-2 * __ldg(q.geo + 3 * (size_t)N + cell), u, D);
        const CellFrame fr = cell_frame(q, nx, (size_t)N, cell);
        double size = 0.0;
#pragma unroll
        for (int k = 0; k < 9; ++k) size += fabs(D[0][k]);
        Extremes x;
        double mq;
        bool bad = false;
        if (size < 0.5 * kQuadGuard) {
            const NormalCell k = normal_cell(fr);
            x.mx = x.mn = q2v(D[0], k.m.x, k.m.y);
            auto visit = [&](double px, double py) {
                const double v = q2v(D[0], px, py);
                x.up(v); x.down(v);
            };
            for (int n = part; n < kNQ * kNQ; n += 4) {
                const double s = q.gq[n / kNQ], r = q.gq[n % kNQ];
                visit(fma(fma(k.d.x, s, k.b.x), r, fma(k.c.x, s, k.m.x)), fma(fma(k.d.y, s, k.b.y), r, fma(k.c.y, s, k.m.y)));
            }
            mq = x.mx;
            long long id;
            bool wall, rev;
            cell_edge(nx, ny, i, j, 0, ny, part, id, wall, rev);
            id = checked_index(a.status, id, nx * (ny + 1) + (nx + 1) * ny, active);
            const P2 p = part == 0 ? k.n[0] : part == 1 ? k.n[1] : part == 2 ? k.n[2] : k.n[3];
            const P2 v = part == 0 ? k.n[1] : part == 1 ? k.n[2] : part == 2 ? k.n[3] : k.n[0];
            const P2 mid = P2{0.5 * (p.x + v.x), 0.5 * (p.y + v.y)}, half = P2{0.5 * (v.x - p.x), 0.5 * (v.y - p.y)};
            P2 nrm;
            double len;
            edge_geometry(p, v, len, nrm);
            for (int g = 0; g < kNQ; ++g) {
                const double px = fma(half.x, q.gq[g], mid.x), py = fma(half.y, q.gq[g], mid.y);
                const double sp = __ldg(q.sp + id * kNQ + (rev ? kNQ - 1 - g : g)) * fr.inv_h;
                const double sx = sp * nrm.x, sy = sp * nrm.y;
                visit(px, py);
                if (wall) {
                    for (int n = 1; n <= 4; ++n) visit(fma(-n, sx, px), fma(-n, sy, py));
                } else {
                    visit(fma(-1.5, sx, px), fma(-1.5, sy, py));
                    visit(fma(-0.5, sx, px), fma(-0.5, sy, py));
                }
            }
        } else {
            double Dc[9], ext[4];
#pragma unroll
            for (int k = 0; k < 9; ++k) Dc[k] = D[0][k];
            quad_scan_exact(a, cell, Dc, Dc, ext, &bad);
            x = Extremes{ext[0], ext[1]};
            mq = ext[0];
        }
        rest |= small_limit(m.ph, active, part, f, cell, mean, lo, hi, x, mq, st, bad, D[0], a.rec, a.flags, a.status,
                    [&](double& t0, double& t1) {
                        t0 = t1 = m.ph.Tep;
                        if (m.ph.litho) {
                            double ylo = fr.c[0].y, yhi = fr.c[0].y;
#pragma unroll
                            for (int k = 1; k < 4; ++k) { ylo = fmin(ylo, fr.c[k].y); yhi = fmax(yhi, fr.c[k].y); }
                            t0 = tep_at(m.ph, ylo);
                            t1 = tep_at(m.ph, yhi);
                        }
                    });
    }
    if (__any_sync(kAll, rest)) small_cells_rest<true, false>(m, kind, group, groups);
}

// Cell quadrature of the plain cells: lane b < 5 takes row b.
template <bool kQuad, bool kLitho>
__device__ __noinline__ void small_phase(const SmallArgs& m, int kind, int group, int groups) {
    const int nx = m.nx, N = nx * m.ny, l = threadIdx.x & 7, b = min(l, kNQ - 1);
    const CellPhaseArgs& a = m.phase[kind];
    for (int base = group - ((threadIdx.x & 31) >> 3); base < N; base += groups) {
        const int c0 = base + (int)((threadIdx.x & 31) >> 3);
        bool active = c0 < N;
        const int cell = checked_index(a.status, active ? c0 : N - 1, N, active);
        const unsigned char fl = a.flags[cell];
        double Trow = 0.0, Prow = 0.0;
        if (fl & FLAG_PLAIN) {
            double DH[9], DC[9];
            load_rec(a.rec, cell, DH, DC);
            DH[0] += MP_LD(a.H + cell);
            DC[0] += MP_LD(a.C + cell);
            if (kQuad) {
                const QuadDev& q = m.quad[kind].q;
                const CellFrame f = cell_frame(q, nx, (size_t)N, cell);
                const NormalCell k = normal_cell(f);
                double j0, jr, js;
                k.mean_jacobian(j0, jr, js);
                const double s = q.gq[b], ws = q.gw[b], js0 = fma(js, s, j0);
                const double x0 = fma(k.c.x, s, k.m.x), y0 = fma(k.c.y, s, k.m.y);
                const double x1 = fma(k.d.x, s, k.b.x), y1 = fma(k.d.y, s, k.b.y);
#pragma unroll
                for (int r = 0; r < kNQ; ++r) {
                    const double x = fma(x1, q.gq[r], x0), y = fma(y1, q.gq[r], y0);
                    const double w = ws * q.gw[r] * fma(jr, q.gq[r], js0);
                    const double tep = m.ph.litho ? tep_at(m.ph, fma(y, 1.0 / f.inv_h, f.cy)) : m.ph.Tep;
                    PhaseLean pl;
                    phase_plain<false>(m.ph.sk, q2v(DH, x, y), q2v(DC, x, y), tep, pl);
                    Trow = fma(w, pl.T, Trow);
                    Prow = fma(w, pl.phil, Prow);
                }
            } else {
                const StageHot& t = m.tab;
                const double y = t.g[b];
                double h0, h1, h2, d0, d1, d2;
                q2_row(DH, y, h0, h1, h2);
                q2_row(DC, y, d0, d1, d2);
                const double tep = (kLitho && m.ph.litho) ? tep_at(m.ph, height(t, cell / nx, y)) : m.ph.Tep;
#pragma unroll
                for (int r = 0; r < kNQ; ++r) {
                    const double x = t.g[r];
                    PhaseLean pl;
                    phase_plain<false>(m.ph.sk, quad(h0, h1, h2, x), quad(d0, d1, d2, x), tep, pl);
                    const double w = t.cw[b * kNQ + r];
                    Trow = fma(w, pl.T, Trow);
                    Prow = fma(w, pl.phil, Prow);
                }
            }
        }
        const double T = rows_sum(Trow), P = rows_sum(Prow);
        if (active && l == 0 && (fl & FLAG_PLAIN)) {
            if (m.ph.litho) a.flags[cell] = (unsigned char)(fl | (P > 0.0 ? FLAG_WET : 0));
            a.T[cell] = T;
            a.phi[cell] = P;
        }
    }
}

// Faces: lane p < 5 takes the p-th Gauss point in the kernels' order.
template <bool kQuad, bool kLitho>
__device__ __noinline__ void small_faces(const SmallArgs& m, int kind, int group, int groups) {
    const int nx = m.nx, ny = m.ny, N = nx * ny, edges = nx * (ny + 1) + (nx + 1) * ny;
    const int l = threadIdx.x & 7, p = min(l, kNQ - 1);
    const FaceArgs& a = m.face[kind];
    const Physics& ph = m.ph;
    bool rest = false;
    for (int base = group - ((threadIdx.x & 31) >> 3); base < edges; base += groups) {
        const int k0 = base + (int)((threadIdx.x & 31) >> 3);
        bool active = k0 < edges;
        const EdgeAt at = edge_by_kind(nx, ny, active ? k0 : edges - 1);
        EdgeCells g = edge_cells(a, at);
        g.e = checked_index(a.status, g.e, edges, active);
        g.L = checked_index(a.status, g.L, N, active);
        if (!g.boundary) g.R = checked_index(a.status, g.R, N, active);
        const unsigned char fl = a.flags[g.L] & (g.boundary ? 0xff : a.flags[g.R]);
        const bool plain = (fl & FLAG_PLAIN) != 0, wet = (fl & FLAG_WET) != 0;
        PointFlux pf{0.0, 0.0, 0.0, 0.0};
        double w[kNQ], half = 0.0;
#pragma unroll
        for (int n = 0; n < kNQ; ++n) w[n] = kQuad ? m.quad[kind].q.gw[n] : m.tab.gw[face_point_at(n)];
        int st = 0;
        if (plain) {
            const double sgn = g.reverse ? -1.0 : 1.0;
            double hL, cL, hR = 0.0, cR = 0.0, tep;
            int v;                           // canonical Gauss point
            if (kQuad) {
                const QuadStageArgs& qa = m.quad[kind];
                const QuadEdge e = quad_edge(qa.q, nx, ny, 0, ny, at.horizontal, at.i, at.j);
                P2 nrm;
                double len;
                edge_geometry(e.a, e.b, len, nrm);
                half = 0.5 * len;
                const double s = qa.q.gq[p];
                v = g.reverse ? kNQ - 1 - p : p;
                tep = ph.litho ? tep_at(ph, lerp_edge(s, e.a, e.b).y) : ph.Tep;
                auto side = [&](long long cell, double& h, double& c) {
                    const double cx = __ldg(qa.q.geo + cell), cy = __ldg(qa.q.geo + N + cell),
                                 inv_h = 1.0 / __ldg(qa.q.geo + 2 * (size_t)N + cell);
                    double DH[9], DC[9];
                    load_rec(a.rec, cell, DH, DC);
                    DH[0] += MP_LD(a.H + cell);
                    DC[0] += MP_LD(a.C + cell);
                    const P2 u = normalised(e.a, cx, cy, inv_h), z = normalised(e.b, cx, cy, inv_h);
                    const double x = fma(0.5 * (z.x - u.x), s, 0.5 * (u.x + z.x)), y = fma(0.5 * (z.y - u.y), s, 0.5 * (u.y + z.y));
                    h = q2v(DH, x, y);
                    c = q2v(DC, x, y);
                };
                side(g.L, hL, cL);
                if (!g.boundary) side(g.R, hR, cR);
            } else {
                const StageHot& t = m.tab;
                v = face_point_at(p);
                const double x = t.g[v], x2 = x * x;
                half = 0.5 * (at.horizontal ? t.len_h : t.len_v);
                tep = face_tep<kLitho>(t, a, ph, at, x);
                double h[3], c[3];
                edge_line(a, g.L, at.horizontal, at.horizontal == g.reverse ? 1.0 : -1.0, h, c);
                hL = fma(h[1], x, fma(h[2], x2, h[0]));
                cL = fma(c[1], x, fma(c[2], x2, c[0]));
                if (!g.boundary) {
                    edge_line(a, g.R, at.horizontal, at.horizontal ? 1.0 : -1.0, h, c);
                    hR = fma(h[1], x, fma(h[2], x2, h[0]));
                    cR = fma(c[1], x, fma(c[2], x2, c[0]));
                }
            }
            const double vs = sgn * __ldg(a.vsn + g.e * kNQ + v), ud = sgn * __ldg(a.udn + g.e * kNQ + v);
            PhaseLean A, B;
            phase_plain<true>(ph.sk, hL, cL, tep, A);
            if (g.boundary) {
                pf = wall_point_plain(ph, A, cL, wet, vs, ud, tep, st);
            } else {
                phase_plain<true>(ph.sk, hR, cR, tep, B);
                pf = face_point_plain(ph, A, B, cL, cR, wet, vs, ud, st);
            }
        }
        const double fluxH = points_sum(w, pf.fh), fluxC = points_sum(w, pf.fc), fluxMix = points_sum(w, pf.vn),
                     rate = points_sum(w, pf.speed);
#pragma unroll
        for (int n = 0; n < kNQ; ++n) {
            const int s = __shfl_sync(kAll, st, n, kGroup);
            st = st ? st : s;
        }
        rest = rest || (active && (!plain || (!kQuad && ph.diffusion)));
        if (active && l == 0 && plain) {
            if (st) record_error(a.status, PART_FACES, g.L, st);
            store_face(a, g.e, half, fluxH, fluxC, rate, fluxMix);
        }
    }
    if (__any_sync(kAll, rest)) small_edges_rest<kQuad, kLitho>(m, kind, group, groups);
    if (kQuad && ph.diffusion) small_quad_diffusion(m, kind, group, groups);
}

template <bool kQuad>
__device__ __noinline__ void small_sums(const SmallArgs& m, int kind, int rank, int blocks, double dt) {
    const int per = sum_cells_per_block(m.nx * m.ny), chunks = (m.nx * m.ny + per - 1) / per;
    for (int b = rank; b < chunks; b += blocks) {
        Partial v = partial_identity();
        if (threadIdx.x < kRedBlock) v = sum_cells<false, kQuad>(m.sum[kind], (long long)b * per, &dt);
        v = block_reduce(v);
        if (threadIdx.x == 0) m.partial[b] = v;
    }
}

template <bool kQuad, bool kLitho>
__global__ void __launch_bounds__(kSmallThreads, 1) small_steps_kernel(const __grid_constant__ SmallArgs m) {
    static_assert(kSmallThreads >= kRedBlock && kSmallCells <= kRedBlock * kRedBlock, "the reductions' block");
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ Board own;
    const Board* board = cluster.map_shared_rank(&own, 0);
    const int blocks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
    const bool lead = rank == 0 && threadIdx.x == 0;
    // Elements go to the cluster's warps in turn, four groups of lanes each,
    // neighbouring warps' elements to different blocks.
    const int warp = (int)(threadIdx.x >> 5) * blocks + rank;
    const int group = warp * 4 + (int)((threadIdx.x & 31) >> 3), groups = blocks * (kSmallThreads / 32) * 4;
    const int first = warp * 32 + (int)(threadIdx.x & 31), stride = blocks * kSmallThreads;
    const int N = m.nx * m.ny;
    const int per = sum_cells_per_block(N), chunks = (N + per - 1) / per;

    // Add the chunks' shares up as finish_block does, then let the lead thread
    // run `rule` on the totals and publish its decision. The first barrier is
    // also what lets the lead write the board: every block has read the
    // previous decision before it arrives.
    auto conclude = [&](auto&& rule) {
        cluster.sync();
        if (rank == 0) {
            Partial v = partial_identity();
            if ((int)threadIdx.x < chunks) fold_partial(v, m.partial[threadIdx.x]);
            v = block_reduce(v);
            if (threadIdx.x == 0) {
                own.tot = Totals{v.maxRate, v.divergence, v.bH, v.bC, v.HI, v.CI, v.Hmin, v.Cmin, v.Cmax, v.nonfinite, v.sH};
                rule();
            }
        }
        cluster.sync();
    };
    auto word = [&]() { return *(volatile unsigned long long*)m.status; };
    // One stage evaluation; dt scales the Runge-Kutta combination.
    auto stage = [&](int kind, double dt) {
        if (kQuad) small_quad_recon(m, kind, group, groups);
        else small_recon<kLitho>(m, kind, group, groups);
        cluster.sync();
        // T and phi of the accepted state; with a lithostatic pressure every
        // stage's wet flags, which the faces read.
        if (kind == KIND_P || m.ph.litho) small_phase<kQuad, kLitho>(m, kind, group, groups);
        if (m.ph.litho) cluster.sync();
        small_faces<kQuad, kLitho>(m, kind, group, groups);
        cluster.sync();
        small_sums<kQuad>(m, kind, rank, blocks, dt);
    };

    if (lead) {
        own.c = *m.ctl;
        *m.status = ~0ULL;
    }
    const int nsteps = m.hdr->nsteps;
    int step = 0, attempts_total = 0, stop = 0;
    for (; step < nsteps && !stop; ++step) {
        if (lead) {
            begin_one(own.c, m.reports[step], m.opts, false);
            attempt_one(own.c, m.opts);
            own.go = own.c.pending;
            own.dt = own.c.dt;
        }
        cluster.sync();
        for (int attempt = 0; attempt < kMaxAttempts; ++attempt) {
            const int go = board->go;
            const double dt = board->dt;
            if (!go) break;
            ++attempts_total;
            for (int b = rank; b < chunks; b += blocks) {
                Partial v = partial_identity();
                if (threadIdx.x < kRedBlock)
                    v = axpy_cells(N, m.H0, m.C0, m.LH, m.LC, dt, m.tab.area, m.H1, m.C1, (long long)b * per, m.cell_area);
                v = block_reduce(v);
                if (threadIdx.x == 0) m.partial[b] = v;
            }
            conclude([&] {
                own.c.valid = own.c.pending && admissible_dev(own.tot, m.opts.Xe);
                own.go = own.c.valid;
                *m.status = ~0ULL;
            });
            for (int which = 2; which <= 2 + m.opts.rk3; ++which) {
                const int last = which == 2 + m.opts.rk3;
                auto rule = [&] {
                    after_stage_one(own.c, m.opts, word(), own.tot, which, last);
                    *m.status = ~0ULL;
                    if (last) attempt_one(own.c, m.opts);
                    own.go = last ? own.c.pending : own.c.valid;
                    own.dt = own.c.dt;
                };
                if (board->go) {
                    stage(which == 2 ? KIND_B : KIND_C, dt);
                    conclude(rule);
                } else {
                    // Nothing evaluated: the rule alone (halve dt at the end).
                    cluster.sync();
                    if (lead) rule();
                    cluster.sync();
                }
            }
        }
        cluster.sync();   // every block has read the decision that ended the loop
        if (lead) {
            // Unreachable by the retry rule (40 retries fail the next attempt).
            if (own.c.pending) fail_inst(own.c, MP_ERR_NOT_CONVERGED, FAIL_RETRIES);
            commit_one(own.c, m.reports[step], m.opts);
            own.go = own.c.done;
        }
        cluster.sync();
        if (board->go) {
            for (int k = first; k < N; k += stride) {
                m.H[k] = m.newH[k];
                m.C[k] = m.newC[k];
            }
            cluster.sync();
            stage(KIND_P, 0.0);
            conclude([&] {
                after_rhs_one(own.c, m.reports[step], m.opts, word(), own.tot);
                *m.status = ~0ULL;
                own.go = own.c.status == 0;
            });
        } else {
            cluster.sync();
            if (lead) {
                after_rhs_one(own.c, m.reports[step], m.opts, ~0ULL, own.tot);
                own.go = own.c.status == 0;
            }
            cluster.sync();
        }
        stop = !board->go;
        cluster.sync();   // every block has read the board before the next step writes it
    }
    if (lead) {
        *m.ctl = own.c;
        m.hdr->step = step;
        m.hdr->total_attempts = attempts_total;
        m.hdr->stop = stop;
    }
}

const void* small_kernel(bool quad, bool litho) {
    return quad ? (const void*)small_steps_kernel<true, false>
                : litho ? (const void*)small_steps_kernel<false, true> : (const void*)small_steps_kernel<false, false>;
}

cudaLaunchConfig_t small_config(int blocks, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(kSmallThreads);
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

// Blocks of the cluster: 16 where this GPU can hold one, else 8, else 0.
int small_blocks(const void* f) {
    for (int blocks : {16, 8}) {
        if (cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, blocks > 8) != cudaSuccess) { cudaGetLastError(); continue; }
        cudaLaunchAttribute attr[1];
        const cudaLaunchConfig_t cfg = small_config(blocks, attr);
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, f, &cfg) == cudaSuccess && n > 0) return blocks;
        cudaGetLastError();
    }
    return 0;
}

}  // namespace

// Four SSPRK3 steps, this kernel / the graph (us; retries differ from mesh to
// mesh). Uniform: 20x20 338 / 523, 25x40 509 / 647, 32x48 521 / 574, 32x64 and
// beyond slower; with a lithostatic pressure, whose wet flags need the
// quadrature in every stage, 25x40 440 / 474, 32x40 496 / 486; with diffusion
// 25x40 688 / 835, 32x40 636 / 637. Perturbed: 20x24 601 / 955, 25x40 603 / 735,
// 32x48 slower, lithostatic 25x40 634 / 724; with diffusion 20x24 807 / 1240,
// 25x40 882 / 951. Where no cell is plain the tested forms have a lane per
// element in both and the graph has more of the GPU: pure component 20x20
// 514 / 526, 32x48 617 / 537, with diffusion 20x20 696 / 665, 25x40 1019 / 847;
// perturbed 25x40 886 / 790, with diffusion 20x24 878 / 927, 20x32 998 / 943,
// 25x40 1111 / 919. The limits are where the ordinary cells gain and those do
// not lose more. A cluster of 8 blocks has half the throughput: 20x20 384,
// 24x32 597 / 652, 25x40 670 / 647, perturbed 20x24 717 / 955, 25x32 802 / 746.
int small_steps_blocks(const SmallMesh& m) {
    const long long cells = (long long)m.nx * m.ny;
    const long long limit = m.quad ? (m.ph->diffusion ? kSmallQuadDiffusion : kSmallQuadCells)
                                   : (m.ph->diffusion || m.ph->litho ? kSmallCellsMore : kSmallCells);
    if (cells > limit || m.ph->source) return 0;
    const int blocks = small_blocks(small_kernel(m.quad, m.ph->litho != 0));
    return 16 * cells <= limit * blocks ? blocks : 0;
}

mp_status launch_small_steps(const SmallMesh& s, int blocks, cudaStream_t stream) {
    SmallArgs m{};
    m.ph = *s.ph;
    m.opts = s.opts;
    m.nx = s.nx; m.ny = s.ny;
    if (!s.quad) m.tab = *s.tab;
    const bool rk3 = s.opts.rk3 != 0;
    const double area = s.quad ? 1.0 : s.tab->area;
    for (int k = 0; k < NKIND; ++k) {
        const double* inH = k == KIND_P ? s.H : (k == KIND_B ? s.S1H : s.S2H);
        const double* inC = k == KIND_P ? s.C : (k == KIND_B ? s.S1C : s.S2C);
        double* outH = k == KIND_P ? s.LH : (k == KIND_B ? s.S2H : s.S1H);
        double* outC = k == KIND_P ? s.LC : (k == KIND_B ? s.S2C : s.S1C);
        m.recon[k] = ReconArgs{s.nx, s.ny, nullptr, inH, inC, s.rec, s.flags, s.status, nullptr};
        m.phase[k] = CellPhaseArgs{s.nx, s.ny, nullptr, inH, inC, s.rec, s.flags, s.T, s.phi, s.status};
        m.face[k] = FaceArgs{s.nx, s.ny, nullptr, inH, inC, s.rec, s.flags, s.vsn, s.udn, s.face, s.status};
        if (s.quad) {
            QuadStageArgs& q = m.quad[k];
            q.nx = s.nx; q.ny = s.ny; q.gj0 = 0; q.gny = s.ny;
            q.H = inH; q.C = inC; q.rec = s.rec; q.flags = s.flags; q.T = s.T; q.phi = s.phi;
            q.vsn = s.vsn; q.udn = s.udn; q.face = s.face; q.status = s.status;
            q.q = s.q;
        }
        const double a0 = k == KIND_B ? (rk3 ? 0.75 : 0.5) : 1.0 / 3.0, a1 = k == KIND_B ? (rk3 ? 0.25 : 0.5) : 2.0 / 3.0;
        m.sum[k] = SumArgs{s.nx, s.ny, area, 1.0 / area, s.face, inH, inC, s.H, s.C, outH, outC, s.rate,
                           k == KIND_P ? (int)SUM_STORE_L : (int)SUM_RK, a0, a1, 0.0, Shares{s.partial, nullptr, nullptr, 0}, nullptr};
        m.sum[k].cell_area = s.cell_area;
        m.sum[k].status = s.status;
    }
    m.H0 = s.H; m.C0 = s.C; m.LH = s.LH; m.LC = s.LC; m.H1 = s.S1H; m.C1 = s.S1C;
    m.newH = rk3 ? s.S1H : s.S2H; m.newC = rk3 ? s.S1C : s.S2C;
    m.H = s.H; m.C = s.C;
    m.tab.area = area;
    m.cell_area = s.cell_area;
    m.partial = s.partial; m.status = s.status; m.ctl = s.ctl; m.hdr = s.hdr; m.reports = s.reports;
    const void* f = small_kernel(s.quad, s.ph->litho != 0);
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = small_config(blocks, attr);
    cfg.stream = stream;
    void* args[] = {&m};
    MP_CUDA(cudaLaunchKernelExC(&cfg, f, args));
    return MP_OK;
}

}  // namespace mp
