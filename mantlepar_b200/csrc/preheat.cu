// Legacy dry preheat on B200 (mantle::couple::AdvanceLegacyPreheat,
// src/couple/preheat.cpp:65-287): H_t + div(us H - kappa grad H) = 0 with C
// fixed and the Stokes velocity frozen, forward Euler.
//
// One step is one kernel (pre_step_kernel): per cell the unlimited deviation
// polynomial of H (StateReconstruction::Update(s, false): limiter 1), per edge
// the traces of both sides at the 5 Gauss points, the linear-law Lax-Friedrichs
// flux or the boundary policy and the diffusion of the cell averages, then the
// face fluxes summed in the reference's face order and H + dt*rhs into the
// other state buffer, with block partials; the last block to finish folds them
// in a fixed order and applies the step's checks (finite candidate, heat
// balance), accepting or stopping. The step sizes do not depend on the state (the rate is fixed at Build), so
// the host plans a batch of steps and issues them without waiting; a failed
// step sets the status words and every kernel queued after it does no work.
//
// On a general quad mesh (mp_preheat_create_quads; the reference's preheat
// runs on any mesh family, preheat.cpp:86-117) the step, rate and diagnostics
// kernels have quad forms that read the per-cell tables, map every point from
// the cell's corners and use physical edge lengths, normal-line spacing per
// edge point and per-cell areas.
#include "common.hpp"
#include "phase_math.cuh"
#include "stage_device.cuh"
#include "stage_kernels.cuh"
#include "quad_device.cuh"
#include "quad_tables.hpp"
#include "tables.hpp"

#include <algorithm>
#include <cmath>
#include <limits>
#include <vector>

#include <cuda_pipeline.h>

namespace mp {

PhaseConst phase_const(const mp_material& p, const mp_derived& d);
mp_status derive_checked(const mp_material& p, mp_derived& d);

namespace {

// Boundary and flux constants of the preheat kernels.
struct PreheatPhys {
    double kappa;
    int diffusion;         // kappa > 0 or a wall prescribes a flux
    int wall_type[4];      // MP_THERMAL_* per wall: bottom, top, left, right
    double wall_value[4];
    int Hpol;              // MP_BC_* of H
    double inflowH;
    int lf_global;
    double lf_speed;
    // Diffusion of constant samples (preheat.cpp:183-194 with
    // diffusiveflux.cpp:105-200): interior samples [L, L, R, R], wall samples
    // [L, L, L, L, wall value], gradient sum_k c_k (v_k - v_last) / ds, so the
    // flux is -kappa times these sums of c_k times (v_L - v_last) / ds.
    double c_int, c_bnd;
    double dif[2][2];      // uniform mesh: -kappa times these, integrated over a [horizontal, vertical] [interior, wall] edge
    double inv_area;
};

// Block partial of the preheat reductions.
struct PrePartial {
    double integral, minimum, maximum, bflux, nonfinite;
};
__device__ __forceinline__ PrePartial pre_identity() { return PrePartial{0.0, INFINITY, -INFINITY, 0.0, 0.0}; }

// Device record of one step (the host adds step, time, dt and courant).
struct PreRow {
    double integral, minimum, maximum, bflux, balance;
};

// Device control block of a preheat instance.
struct PreCtl {
    double prev_integral;      // integral of the latest accepted state
    unsigned int ticket;       // blocks finished in the running launch
    unsigned int accepted;     // steps accepted (running count)
    PrePartial last;           // totals of the latest rhs / measure / rate launch
};

enum PreMode : int { PRE_STEP = 0, PRE_RHS = 1 };

constexpr int kPreBlock = 256;
constexpr int kPrePer = 4;                      // cells per thread in the per-cell kernels
constexpr int kPreCells = kPreBlock * kPrePer;

// The status words: [0] the first failure, which every block of a launch may
// lower while the others still run, and [1] set by a launch's last block once
// the step has failed. Launches queued after it go by [1], so that every block
// of the failing launch does its work and the failure reported is the first by
// part and key, whichever block met one first.
__device__ __forceinline__ bool halted(const unsigned long long* status) {
    return *(volatile const unsigned long long*)(status + 1) != ~0ULL;
}

// Fixed-tree block reduction; the result is valid in thread 0.
__device__ PrePartial pre_block_reduce(PrePartial v) {
    __shared__ double sh[kPreBlock / 32][5];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double r[5] = {warp_sum(v.integral), warp_min(v.minimum), warp_max(v.maximum), warp_sum(v.bflux),
                   warp_max(v.nonfinite)};
    if (lane == 0)
        for (int k = 0; k < 5; ++k) sh[warp][k] = r[k];
    __syncthreads();
    PrePartial out = pre_identity();
    if (warp == 0) {
        const int nw = blockDim.x >> 5;
        double s[5] = {0.0, INFINITY, -INFINITY, 0.0, 0.0};
        if (lane < nw) for (int k = 0; k < 5; ++k) s[k] = sh[lane][k];
        out = PrePartial{warp_sum(s[0]), warp_min(s[1]), warp_max(s[2]), warp_sum(s[3]), warp_max(s[4])};
    }
    __syncthreads();
    return out;
}

__device__ __forceinline__ void pre_fold(PrePartial& a, const PrePartial* p) {
    a.integral += __ldcg(&p->integral);
    a.minimum = fmin(a.minimum, __ldcg(&p->minimum));
    a.maximum = fmax(a.maximum, __ldcg(&p->maximum));
    a.bflux += __ldcg(&p->bflux);
    a.nonfinite = fmax(a.nonfinite, __ldcg(&p->nonfinite));
}

// Write this block's partial; the last block of the launch folds all of them
// in block order (the same sums whichever block finishes last) and returns
// true in every thread with the totals in `tot` (valid in thread 0).
__device__ bool pre_finish_blocks(PrePartial v, PrePartial* partial, PreCtl* ctl, PrePartial& tot) {
    __shared__ bool last;
    const unsigned blocks = gridDim.x * gridDim.y;
    const PrePartial b = pre_block_reduce(v);
    if (threadIdx.x == 0) {
        partial[blockIdx.y * gridDim.x + blockIdx.x] = b;
        __threadfence();
        last = atomicAdd(&ctl->ticket, 1u) == blocks - 1;
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
    PrePartial a = pre_identity();
    for (unsigned k = threadIdx.x; k < blocks; k += blockDim.x) pre_fold(a, partial + k);
    tot = pre_block_reduce(a);
    if (threadIdx.x == 0) ctl->ticket = 0;
    return true;
}

// Edge e of a uniform mesh (preheat.cpp:86-95): its direction, whether it is a
// wall and which, and whether the canonical normal points into the wall cell.
struct EdgeGeo {
    bool horizontal, boundary, reverse;
    int wall;
};

__device__ __forceinline__ EdgeGeo edge_geo(int nx, int ny, long long e) {
    const long long nI = (long long)nx * (ny + 1);
    EdgeGeo g;
    g.wall = -1;
    g.horizontal = e < nI;
    if (g.horizontal) {
        const int j = (int)((unsigned)e / (unsigned)nx);
        g.boundary = j == 0 || j == ny;
        g.reverse = j == ny;
        if (g.boundary) g.wall = j == 0 ? 0 : 1;
    } else {
        const int i = (int)((unsigned)(e - nI) % (unsigned)(nx + 1));
        g.boundary = i == 0 || i == nx;
        g.reverse = i == 0;
        if (g.boundary) g.wall = i == 0 ? 2 : 3;
    }
    return g;
}

// Relative roundoff allowance of a speed bound (advectiveflux.cpp:82-87).
__device__ __forceinline__ bool speed_bounds(double bound, double required) {
    return bound >= required || required - bound <= 64.0 * 2.220446049250313e-16 * fmax(bound, required);
}

// ------------------------------------------------------------------ kernels

// Arguments of one step (or RHS evaluation).
struct PreStepArgs {
    int nx, ny, passes, mode, row;
    double dt;
    const double* H;
    const double* vn;
    const double* edge;        // quad mesh: pre_quad_edge_kernel's table
    double* Hout;
    double* rhs;
    PreRow* rows;
    PrePartial* partial;
    PreCtl* ctl;
    unsigned long long* status;
};

constexpr int kStepBlock = 128;
constexpr int kStepRows = kStepBlock / 32;      // rows a block advances at a time, one per warp
constexpr int kStepCols = 30;                   // columns a warp owns; its outer lanes are the neighbours'
constexpr int kStepPasses = 32;

// What the flux of one edge needs besides the traces.
struct PreEdge {
    bool boundary;
    bool right;                // the wall cell is the right argument
    int wall;
    double sgn;                // -1: the canonical normal points into the wall cell
    double half;               // half its length
    double dif_int, dif_bnd;   // d flux / d (v_L - v_last)
};

// Whether the gradient at a wall of prescribed temperature, sum_k c_k x / ds in
// the order of its samples (c = 1/4, -4/3, 3, -4), overflows although the flux d,
// in which kappa scales it, may not. Out of line: |x| beyond 1e280.
__device__ __noinline__ bool wall_gradient_overflows(double kappa, double half, double x, double d) {
    return !isfinite(4.0 * x) || (kappa > 0.0 && !isfinite(d / (2.0 * half * kappa)));
}

// Edge flux of preheat.cpp:166-196: advection and diffusion of H out of the
// left (wall) cell. The traces and the velocity are finite exactly when every
// Lax-Friedrichs flux is or overflows, and the sum of them shows both, so the
// interior's points are tested one by one only when it is not finite.
__device__ __forceinline__ double pre_flux(const PreheatPhys& pp, const PreEdge& g, const double* gw, const double* v,
                                           const double (&uL)[kNQ], const double (&uR)[kNQ], double mL, double mR,
                                           int& st) {
    double sum = 0.0;
    if (!g.boundary) {
        bool low = false;
#pragma unroll
        for (int q = 0; q < kNQ; ++q) {
            const double vq = v[q];
            const double a = pp.lf_global ? pp.lf_speed : fabs(vq);
            if (pp.lf_global) low |= !(a >= fabs(vq));
            sum = fma(gw[q], fma(vq, uL[q] + uR[q], -(a * (uR[q] - uL[q]))), sum);
        }
        sum *= 0.5 * g.half;
        const double flux = pp.diffusion ? fma(g.dif_int, mL - mR, sum) : sum;
        if (low || !isfinite(flux)) {
#pragma unroll
            for (int q = 0; q < kNQ; ++q) {
                const double vq = v[q], a = pp.lf_global ? pp.lf_speed : fabs(vq);
                if (!isfinite(vq) || !isfinite(uL[q]) || !isfinite(uR[q]) || !speed_bounds(a, fabs(vq)))
                    st = st ? st : E_OUTOFRANGE;
                if (!isfinite(0.5 * (vq * uL[q] + vq * uR[q] - a * (uR[q] - uL[q])))) st = st ? st : E_FP;
            }
            if (pp.diffusion && !isfinite(g.dif_int * (mL - mR))) st = st ? st : E_FP;
        }
        return flux;
    }
    // EvaluateAdvectionBoundary (initialization.cpp:469-489) and the physical
    // boundary flux (advectiveflux.cpp:229-271).
#pragma unroll
    for (int q = 0; q < kNQ; ++q) {
        const double vq = g.sgn * v[q], u = g.right ? uR[q] : uL[q];
        if (!isfinite(vq) || !isfinite(u)) st = st ? st : E_OUTOFRANGE;
        double f;
        if (pp.Hpol == MP_BC_ZERO_FLUX || vq == 0.0) f = 0.0;
        else if (vq < 0.0) {
            if (pp.Hpol != MP_BC_INFLOW_OUTFLOW) st = st ? st : E_OUTOFRANGE;
            f = vq * pp.inflowH;
        } else f = vq * u;
        if (!isfinite(f)) st = st ? st : E_FP;
        sum = fma(gw[q], f, sum);
    }
    sum *= g.half;
    if (pp.diffusion) {
        const double wv = pp.wall_value[g.wall];
        if (pp.wall_type[g.wall] == MP_THERMAL_FLUX) {
            double w = 0.0;
#pragma unroll
            for (int q = 0; q < kNQ; ++q) w += gw[q];
            sum = fma(w * g.half, wv, sum);
        } else if (pp.wall_type[g.wall] == MP_THERMAL_TEMPERATURE) {
            const double x = (g.right ? mR : mL) - wv, d = g.dif_bnd * x;
            if (!isfinite(d) || (!(fabs(x) < 1e280) && wall_gradient_overflows(pp.kappa, g.half, x, d))) st = st ? st : E_FP;
            sum += d;
        }
    }
    return sum;
}

// One forward-Euler step (or the RHS) in one pass over memory. A block owns 30
// columns and walks up its rows four at a time, a row per warp and a column per
// lane. Each thread reconstructs its cell, hands its right trace to the next
// lane and its top trace to the next row (shared memory; the last row of a
// group stays for the next group), forms the fluxes of its cell's left and
// bottom edges, and finishes the cell below, whose four fluxes are then known.
// The outer lanes and the first and last row are the neighbours' cells,
// reconstructed again. Edge velocities come through shared memory in whole rows
// while the cells are reconstructed.
// Bound by instruction issue and FP64 latency on a uniform mesh, whose 96 bytes
// per cell take a third of the time, and by the cells' tables on a quad mesh.
// Separate kernels for the reconstruction, the faces and the update moved 280
// bytes per cell and waited for each other: 19 + 48 + 16 us at 640x1280 and
// 135 + 118 + 19 on a quad mesh, now 53 and 205. 16 steps at 1280x2560 take
// 2.63 ms at five blocks per SM (four 2.77, six 2.63 but 3 % more below); the
// quad form spills above four.
template <bool kQuad, class Tab>
__global__ void __launch_bounds__(kStepBlock, kQuad ? 4 : 5) pre_step_kernel(const __grid_constant__ PreStepArgs a,
                                                                 const __grid_constant__ PreheatPhys pp,
                                                                 const __grid_constant__ Tab tab) {
    constexpr int kTr = kQuad ? kNQ : 3;        // a trace: its values at the edge's points, or its coefficients
    __shared__ double top[2][kStepRows][kTr + 1][32];
    __shared__ double low[2][kStepRows][3][32];
    __shared__ double vbuf[kStepRows][2][32 * kNQ];
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int nx = a.nx, ny = a.ny;
    const long long nI = (long long)nx * (ny + 1);
    const size_t N = (size_t)nx * ny;
    PrePartial acc = pre_identity();
    if (!__syncthreads_or(halted(a.status))) {
        const int rows = a.passes * kStepRows - 2;
        const int y0 = blockIdx.y * rows, y1 = min(y0 + rows, ny);
        const int x0 = blockIdx.x * kStepCols, i = x0 - 1 + lane, x1 = min(x0 + kStepCols, nx);
        const bool mine = lane >= 1 && lane <= kStepCols && i < nx;
        const double* gw;
        if constexpr (kQuad) gw = tab.gw; else gw = tab.d.gw;
        auto point_values = [&](const double (&tr)[kTr], double (&u)[kNQ]) {
#pragma unroll
            for (int q = 0; q < kNQ; ++q) {
                if constexpr (kQuad) u[q] = tr[q];
                else u[q] = quad(tr[0], tr[1], tr[2], tab.d.g[q]);
            }
        };
        for (int pass = 0; pass < a.passes; ++pass) {
            const int base = y0 - 1 + pass * kStepRows, j = base + ty, par = pass & 1;
            if (base > y1) break;
            const bool vrow = j >= y0 && j < y1;        // its vertical edges count
            const bool hrow = j >= y0 && j <= y1;       // the edges below it count
            double* vv = vbuf[ty][0];
            double* vh = vbuf[ty][1];
            if (vrow) {
                const double* src = a.vn + (nI + (long long)j * (nx + 1) + x0) * kNQ;
                for (int k = lane; k < (x1 - x0 + 1) * kNQ; k += 32) __pipeline_memcpy_async(vv + k, src + k, sizeof(double));
            }
            if (hrow) {
                const double* src = a.vn + ((long long)j * nx + x0) * kNQ;
                for (int k = lane; k < (x1 - x0) * kNQ; k += 32) __pipeline_memcpy_async(vh + k, src + k, sizeof(double));
            }
            __pipeline_commit();
            const bool cell_in = j >= 0 && j < ny && j <= y1 && i >= 0 && i < nx;
            const long long cell = (long long)j * nx + i;
            double m = 0.0, tl[kTr] = {}, tr[kTr] = {}, tb[kTr] = {}, tt[kTr] = {};
            if (cell_in) {
                double u[1][3][3];
                const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = j == 0 ? 0 : (j == ny - 1 ? 2 : 1);
                const double* Hc = a.H + cell;
                const int west = ci == 0 ? 0 : -1, east = ci == 2 ? 0 : 1, rows3[3] = {cj == 0 ? 0 : -nx, 0, cj == 2 ? 0 : nx};
#pragma unroll
                for (int dj = 0; dj < 3; ++dj) {
                    const double* r = Hc + rows3[dj];
                    u[0][dj][0] = __ldg(r + west);
                    u[0][dj][1] = __ldg(r);
                    u[0][dj][2] = __ldg(r + east);
                }
                m = u[0][1][1];
                double D[1][9];
                int st;
                if constexpr (kQuad) st = reconstruct_quad<1>(tab, N, cell, ci, cj, 1e-2 * __ldg(tab.geo + 3 * N + cell), u, D);
                else st = reconstruct(tab.d, candidate_mask(ci, cj), u[0], D[0]);
                if (st) record_error(a.status, PART_UPDATE, cell, st);
                D[0][0] += m;
                if constexpr (kQuad) {
                    const double cx = __ldg(tab.geo + cell), cy = __ldg(tab.geo + N + cell);
                    const double inv_h = 1.0 / __ldg(tab.geo + 2 * N + cell);
                    const P2 c0 = normalised(vtx(tab, nx, i, j), cx, cy, inv_h),
                             c1 = normalised(vtx(tab, nx, i + 1, j), cx, cy, inv_h),
                             c2 = normalised(vtx(tab, nx, i + 1, j + 1), cx, cy, inv_h),
                             c3 = normalised(vtx(tab, nx, i, j + 1), cx, cy, inv_h);
                    auto along = [&](P2 s, P2 e, double (&v)[kTr]) {
                        const P2 mid = P2{0.5 * (s.x + e.x), 0.5 * (s.y + e.y)}, half = P2{0.5 * (e.x - s.x), 0.5 * (e.y - s.y)};
#pragma unroll
                        for (int q = 0; q < kNQ; ++q)
                            v[q] = q2v(D[0], fma(half.x, tab.gq[q], mid.x), fma(half.y, tab.gq[q], mid.y));
                    };
                    along(c0, c3, tl); along(c1, c2, tr); along(c0, c1, tb); along(c3, c2, tt);
                } else {
                    q2_col(D[0], -1.0, tl[0], tl[1], tl[2]); q2_col(D[0], 1.0, tr[0], tr[1], tr[2]);
                    q2_row(D[0], -1.0, tb[0], tb[1], tb[2]); q2_row(D[0], 1.0, tt[0], tt[1], tt[2]);
                }
            }
#pragma unroll
            for (int k = 0; k < kTr; ++k) {
                tr[k] = __shfl_up_sync(~0u, tr[k], 1);
                top[par][ty][k][lane] = tt[k];
            }
            top[par][ty][kTr][lane] = m;
            const double mw = __shfl_up_sync(~0u, m, 1);
            __pipeline_wait_prior(0);
            __syncthreads();
            // Left edge: the cells (i-1, j) and (i, j).
            double fl = 0.0, fb = 0.0, ms = 0.0;
            if (vrow && lane >= 1 && i <= x1) {
                const long long e = nI + (long long)j * (nx + 1) + i;
                double uw[kNQ], uo[kNQ];
                point_values(tr, uw);
                point_values(tl, uo);
                PreEdge g;
                g.boundary = i == 0 || i == nx;
                g.right = i == 0;
                g.wall = i == 0 ? 2 : 3;
                g.sgn = i == 0 ? -1.0 : 1.0;
                if constexpr (kQuad) {
                    const double2 w = __ldg(reinterpret_cast<const double2*>(a.edge) + e);
                    g.half = w.x; g.dif_int = -pp.kappa * pp.c_int * w.y; g.dif_bnd = -pp.kappa * pp.c_bnd * w.y;
                } else {
                    g.half = 0.5 * tab.d.len_v; g.dif_int = pp.dif[1][0]; g.dif_bnd = pp.dif[1][1];
                }
                int st = 0;
                fl = pre_flux(pp, g, gw, vv + (lane - 1) * kNQ, uw, uo, mw, m, st);
                if (st) record_error(a.status, PART_FACES, e, st);
            }
            // Bottom edge: the cells (i, j) and (i, j-1).
            if (hrow && mine) {
                const int sp = ty > 0 ? par : par ^ 1, sr = ty > 0 ? ty - 1 : kStepRows - 1;
                const long long e = (long long)j * nx + i;
                double ts[kTr], us[kNQ], uo[kNQ];
#pragma unroll
                for (int k = 0; k < kTr; ++k) ts[k] = top[sp][sr][k][lane];
                ms = top[sp][sr][kTr][lane];
                point_values(ts, us);
                point_values(tb, uo);
                PreEdge g;
                g.boundary = j == 0 || j == ny;
                g.right = j == ny;
                g.wall = j == 0 ? 0 : 1;
                g.sgn = j == ny ? -1.0 : 1.0;
                if constexpr (kQuad) {
                    const double2 w = __ldg(reinterpret_cast<const double2*>(a.edge) + e);
                    g.half = w.x; g.dif_int = -pp.kappa * pp.c_int * w.y; g.dif_bnd = -pp.kappa * pp.c_bnd * w.y;
                } else {
                    g.half = 0.5 * tab.d.len_h; g.dif_int = pp.dif[0][0]; g.dif_bnd = pp.dif[0][1];
                }
                int st = 0;
                fb = pre_flux(pp, g, gw, vh + (lane - 1) * kNQ, uo, us, m, ms, st);
                if (st) record_error(a.status, PART_FACES, e, st);
            }
            low[par][ty][0][lane] = fb;
            low[par][ty][1][lane] = fl;
            low[par][ty][2][lane] = __shfl_down_sync(~0u, fl, 1);
            __syncthreads();
            // The cell below: its fluxes in id order with each side's sign
            // (preheat.cpp:195-197), the candidate and the partials.
            if (hrow && j > y0 && mine) {
                const int sp = ty > 0 ? par : par ^ 1, sr = ty > 0 ? ty - 1 : kStepRows - 1;
                const double b = low[sp][sr][0][lane], l = low[sp][sr][1][lane], r = low[sp][sr][2][lane];
                const double sum = ((-b) + (j == ny ? -fb : fb)) + (i == 0 ? -l : l) - r;
                const long long done = cell - nx;
                double area, rate;
                if constexpr (kQuad) {
                    area = __ldg(tab.geo + 3 * N + done);
                    rate = sum / area;
                } else {
                    area = tab.d.area;
                    rate = sum * pp.inv_area;
                }
                if (j == 1) acc.bflux += b;
                if (j == ny) acc.bflux += fb;
                if (i == 0) acc.bflux += l;
                if (i == nx - 1) acc.bflux += r;
                double cand = ms;
                if (a.mode == PRE_RHS) a.rhs[done] = rate;
                else {
                    cand = __dadd_rn(ms, __dmul_rn(a.dt, rate));
                    a.Hout[done] = cand;
                }
                acc.integral = fma(cand, area, acc.integral);
                acc.minimum = fmin(acc.minimum, cand);
                acc.maximum = fmax(acc.maximum, cand);
                if (!isfinite(cand)) acc.nonfinite = 1.0;
            }
        }
    }
    PrePartial tot;
    if (!pre_finish_blocks(acc, a.partial, a.ctl, tot) || threadIdx.x != 0) return;
    if (a.mode != PRE_STEP) { a.ctl->last = tot; return; }
    // The step's checks (preheat.cpp:267-273), unless a cell or an edge failed.
    const double prev = a.ctl->prev_integral;
    const double bal = tot.integral - prev + a.dt * tot.bflux;
    const double tol = 1e-10 * (1.0 + fabs(tot.integral) + fabs(prev) + fabs(a.dt * tot.bflux));
    if (*(volatile unsigned long long*)a.status == ~0ULL) {
        if (tot.nonfinite != 0.0) record_error(a.status, PART_CELLS, 0, E_FP);
        else if (!(fabs(bal) <= tol)) record_error(a.status, PART_CELLS, 0, MP_ERR_PLIB);
        else {
            a.rows[a.row] = PreRow{tot.integral, tot.minimum, tot.maximum, tot.bflux, bal};
            a.ctl->prev_integral = tot.integral;
            a.ctl->accepted += 1;
            return;
        }
    }
    a.status[1] = 0;
}

// Integral, minimum and maximum of a state.
__global__ void __launch_bounds__(kPreBlock) pre_measure_kernel(long long N, double area,
                                                                const double* __restrict__ cell_area,
                                                                const double* __restrict__ H, PrePartial* partial,
                                                                PreCtl* ctl) {
    PrePartial v = pre_identity();
#pragma unroll
    for (int k = 0; k < kPrePer; ++k) {
        const long long cell = (long long)blockIdx.x * kPreCells + k * kPreBlock + threadIdx.x;
        if (cell >= N) continue;
        const double h = __ldg(H + cell);
        v.integral += h * (cell_area ? __ldg(cell_area + cell) : area);
        v.minimum = fmin(v.minimum, h);
        v.maximum = fmax(v.maximum, h);
        v.nonfinite = fmax(v.nonfinite, isfinite(h) ? 0.0 : 1.0);
    }
    PrePartial tot;
    if (pre_finish_blocks(v, partial, ctl, tot) && threadIdx.x == 0) ctl->last = tot;
}

// Build (preheat.cpp:130-156), per edge: LF speed sum_q L w_q alpha / 2 and
// the diffusion derivatives at zero samples summed per side; writes
// (speed + |derivative|) / area for the left [e] and right [NE + e] cell.
__global__ void __launch_bounds__(128) pre_rate_edge_kernel(int nx, int ny, double area, const double* __restrict__ vn,
                                                            double* __restrict__ rr, unsigned long long* status,
                                                            const __grid_constant__ PreheatPhys pp,
                                                            const __grid_constant__ ParamTables p) {
    const long long nE = (long long)nx * (ny + 1) + (long long)(nx + 1) * ny;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nE) return;
    const StageHot& t = p.d;
    const EdgeGeo g = edge_geo(nx, ny, e);
    const int o = g.horizontal ? 0 : 1;
    const double len = g.horizontal ? t.len_h : t.len_v;
    int st = 0;
    double speed = 0.0;
#pragma unroll
    for (int q = 0; q < kNQ; ++q) {
        const int cq = g.reverse ? kNQ - 1 - q : q;
        const double v = __ldg(vn + e * kNQ + cq);
        const double ns = fabs(v);
        if (!isfinite(v)) st = E_OUTOFRANGE;
        const double a = pp.lf_global ? pp.lf_speed : ns;
        if (!(a + 1e-14 >= ns)) st = E_OUTOFRANGE;
        // .5 * length * w_q * alpha, rounded as the reference writes it.
        speed = __dadd_rn(speed, __dmul_rn(__dmul_rn(__dmul_rn(0.5, len), t.gw[q]), a));
    }
    // d flux / d sample = -w kappa c_k / ds per sample (the last sample gets
    // -sum of the others' coefficients); interior samples k < 2 are the
    // left cell's, wall samples k < 4 all the wall cell's.
    double d0 = 0.0, d1 = 0.0;
    const int type = g.boundary ? pp.wall_type[g.wall] : MP_THERMAL_TEMPERATURE;
    if (type == MP_THERMAL_TEMPERATURE) {
        const double ds = t.dif_ds[o][g.boundary ? 1 : 0];
        double clast = 0.0;
#pragma unroll
        for (int k = 0; k < 3; ++k) clast -= t.dif_c_int[k];
#pragma unroll
        for (int q = 0; q < kNQ; ++q) {
            const double scale = -t.dif_w[o][q] * pp.kappa / ds;
            if (g.boundary) {
#pragma unroll
                for (int k = 0; k < 4; ++k) d0 += scale * t.dif_c_bnd[k];   // k = 4: the wall value
            } else {
                d0 += scale * t.dif_c_int[0];
                d0 += scale * t.dif_c_int[1];
                d1 += scale * t.dif_c_int[2];
                d1 += scale * clast;
            }
        }
    }
    const double d[2] = {d0, d1};
    rr[e] = (speed + fabs(d[0])) / area;
    rr[nE + e] = (speed + fabs(d[1])) / area;
    if (st) record_error(status, PART_FACES, e, st);
}

// Per-cell rate: the faces' shares in id order (bottom, top, left, right),
// the side of each face that this cell is; the last block keeps the maximum.
__global__ void __launch_bounds__(kPreBlock) pre_rate_cell_kernel(int nx, int ny, const double* __restrict__ rr,
                                                                   double* __restrict__ rate, PrePartial* partial,
                                                                   PreCtl* ctl) {
    const long long N = (long long)nx * ny;
    const long long nI = (long long)nx * (ny + 1), nE = nI + (long long)(nx + 1) * ny;
    PrePartial v = pre_identity();
#pragma unroll
    for (int k = 0; k < kPrePer; ++k) {
        const long long cell = (long long)blockIdx.x * kPreCells + k * kPreBlock + threadIdx.x;
        if (cell >= N) continue;
        const int i = (int)(cell % nx), j = (int)(cell / nx);
        const long long eb = (long long)j * nx + i, et = eb + nx;
        const long long el = nI + (long long)j * (nx + 1) + i, er = el + 1;
        double r = 0.0;
        r = __dadd_rn(r, __ldg(rr + eb));
        r = __dadd_rn(r, __ldg(rr + (j == ny - 1 ? 0 : nE) + et));
        r = __dadd_rn(r, __ldg(rr + (i == 0 ? 0 : nE) + el));
        r = __dadd_rn(r, __ldg(rr + er));
        rate[cell] = r;
        v.maximum = fmax(v.maximum, r);
        v.nonfinite = fmax(v.nonfinite, isfinite(r) ? 0.0 : 1.0);
    }
    PrePartial tot;
    if (pre_finish_blocks(v, partial, ctl, tot) && threadIdx.x == 0) ctl->last = tot;
}

// Diagnostics (preheat.cpp:202-233): the unlimited reconstructions of H and C
// and the 5x5 quadrature of the phase's T and phi.
__global__ void __launch_bounds__(128) pre_diag_kernel(int nx, int ny, const double* __restrict__ H,
                                                       const double* __restrict__ C, double* __restrict__ T,
                                                       double* __restrict__ phi, unsigned long long* status, Physics ph,
                                                       const __grid_constant__ ParamTables p) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= nx || j >= ny) return;
    const StageHot& t = p.d;
    const long long cell = (long long)j * nx + i;
    const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = j == 0 ? 0 : (j == ny - 1 ? 2 : 1);
    double D[2][9];
    double m[2];
    int st = 0;
    for (int f = 0; f < 2; ++f) {
        const double* F = f ? C : H;
        double u[3][3];
        for (int dj = 0; dj < 3; ++dj)
            for (int di = 0; di < 3; ++di) {
                const int ii = min(max(i + di - 1, 0), nx - 1), jj = min(max(j + dj - 1, 0), ny - 1);
                u[dj][di] = __ldg(F + (size_t)jj * nx + ii);
            }
        m[f] = u[1][1];
        const int s = reconstruct(t, candidate_mask(ci, cj), u, D[f]);
        st = st ? st : s;
    }
    if (st) { record_error(status, PART_UPDATE, cell, st); return; }
    double Ts = 0.0, Ps = 0.0;
    for (int b = 0; b < kNQ; ++b) {
        double h0, h1, h2, c0, c1, c2;
        const double y = t.g[b];
        q2_row(D[0], y, h0, h1, h2);
        q2_row(D[1], y, c0, c1, c2);
        const double tep = tep_at(ph, height(t, j, y));
        for (int q = 0; q < kNQ; ++q) {
            const double x = t.g[q];
            PhaseLean pl;
            const int s = phase_stage_lean(ph.sk, m[0] + quad(h0, h1, h2, x), m[1] + quad(c0, c1, c2, x), tep, pl);
            if (s) { st = st ? st : s; continue; }
            const double w = t.cw[b * kNQ + q];
            Ts += w * pl.T;
            Ps += w * pl.phil;
        }
    }
    if (st) record_error(status, PART_CELLS, cell, st);
    T[cell] = Ts;
    phi[cell] = Ps;
}

// ------------------------------------------------- general quad mesh forms

// Per edge of a quad mesh, half its length and that times sum_q w_q / ds_q
// (ds: the normal-line spacing of each edge point), for pre_step_kernel.
__global__ void __launch_bounds__(128) pre_quad_edge_kernel(int nx, int ny, double* __restrict__ edge, QuadDev q) {
    const long long nE = (long long)nx * (ny + 1) + (long long)(nx + 1) * ny;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nE) return;
    const QuadEdge g = quad_edge(q, nx, ny, 0, ny, e);
    double len;
    P2 nrm;
    edge_geometry(g.a, g.b, len, nrm);
    double sum = 0.0;
    for (int k = 0; k < kNQ; ++k) sum += q.gw[k] / __ldg(q.sp + e * kNQ + k);
    edge[2 * e] = 0.5 * len;
    edge[2 * e + 1] = 0.5 * len * sum;
}

// Build (preheat.cpp:130-156) on a general quad mesh: per edge the LF speed
// sum_q L w_q alpha / 2 and the diffusion derivatives at zero samples per
// side; (speed + |derivative|) / area of the left [e] and right [NE + e] cell.
__global__ void __launch_bounds__(128) pre_quad_rate_edge_kernel(int nx, int ny, const double* __restrict__ vn,
                                                                 double* __restrict__ rr, unsigned long long* status,
                                                                 const __grid_constant__ PreheatPhys pp, QuadDev q) {
    const long long nE = (long long)nx * (ny + 1) + (long long)(nx + 1) * ny;
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nE) return;
    const size_t N = (size_t)nx * ny;
    const QuadEdge g = quad_edge(q, nx, ny, 0, ny, e);
    double len;
    P2 nrm;
    edge_geometry(g.a, g.b, len, nrm);
    int st = 0;
    double speed = 0.0;
#pragma unroll
    for (int k = 0; k < kNQ; ++k) {
        const int cq = g.reverse ? kNQ - 1 - k : k;
        const double v = __ldg(vn + e * kNQ + cq);
        const double ns = fabs(v);
        if (!isfinite(v)) st = E_OUTOFRANGE;
        const double a = pp.lf_global ? pp.lf_speed : ns;
        if (!(a + 1e-14 >= ns)) st = E_OUTOFRANGE;
        speed = __dadd_rn(speed, __dmul_rn(__dmul_rn(__dmul_rn(0.5, len), q.gw[k]), a));
    }
    double d0 = 0.0, d1 = 0.0;
    const int type = g.boundary ? pp.wall_type[g.wall] : MP_THERMAL_TEMPERATURE;
    if (type == MP_THERMAL_TEMPERATURE) {
        double clast = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) clast -= q.dif_c_int[c];
#pragma unroll
        for (int k = 0; k < kNQ; ++k) {
            const int cq = g.reverse ? kNQ - 1 - k : k;
            const double sp = __ldg(q.sp + e * kNQ + cq);
            const double scale = -(len * q.gw[k] / 2) * pp.kappa / sp;
            if (g.boundary) {
#pragma unroll
                for (int c = 0; c < 4; ++c) d0 += scale * q.dif_c_bnd[c];
            } else {
                d0 += scale * q.dif_c_int[0];
                d0 += scale * q.dif_c_int[1];
                d1 += scale * q.dif_c_int[2];
                d1 += scale * clast;
            }
        }
    }
    const double aL = __ldg(q.geo + 3 * N + g.L), aR = g.boundary ? aL : __ldg(q.geo + 3 * N + g.R);
    rr[e] = (speed + fabs(d0)) / aL;
    rr[nE + e] = (speed + fabs(d1)) / aR;
    if (st) record_error(status, PART_FACES, e, st);
}

// Diagnostics (preheat.cpp:202-233) on a general quad mesh: the unlimited
// reconstructions of H and C and the 5x5 quadrature of T and phi on the
// bilinear map, weights w_a w_b J / area.
__global__ void __launch_bounds__(128) pre_quad_diag_kernel(int nx, int ny, const double* __restrict__ H,
                                                            const double* __restrict__ C, double* __restrict__ T,
                                                            double* __restrict__ phi, unsigned long long* status,
                                                            Physics ph, QuadDev q) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= nx || j >= ny) return;
    const long long cell = (long long)j * nx + i;
    const size_t N = (size_t)nx * ny;
    const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = j == 0 ? 0 : (j == ny - 1 ? 2 : 1);
    const CellFrame f = cell_frame(q, nx, N, cell);
    const double eA = 1e-2 * f.area;
    double u[2][3][3];
    for (int dj = 0; dj < 3; ++dj)
        for (int di = 0; di < 3; ++di) {
            const int ii = min(max(i + di - 1, 0), nx - 1), jj = min(max(j + dj - 1, 0), ny - 1);
            u[0][dj][di] = __ldg(H + (size_t)jj * nx + ii);
            u[1][dj][di] = __ldg(C + (size_t)jj * nx + ii);
        }
    const double m[2] = {u[0][1][1], u[1][1][1]};
    double D[2][9];
    int st = reconstruct_quad<2>(q, N, cell, ci, cj, eA, u, D);
    if (st) { record_error(status, PART_UPDATE, cell, st); return; }
    double Ts = 0.0, Ps = 0.0;
    for (int b = 0; b < kNQ; ++b)
        for (int a = 0; a < kNQ; ++a) {
            const P2 p = bilinear(q.gq[a], q.gq[b], f.c);
            const double x = (p.x - f.cx) * f.inv_h, y = (p.y - f.cy) * f.inv_h;
            const double tep = ph.litho ? tep_at(ph, p.y) : ph.Tep;
            PhaseLean pl;
            const int s = phase_stage_lean(ph.sk, m[0] + q2v(D[0], x, y), m[1] + q2v(D[1], x, y), tep, pl);
            if (s) { st = st ? st : s; continue; }
            const double w = q.gw[a] * q.gw[b] * jacobian(q.gq[a], q.gq[b], f.c) / f.area;
            Ts += w * pl.T;
            Ps += w * pl.phil;
        }
    if (st) record_error(status, PART_CELLS, cell, st);
    T[cell] = Ts;
    phi[cell] = Ps;
}

}  // namespace
}  // namespace mp

// -------------------------------------------------------------------- handle

struct mp_preheat {
    mp_mesh_desc mesh;
    mp_preheat_opts opts;
    mp_derived der;
    mp::Physics ph;                 // phase constants and pressure model (diagnostics)
    mp::PreheatPhys pp;
    cudaStream_t stream = nullptr;
    int nx = 0, ny = 0;
    size_t N = 0, NE = 0;
    mp::StageTables host_tab;
    mp::ParamTables ptab;
    double* Hb[2] = {nullptr, nullptr};   // state ping-pong; Hb[cur] is accepted
    int cur = 0;
    double *C = nullptr, *vn = nullptr, *edge = nullptr, *rr = nullptr, *rate = nullptr;
    double *rhs = nullptr, *T = nullptr, *phi = nullptr;
    mp::PrePartial* partial = nullptr;
    mp::PreCtl* ctl = nullptr;
    mp::PreRow* rows = nullptr;     // kBatch rows
    mp::PreCtl* h_ctl = nullptr;    // pinned mirrors
    mp::PreRow* h_rows = nullptr;
    unsigned long long* d_status = nullptr;   // two words (halted)
    unsigned long long* h_status = nullptr;
    int blocks = 0;                 // of the per-cell kernels
    int passes = 1;                 // row groups per block of pre_step_kernel
    double time = 0.0;
    long long accepted = 0;
    long long steps = 0;            // steps of the current run
    bool ready = false;             // begin() done for the current state
    double rate_max = 0.0, limit = 0.0;
    unsigned int acc_seen = 0;      // ctl->accepted after the last batch
    // General quad mesh (mp_preheat_create_quads): per-cell tables in HBM.
    bool quad = false;
    mp::QuadDev qdev{};
    double* qbuf = nullptr;         // one allocation holding every table
};

namespace mp {
namespace {

constexpr int kBatch = 512;         // steps issued per host round trip

void pre_free(mp_preheat* p) {
    void* bufs[] = {p->Hb[0], p->Hb[1], p->C, p->vn, p->edge, p->rr, p->rate, p->rhs, p->T, p->phi,
                    p->partial, p->ctl, p->rows, p->d_status, p->qbuf};
    for (void* b : bufs) if (b) cudaFree(b);
    if (p->h_ctl) cudaFreeHost(p->h_ctl);
    if (p->h_rows) cudaFreeHost(p->h_rows);
    if (p->h_status) cudaFreeHost(p->h_status);
}

mp_status pre_status(mp_preheat* p, const char* where) {
    const unsigned long long v = *p->h_status;
    if (v == ~0ULL) return MP_OK;
    const int part = (int)(v >> 56);
    const long long at = (long long)((v >> 8) & ((1ULL << 48) - 1));
    const int code = (int)(v & 0xff);
    const char* what = code == MP_ERR_PLIB ? "Preheat heat balance failed; candidate rejected"
                     : code == MP_ERR_FP ? (part == PART_CELLS ? "Nonfinite preheat candidate rejected"
                                                               : "non-finite reconstruction or flux")
                     : code == MP_ERR_ARG_OUTOFRANGE ? "non-finite trace or velocity, backflow on an outflow-only "
                                                       "wall, or a global LF speed below a normal speed"
                     : "phase evaluation failed";
    set_error("%s: %s %lld: %s", where, part == PART_FACES ? "edge" : "cell", at, what);
    return (mp_status)code;
}

mp_status reset_status(mp_preheat* p) {
    MP_CUDA(cudaMemsetAsync(p->d_status, 0xff, 2 * sizeof(unsigned long long), p->stream));
    return MP_OK;
}

mp_status read_status(mp_preheat* p) {
    MP_CUDA(cudaMemcpyAsync(p->h_status, p->d_status, sizeof(unsigned long long), cudaMemcpyDeviceToHost, p->stream));
    MP_CUDA(cudaMemcpyAsync(p->h_ctl, p->ctl, sizeof(PreCtl), cudaMemcpyDeviceToHost, p->stream));
    MP_CUDA(cudaStreamSynchronize(p->stream));
    return MP_OK;
}

// Blocks of one pre_step_kernel launch.
dim3 step_grid(int nx, int ny, int passes) {
    const int rows = passes * kStepRows - 2;
    return dim3((nx + kStepCols - 1) / kStepCols, (ny + rows - 1) / rows);
}

// Row groups per block: each block repeats two rows of its neighbours, so long
// blocks waste less, but they have to fill the GPU. Waves of resident blocks
// times the groups of each (and one for a block's start and end) is the time of
// a launch; the smallest is taken, the shorter blocks of two that are equal.
mp_status choose_passes(mp_preheat* p) {
    int sms = 0, resident = 0, dev = 0;
    MP_CUDA(cudaGetDevice(&dev));
    MP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    MP_CUDA(p->quad ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, pre_step_kernel<true, QuadDev>, kStepBlock, 0)
                    : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, pre_step_kernel<false, ParamTables>,
                                                                    kStepBlock, 0));
    const long long slots = (long long)sms * std::max(resident, 1);
    long long best = -1;
    for (int n = 1; n <= kStepPasses; ++n) {
        const dim3 g = step_grid(p->nx, p->ny, n);
        if (g.y > 65535) continue;
        const long long cost = ((long long)g.x * g.y + slots - 1) / slots * (n + 1);
        if (best < 0 || cost < best) { best = cost; p->passes = n; }
    }
    return MP_OK;
}

// One RHS evaluation / step on the state H.
void launch_step(mp_preheat* p, const double* H, double* Hout, int mode, double dt, int row) {
    PreStepArgs a{};
    a.nx = p->nx; a.ny = p->ny; a.passes = p->passes; a.mode = mode; a.row = row;
    a.dt = dt;
    a.H = H; a.vn = p->vn; a.edge = p->edge;
    a.Hout = Hout; a.rhs = p->rhs;
    a.rows = p->rows; a.partial = p->partial; a.ctl = p->ctl; a.status = p->d_status;
    const dim3 grid = step_grid(p->nx, p->ny, p->passes);
    if (p->quad) pre_step_kernel<true><<<grid, kStepBlock, 0, p->stream>>>(a, p->pp, p->qdev);
    else pre_step_kernel<false><<<grid, kStepBlock, 0, p->stream>>>(a, p->pp, p->ptab);
    count_launch();
}

// Step plan of Run (preheat.cpp:256-265): dt of the next step from the
// controls, or a failure status.
mp_status plan_step(const mp_preheat* p, double time, long long steps, double& dt, double& next) {
    const mp_preheat_opts& o = p->opts;
    if (steps >= o.max_steps) { set_error("maximum_steps reached before time.end"); return MP_ERR_NOT_CONVERGED; }
    const double remaining = o.end - time;
    dt = o.control == MP_TIME_FIXED ? o.dt_initial : std::min(o.dt_max, p->limit);
    if (o.control == MP_TIME_CFL && steps == 0) dt = std::min(dt, o.dt_initial);
    dt = std::min(dt, remaining);
    const double roundoff = 8 * std::numeric_limits<double>::epsilon() *
                            std::max({std::fabs(o.end), std::fabs(time), dt});
    if (remaining - dt <= roundoff) dt = remaining;
    if (!(dt <= p->limit * (1 + 1e-12))) {
        set_error("Requested step %g exceeds advection/diffusion limit %g; reduce step or use control: cfl", dt, p->limit);
        return MP_ERR_ARG_OUTOFRANGE;
    }
    if (!(dt >= o.dt_min || dt == remaining)) { set_error("Stable step is below time.step.minimum"); return MP_ERR_ARG_OUTOFRANGE; }
    if (!(time + dt > time && std::isfinite(dt))) { set_error("Time step does not advance finite time"); return MP_ERR_FP; }
    next = dt == remaining ? o.end : time + dt;
    return MP_OK;
}

}  // namespace
}  // namespace mp

// -------------------------------------------------------------------- C ABI

namespace {
mp_status preheat_create_impl(const mp_mesh_desc* mesh, const double* xy, const mp_preheat_opts* opts,
                              mp_stream_t stream, mp_preheat** out) {
    using namespace mp;
    if (!mesh || !opts || !out) { set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (mesh->nx < 2 || mesh->ny < 2) { set_error("Preheat requires at least 2x2 cells"); return MP_ERR_ARG_SIZ; }
    if (mesh_too_large(mesh->nx, mesh->ny)) { set_error("mesh has 2^31 edges or more"); return MP_ERR_ARG_SIZ; }
    if (!(opts->cfl > 0 && opts->cfl <= 1)) { set_error("Explicit preheat requires time.step.cfl <= 1"); return MP_ERR_ARG_OUTOFRANGE; }
    if (opts->control != MP_TIME_CFL && opts->control != MP_TIME_FIXED) { set_error("unknown time control"); return MP_ERR_ARG_OUTOFRANGE; }
    if (!(std::isfinite(opts->end) && opts->dt_initial > 0 && opts->dt_max > 0 && opts->dt_min >= 0 && opts->max_steps >= 0)) {
        set_error("time controls must be finite and positive");
        return MP_ERR_ARG_OUTOFRANGE;
    }
    if (!(std::isfinite(opts->diffusivity) && opts->diffusivity >= 0.0)) { set_error("Diffusivity must be finite and nonnegative"); return MP_ERR_ARG_OUTOFRANGE; }
    if (opts->H_policy < 0 || opts->H_policy > 2 || !std::isfinite(opts->inflow_H)) { set_error("unknown boundary policy"); return MP_ERR_ARG_OUTOFRANGE; }
    if (opts->lf_global && !(std::isfinite(opts->lf_global_speed) && opts->lf_global_speed >= 0)) {
        set_error("Global LF speed must be finite and nonnegative");
        return MP_ERR_ARG_OUTOFRANGE;
    }
    for (int w = 0; w < 4; ++w)
        if (opts->thermal_type[w] < 0 || opts->thermal_type[w] > 2 || !std::isfinite(opts->thermal_value[w])) {
            set_error("thermal condition of wall %d: unknown type or non-finite value", w);
            return MP_ERR_ARG_OUTOFRANGE;
        }
    mp_derived der;
    MP_TRY(derive_checked(opts->material, der));
    QuadTables qt;
    if (xy) {
        long long bad = -1;
        if (validate_quads(mesh->nx, mesh->ny, xy, &bad)) {
            set_error("Mesh has non-real/non-finite coordinates or an inverted, degenerate, or nearly singular "
                      "quadrilateral (cell %lld)", bad);
            return MP_ERR_ARG_WRONG;
        }
        // Vertices and edge spacing on the host; the per-cell tables are
        // built on the GPU below.
        const int qs = build_quad_tables(mesh->nx, mesh->ny, xy, 0, qt, 0, mesh->ny, false);
        if (qs) { set_error("per-cell stencil table construction failed"); return (mp_status)qs; }
    }
    mp_preheat* p = new mp_preheat;
    p->mesh = *mesh; p->opts = *opts; p->der = der;
    p->stream = (cudaStream_t)stream;
    p->nx = mesh->nx; p->ny = mesh->ny;
    p->N = (size_t)p->nx * p->ny;
    p->NE = (size_t)p->nx * (p->ny + 1) + (size_t)(p->nx + 1) * p->ny;
    Physics& ph = p->ph;
    ph = Physics{};
    ph.k = phase_const(opts->material, der);
    ph.sk = stage_const(ph.k);
    if (opts->pressure_model == MP_PRESSURE_CONSTANT) {
        double Tep;
        if (!(opts->pressure >= 0) || eutectic_temperature(ph.k, opts->pressure, Tep)) {
            delete p; set_error("pressure must be finite and nonnegative"); return MP_ERR_ARG_OUTOFRANGE;
        }
        ph.Tep = Tep;
        ph.litho = 0;
    } else if (opts->pressure_model == MP_PRESSURE_LITHOSTATIC) {
        if (!(std::isfinite(opts->pressure) && opts->pressure >= mesh->y1)) {
            delete p; set_error("surface_y must be at or above the mesh top"); return MP_ERR_ARG_OUTOFRANGE;
        }
        const long double b = (long double)opts->material.rho * opts->material.g * der.l0 / opts->material.nu / der.dT;
        ph.litho = 1; ph.tep_a = der.TDe0; ph.tep_b = (double)b; ph.surface = opts->pressure;
    } else {
        delete p; set_error("unknown pressure model"); return MP_ERR_ARG_OUTOFRANGE;
    }
    PreheatPhys& pp = p->pp;
    pp.kappa = opts->diffusivity;
    pp.diffusion = opts->diffusivity > 0.0;
    for (int w = 0; w < 4; ++w) {
        pp.wall_type[w] = opts->thermal_type[w];
        pp.wall_value[w] = opts->thermal_type[w] == MP_THERMAL_ZERO_FLUX ? 0.0 : opts->thermal_value[w];
        if (opts->thermal_type[w] == MP_THERMAL_FLUX) pp.diffusion = 1;
    }
    pp.Hpol = opts->H_policy; pp.inflowH = opts->inflow_H;
    pp.lf_global = opts->lf_global; pp.lf_speed = opts->lf_global_speed;
    if (!xy) {
        const int tb = build_stage_tables(mesh->nx, mesh->ny, mesh->x0, mesh->x1, mesh->y0, mesh->y1, p->host_tab);
        if (tb) { delete p; set_error("stencil table construction failed"); return (mp_status)tb; }
        make_param_tables(p->host_tab, p->ptab);
    }
    p->blocks = (int)((p->N + kPreCells - 1) / kPreCells);
    p->quad = xy != nullptr;
    const double* ci = xy ? qt.dif_c_int : p->host_tab.dif_c_int;
    const double* cb = xy ? qt.dif_c_bnd : p->host_tab.dif_c_bnd;
    pp.c_int = ci[0] + ci[1];
    pp.c_bnd = cb[0] + cb[1] + cb[2] + cb[3];
    if (!xy)
        for (int o = 0; o < 2; ++o) {
            double w = 0.0;
            for (int q = 0; q < kNQ; ++q) w += p->host_tab.dif_w[o][q];
            pp.dif[o][0] = -pp.kappa * pp.c_int * w / p->host_tab.dif_ds[o][0];
            pp.dif[o][1] = -pp.kappa * pp.c_bnd * w / p->host_tab.dif_ds[o][1];
        }
    pp.inv_area = xy ? 0.0 : 1.0 / p->host_tab.area;
    const mp_status ps = choose_passes(p);
    if (ps != MP_OK) { delete p; return ps; }
    const dim3 grid = step_grid(p->nx, p->ny, p->passes);
    const size_t N = p->N, NE = p->NE, blocks = std::max((size_t)p->blocks, (size_t)grid.x * grid.y);
    cudaError_t e = cudaSuccess;
    auto alloc = [&](void** q, size_t bytes) { if (e == cudaSuccess) e = cudaMalloc(q, bytes); };
    for (double** q : {&p->Hb[0], &p->Hb[1], &p->C, &p->rate, &p->rhs, &p->T, &p->phi}) alloc((void**)q, N * sizeof(double));
    alloc((void**)&p->vn, NE * kNQ * sizeof(double));
    if (xy) alloc((void**)&p->edge, 2 * NE * sizeof(double));
    alloc((void**)&p->rr, 2 * NE * sizeof(double));
    alloc((void**)&p->partial, blocks * sizeof(PrePartial));
    alloc((void**)&p->ctl, sizeof(PreCtl));
    alloc((void**)&p->rows, kBatch * sizeof(PreRow));
    alloc((void**)&p->d_status, 2 * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMallocHost((void**)&p->h_ctl, sizeof(PreCtl));
    if (e == cudaSuccess) e = cudaMallocHost((void**)&p->h_rows, kBatch * sizeof(PreRow));
    if (e == cudaSuccess) e = cudaMallocHost((void**)&p->h_status, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemsetAsync(p->vn, 0, NE * kNQ * sizeof(double), p->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(p->ctl, 0, sizeof(PreCtl), p->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(p->d_status, 0xff, 2 * sizeof(unsigned long long), p->stream);
    if (xy && e == cudaSuccess) {
        const int gs = upload_quad_tables(p->nx, p->ny, xy, qt, 0, p->ny, p->stream, &p->qbuf, p->qdev, &e);
        if (gs == MP_ERR_ARG_WRONG) {
            pre_free(p); delete p;
            set_error("per-cell stencil table construction failed (singular stencil or degenerate cell)");
            return (mp_status)gs;
        }
        if (e == cudaSuccess) {
            pre_quad_edge_kernel<<<(unsigned)((NE + 127) / 128), 128, 0, p->stream>>>(p->nx, p->ny, p->edge, p->qdev);
            count_launch();
            e = cudaGetLastError();
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(p->stream);
    if (e != cudaSuccess) { pre_free(p); delete p; return cuda_status(e, "mp_preheat_create"); }
    *out = p;
    return MP_OK;
}
}  // namespace

extern "C" mp_status mp_preheat_create(const mp_mesh_desc* mesh, const mp_preheat_opts* opts, mp_stream_t stream,
                                       mp_preheat** out) {
    return preheat_create_impl(mesh, nullptr, opts, stream, out);
}

extern "C" mp_status mp_preheat_create_quads(const mp_mesh_desc* mesh, const double* xy, const mp_preheat_opts* opts,
                                             mp_stream_t stream, mp_preheat** out) {
    if (!xy) { mp::set_error("null vertex array"); return MP_ERR_ARG_WRONG; }
    return preheat_create_impl(mesh, xy, opts, stream, out);
}

extern "C" void mp_preheat_destroy(mp_preheat* p) {
    if (!p) return;
    cudaStreamSynchronize(p->stream);
    mp::pre_free(p);
    delete p;
}

extern "C" mp_status mp_preheat_set_velocity(mp_preheat* p, const double* vn) {
    if (!p || !vn) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    MP_CUDA(cudaMemcpyAsync(p->vn, vn, p->NE * mp::kNQ * sizeof(double), cudaMemcpyDefault, p->stream));
    MP_CUDA(cudaStreamSynchronize(p->stream));
    p->ready = false;
    return MP_OK;
}

extern "C" mp_status mp_preheat_set_state(mp_preheat* p, const double* H, const double* C, double time,
                                          long long accepted) {
    if (!p || !H || !C) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (!std::isfinite(time)) { mp::set_error("Nonfinite source time"); return MP_ERR_ARG_OUTOFRANGE; }
    MP_CUDA(cudaMemcpyAsync(p->Hb[0], H, p->N * sizeof(double), cudaMemcpyDefault, p->stream));
    MP_CUDA(cudaMemcpyAsync(p->C, C, p->N * sizeof(double), cudaMemcpyDefault, p->stream));
    MP_CUDA(cudaStreamSynchronize(p->stream));
    p->cur = 0;
    p->time = time;
    p->accepted = accepted;
    p->steps = 0;
    p->ready = false;
    return MP_OK;
}

extern "C" mp_status mp_preheat_get_state(mp_preheat* p, double* H, double* time, long long* accepted) {
    if (!p) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (H) {
        MP_CUDA(cudaMemcpyAsync(H, p->Hb[p->cur], p->N * sizeof(double), cudaMemcpyDefault, p->stream));
        MP_CUDA(cudaStreamSynchronize(p->stream));
    }
    if (time) *time = p->time;
    if (accepted) *accepted = p->accepted;
    return MP_OK;
}

extern "C" mp_status mp_preheat_begin(mp_preheat* p, double* rate, double* limit, mp_preheat_step* first) {
    using namespace mp;
    if (!p) { set_error("null argument"); return MP_ERR_ARG_WRONG; }
    p->ready = false;
    if (!(p->time <= p->opts.end)) { set_error("State time exceeds time.end"); return MP_ERR_ARG_OUTOFRANGE; }
    MP_TRY(reset_status(p));
    if (p->quad)
        pre_quad_rate_edge_kernel<<<(unsigned)((p->NE + 127) / 128), 128, 0, p->stream>>>(p->nx, p->ny, p->vn, p->rr,
                                                                                          p->d_status, p->pp, p->qdev);
    else
        pre_rate_edge_kernel<<<(unsigned)((p->NE + 127) / 128), 128, 0, p->stream>>>(p->nx, p->ny, p->host_tab.area,
                                                                                     p->vn, p->rr, p->d_status, p->pp,
                                                                                     p->ptab);
    pre_rate_cell_kernel<<<p->blocks, kPreBlock, 0, p->stream>>>(p->nx, p->ny, p->rr, p->rate, p->partial, p->ctl);
    count_launch(2);
    MP_CUDA(cudaGetLastError());
    MP_TRY(read_status(p));
    MP_TRY(pre_status(p, "mp_preheat_begin"));
    const PrePartial rt = p->h_ctl->last;
    if (rt.nonfinite != 0.0) { set_error("Nonfinite preheat rate"); return MP_ERR_FP; }
    p->rate_max = rt.maximum;
    p->limit = p->rate_max > 0 ? p->opts.cfl / p->rate_max : p->opts.dt_max;
    // Integral, minimum and maximum of the initial H (preheat.cpp:245-249).
    pre_measure_kernel<<<p->blocks, kPreBlock, 0, p->stream>>>((long long)p->N, p->quad ? 0.0 : p->host_tab.area,
                                                               p->quad ? p->qdev.geo + 3 * p->N : nullptr,
                                                               p->Hb[p->cur], p->partial, p->ctl);
    count_launch();
    MP_CUDA(cudaGetLastError());
    MP_TRY(read_status(p));
    const PrePartial m = p->h_ctl->last;
    MP_CUDA(cudaMemcpyAsync(&p->ctl->prev_integral, &m.integral, sizeof(double), cudaMemcpyHostToDevice, p->stream));
    if (rate) MP_CUDA(cudaMemcpyAsync(rate, p->rate, p->N * sizeof(double), cudaMemcpyDefault, p->stream));
    MP_CUDA(cudaStreamSynchronize(p->stream));
    p->acc_seen = p->h_ctl->accepted;
    p->steps = 0;
    p->ready = true;
    if (limit) *limit = p->limit;
    if (first) {
        *first = mp_preheat_step{};
        first->step = p->accepted; first->time = p->time; first->integral = m.integral;
        first->minimum = m.minimum; first->maximum = m.maximum;
    }
    return MP_OK;
}

extern "C" mp_status mp_preheat_rhs(mp_preheat* p, double* rhs, double* boundary_flux) {
    using namespace mp;
    if (!p) { set_error("null argument"); return MP_ERR_ARG_WRONG; }
    MP_TRY(reset_status(p));
    const double* H = p->Hb[p->cur];
    launch_step(p, H, nullptr, PRE_RHS, 0.0, 0);
    MP_CUDA(cudaGetLastError());
    MP_TRY(read_status(p));
    MP_TRY(pre_status(p, "mp_preheat_rhs"));
    if (rhs) {
        MP_CUDA(cudaMemcpyAsync(rhs, p->rhs, p->N * sizeof(double), cudaMemcpyDefault, p->stream));
        MP_CUDA(cudaStreamSynchronize(p->stream));
    }
    if (boundary_flux) *boundary_flux = p->h_ctl->last.bflux;
    return MP_OK;
}

extern "C" mp_status mp_preheat_advance(mp_preheat* p, long long nsteps, mp_preheat_step* rows, long long* taken) {
    mp::NvtxRange range("mp_preheat advance");
    using namespace mp;
    if (taken) *taken = 0;
    if (!p) { set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (!p->ready) { set_error("call mp_preheat_begin after setting the state and velocity"); return MP_ERR_ARG_WRONGSTATE; }
    long long done = 0;
    while (done < nsteps && p->time < p->opts.end) {
        // Plan a batch: dt and the time after each step.
        double dts[kBatch], times[kBatch];
        int n = 0;
        mp_status plan = MP_OK;
        double t = p->time;
        while (n < kBatch && done + n < nsteps && t < p->opts.end) {
            double dt, next;
            plan = plan_step(p, t, p->steps + n, dt, next);
            if (plan != MP_OK) break;
            dts[n] = dt; times[n] = next; t = next; ++n;
        }
        if (n > 0) {
            MP_TRY(reset_status(p));
            for (int k = 0; k < n; ++k) {
                const double* H = p->Hb[(p->cur + k) & 1];
                double* Hn = p->Hb[(p->cur + k + 1) & 1];
                launch_step(p, H, Hn, PRE_STEP, dts[k], k);
            }
            MP_CUDA(cudaGetLastError());
            MP_CUDA(cudaMemcpyAsync(p->h_rows, p->rows, (size_t)n * sizeof(PreRow), cudaMemcpyDeviceToHost, p->stream));
            MP_TRY(read_status(p));
            const int m = (int)(p->h_ctl->accepted - p->acc_seen);
            p->acc_seen = p->h_ctl->accepted;
            for (int k = 0; k < m; ++k) {
                const PreRow& r = p->h_rows[k];
                ++p->accepted; ++p->steps;
                p->time = times[k];
                if (rows) {
                    mp_preheat_step& o = rows[done + k];
                    o.step = p->accepted; o.time = times[k]; o.dt = dts[k]; o.courant = dts[k] * p->rate_max;
                    o.integral = r.integral; o.minimum = r.minimum; o.maximum = r.maximum;
                    o.boundaryFlux = r.bflux; o.balanceError = r.balance;
                }
            }
            p->cur = (p->cur + m) & 1;
            done += m;
            if (taken) *taken = done;
            if (m < n) {
                const mp_status s = pre_status(p, "mp_preheat_advance");
                if (s != MP_OK) return s;
                set_error("mp_preheat_advance: step %lld was not accepted", p->accepted + 1);
                return MP_ERR_PLIB;
            }
        }
        if (plan != MP_OK) return plan;
    }
    if (taken) *taken = done;
    return MP_OK;
}

extern "C" mp_status mp_preheat_diagnostics(mp_preheat* p, double* T, double* phi) {
    using namespace mp;
    if (!p) { set_error("null argument"); return MP_ERR_ARG_WRONG; }
    MP_TRY(reset_status(p));
    dim3 blk(32, 4), grd((p->nx + 31) / 32, (p->ny + 3) / 4);
    if (p->quad)
        pre_quad_diag_kernel<<<grd, blk, 0, p->stream>>>(p->nx, p->ny, p->Hb[p->cur], p->C, p->T, p->phi, p->d_status,
                                                         p->ph, p->qdev);
    else
        pre_diag_kernel<<<grd, blk, 0, p->stream>>>(p->nx, p->ny, p->Hb[p->cur], p->C, p->T, p->phi, p->d_status,
                                                    p->ph, p->ptab);
    count_launch();
    MP_CUDA(cudaGetLastError());
    MP_TRY(read_status(p));
    MP_TRY(pre_status(p, "mp_preheat_diagnostics"));
    if (T) MP_CUDA(cudaMemcpyAsync(T, p->T, p->N * sizeof(double), cudaMemcpyDefault, p->stream));
    if (phi) MP_CUDA(cudaMemcpyAsync(phi, p->phi, p->N * sizeof(double), cudaMemcpyDefault, p->stream));
    MP_CUDA(cudaStreamSynchronize(p->stream));
    return MP_OK;
}

extern "C" mp_status mp_preheat_run(mp_preheat* p, mp_preheat_report* report, mp_preheat_step* history,
                                    long long capacity, long long* rows, double* T, double* phi) {
    if (rows) *rows = 0;
    if (!p) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    mp_preheat_step first;
    double limit;
    MP_TRY(mp_preheat_begin(p, nullptr, &limit, &first));
    mp_preheat_report rep{};
    rep.initialTime = rep.finalTime = p->time;
    rep.stepLimit = limit;
    rep.initialIntegral = rep.finalIntegral = first.integral;
    long long count = 0;
    if (history && capacity > 0) history[0] = first;
    count = 1;
    std::vector<mp_preheat_step> chunk(mp::kBatch);
    mp_status s = MP_OK;
    while (p->time < p->opts.end) {
        long long got = 0;
        s = mp_preheat_advance(p, mp::kBatch, chunk.data(), &got);
        for (long long k = 0; k < got; ++k) {
            if (history && count < capacity) history[count] = chunk[k];
            ++count;
            rep.finalIntegral = chunk[k].integral;
            rep.boundaryIntegral += chunk[k].dt * chunk[k].boundaryFlux;
        }
        rep.finalTime = p->time;
        if (s != MP_OK || got == 0) break;
    }
    if (rows) *rows = count;
    if (report) *report = rep;
    if (s != MP_OK) return s;
    return mp_preheat_diagnostics(p, T, phi);
}
