// Per-element device functions of the transport stage, shared by the
// single-instance kernels (transport.cu) and the batched kernels (batch.cu).
//
// recon_cell      reconstruction, weights, limiter theta (one cell)
// cellphase_cell  5x5 phase quadrature of T, phi and the wet flag (one cell)
// face_edge       limited values, phase, porosity, LF flux and rate (one edge)
// sum_cell        reference-ordered accumulation and RK combination (one cell)
#ifndef MP_STAGE_KERNELS_CUH
#define MP_STAGE_KERNELS_CUH

#include <cuda_pipeline.h>

#include "common.hpp"
#include "phase_math.cuh"
#include "stage_device.cuh"
#include "tables.hpp"

// Load of an array that some phase of a stage writes: through the read-only
// path in kernels of one phase each, a plain load where one kernel runs every
// phase (small_steps.cu).
#ifndef MP_LD
#define MP_LD(p) __ldg(p)
#endif

namespace mp {
namespace {

constexpr int kRec = 18;          // limited deviation coefficients: 9 for H, 9 for C
// Records lie in groups of 32 cells, coefficient by coefficient: the 18 loads
// of a cell are one address and constant offsets, and a warp's record is one
// stretch of 4.6 KB.
constexpr int kRecStride = 32;
__host__ __device__ __forceinline__ size_t rec_doubles(size_t cells) { return (cells + 31) / 32 * (32 * kRec); }
__device__ __forceinline__ size_t rec_at(long long cell) {
    return (size_t)((unsigned)cell >> 5) * (32 * kRec) + ((unsigned)cell & 31u);
}
constexpr int kRedBlock = 256;
// The accumulation and axpy kernels give each thread several cells (strided by
// the block size, so loads stay coalesced) before one block reduction: as many
// as make one wave of 592 blocks, four on each of a B200's 148 SMs (at
// 640x1280 27 us; four cells and 1.35 waves 35), at least four, and one below kSumOne, where few blocks leave
// most of the GPU idle (61x127, one step with transfers: 311 us, four 323; a
// 40x80 quad mesh, four steps: 818, 863; a batch of 24 uneven meshes the
// same). A constant, so that the grouping, which fixes the order of the sums,
// is a function of the mesh alone.
constexpr int kSumPer = 4;
constexpr long long kSumOne = 16384, kSmallCells = 1536;   // kSmallCells: steps in one cluster (small_steps.cu)
static_assert(kSmallCells <= kSumOne, "the cluster's sums take one cell per thread");
__host__ __device__ __forceinline__ int sum_per(long long cells) {
    const long long wave = 592LL * kRedBlock, per = (cells + wave - 1) / wave;
    return cells <= kSumOne ? 1 : (int)(per > kSumPer ? per : kSumPer);
}
__host__ __device__ __forceinline__ int sum_cells_per_block(long long cells) { return kRedBlock * sum_per(cells); }

enum : int {
    E_OUTOFRANGE = MP_ERR_ARG_OUTOFRANGE, E_FP = MP_ERR_FP, E_WRONG = MP_ERR_ARG_WRONG
};

}  // namespace

struct Physics {
    PhaseConst k;
    StageConst sk;
    double Tep;            // pressure-corrected eutectic temperature (constant pressure)
    double theta;          // Darcy exponent
    double inflowH, inflowC;
    int Hpol, Cpol, lf_global;
    double lf_speed;
    // Thermal diffusion: on when kappa > 0 or a wall prescribes a flux.
    // Walls 0 bottom, 1 top, 2 left, 3 right: 0 zero flux, 1 prescribed
    // temperature, 2 prescribed outward flux (per unit length).
    int diffusion;
    double kappa;
    int wall_type[4];
    double wall_value[4];
    // Phase-law pressure: constant (litho = 0, Tep above), or lithostatic
    // rho g l0 (surface - y): Tep(y) = tep_a + tep_b (surface - y).
    int litho;
    double tep_a, tep_b, surface;
    // Adiabatic source -cooling T v_mix,y (evolve.cpp:359-369), cooling =
    // alpha0 l0 g / cp; on when alpha0 != 0.
    int source;
    double cooling;
};

namespace {

// Pressure-corrected eutectic temperature at height y (one FMA for the
// lithostatic model; the constant model returns the stored value exactly).
__device__ __forceinline__ double tep_at(const Physics& ph, double y) {
    return ph.litho ? fma(ph.tep_b, ph.surface - y, ph.tep_a) : ph.Tep;
}

// Height of a point at normalised eta in the cell of global row gj.
__device__ __forceinline__ double height(const StageHot& t, int gj, double eta) {
    return t.y0 + (gj + 0.5) * t.dy + eta * t.hn;
}

}  // namespace

// Block partials of one stage (sum_kernel) or state check (axpy_kernel).
struct Partial {
    double maxRate, divergence, bH, bC, HI, CI, Hmin, Cmin, Cmax;
    double nonfinite;
    double sH;             // adiabatic source integral
};

namespace {

__device__ __forceinline__ Partial partial_identity() {
    return Partial{-INFINITY, 0.0, 0.0, 0.0, 0.0, 0.0, INFINITY, INFINITY, -INFINITY, 0.0, 0.0};
}

}  // namespace

struct Totals {
    double maxRate, divergence, bH, bC, HI, CI, Hmin, Cmin, Cmax;
    double nonfinite;
    double sH;
};

namespace {

// Fold one block partial into a running partial (fixed field rules).
__device__ __forceinline__ void fold_partial(Partial& v, const Partial& p) {
    v.maxRate = fmax(v.maxRate, p.maxRate); v.divergence = fmax(v.divergence, p.divergence);
    v.bH += p.bH; v.bC += p.bC; v.HI += p.HI; v.CI += p.CI;
    v.Hmin = fmin(v.Hmin, p.Hmin); v.Cmin = fmin(v.Cmin, p.Cmin); v.Cmax = fmax(v.Cmax, p.Cmax);
    v.nonfinite = fmax(v.nonfinite, p.nonfinite);
    v.sH += p.sH;
}

// Row slabs of a decomposed mesh: the local arrays hold rows gj0 .. of a
// global mesh of gny rows (gny = 0: the local mesh is the whole mesh).
// Physical-boundary tests and error keys use global rows.
template <class A>
__device__ __forceinline__ int global_ny(const A& a) { return a.gny > 0 ? a.gny : a.ny; }

// Status word: the smallest key wins. The key orders failures as the
// reference's RHS meets them (evolve.cpp:279-384): reconstruction update,
// limiter, porosity sampling, face loop, cell quadrature; then by cell/edge.
enum : int { PART_UPDATE = 0, PART_LIMIT = 1, PART_POROSITY = 2, PART_FACES = 3, PART_CELLS = 4, PART_CHECK = 7 };
__device__ __forceinline__ void record_error(unsigned long long* status, int part, long long where, int code) {
    atomicMin(status, ((unsigned long long)part << 56) | ((unsigned long long)where << 8) | (unsigned long long)(code & 0xff));
}

// Bounds-checked build (MP_CHECKED, libmantlepar_b200_checked.so): every
// cell and edge index a stage element derives is checked against its array
// before use; one outside [0, n) records MP_ERR_ARG_OUTOFRANGE with part
// PART_CHECK and the index in the status word, and the element returns
// without touching memory. In the default build the check compiles away.
#ifdef MP_CHECKED
#define MP_CHECK_INDEX(status, idx, n)                                                        \
    do {                                                                                      \
        const long long mp_i_ = (long long)(idx);                                            \
        if (!(mp_i_ >= 0 && mp_i_ < (long long)(n))) {                                       \
            if (status) record_error((status), PART_CHECK, mp_i_ < 0 ? 0 : mp_i_, MP_ERR_ARG_OUTOFRANGE); \
            return;                                                                           \
        }                                                                                     \
    } while (0)
#else
#define MP_CHECK_INDEX(status, idx, n) \
    do {                               \
    } while (0)
#endif
// The same where the element may not return, as its warp shuffles or meets a
// barrier further on: an index outside [0, n) is recorded, `active` cleared and
// 0 taken in its place.
template <class T>
__device__ __forceinline__ T checked_index(unsigned long long* status, T idx, long long n, bool& active) {
#ifdef MP_CHECKED
    if (!(idx >= 0 && idx < n)) {
        if (status) record_error(status, PART_CHECK, idx < 0 ? 0 : idx, MP_ERR_ARG_OUTOFRANGE);
        active = false;
        return 0;
    }
#endif
    return idx;
}


// ------------------------------------------------------- reconstruction kernel

// Cell flags byte: bit 0 wet (porosity sampling), bit 1 exact diffusion-sample
// check needed (the cheap bound could not prove admissibility), bit 2 plain:
// every limited value of the cell is a plain phase point (phase_plain).
enum : unsigned char { FLAG_WET = 1, FLAG_CHECK = 2, FLAG_PLAIN = 4 };

// The flag byte of a cell from its neighbour bounds: the limiter keeps every
// limited value at the cell's points (cell and edge Gauss points, diffusion
// samples) within [lo, hi] up to roundoff, and Hliq at (hi_C, lowest tep) is
// the lowest liquidus, so bounds that keep a margin of 1e-12 of the field's
// largest value from the ends of the ranges prove each point's admissibility: the samples' (cell flagged otherwise: they are
// checked one by one), and for a plain cell all of them. Melt begins where H
// passes Tep, so with a constant pressure a plain cell is wet when topH, its
// largest limited enthalpy at the quadrature points, does (with a
// lithostatic pressure the quadrature decides).
__device__ __forceinline__ unsigned char cell_flags(const Physics& ph, double tep_lo, double tep_hi, double loH, double hiH,
                                                    double loC, double hiC, double topH) {
    const double Hliq = tep_lo + (1.0 - hiC * ph.sk.invXe) + ph.k.LD;
    const double slack = 1e-12 * (1.0 + fabs(hiH));
    if (!(tep_lo >= 0.0 && hiH + slack < Hliq)) return FLAG_CHECK;
    if (!(ph.sk.ordinary && tep_lo >= 1e-9 && tep_hi <= 1e100 && loH >= slack && loC >= 1e-90 + 1e-12 * hiC &&
          hiC <= ph.k.Xe * (1.0 - 1e-12)))
        return 0;
    return FLAG_PLAIN | (!ph.litho && topH > ph.Tep ? FLAG_WET : 0);
}

struct ReconArgs {
    int nx, ny;
    const StageHot* tab;   // batched instances: their tables in device memory
    const double* H;
    const double* C;
    double* rec;           // coefficient m of a cell at rec_at(cell) + m * kRecStride, m < 9 for H
    unsigned char* flags;
    unsigned long long* status;
    double* theta;         // optional (2 * ncell): limiter factors for H, C
    int gj0 = 0, gny = 0;  // slab: global row of local row 0, global rows
    const int* gate = nullptr;   // device flag: the launch does nothing while it is 0
};

// Max/min of the deviation polynomial over the class's limiter points by
// per-point evaluation with the finiteness check of every value. Used when
// the data are so large that a value could overflow.
__device__ __noinline__ void scan_lines_exact(const StageHot& t, int l0, int l1, const double* D, double& mx,
                                              double& mn, bool& bad) {
    double rmx = D[0], rmn = D[0];
    bad = bad || !isfinite(D[0]);
    for (int l = l0; l < l1; ++l) {
        double a0, a1, a2;
        if (t.line_dir[l] == 0) q2_row(D, t.line_c[l], a0, a1, a2);
        else q2_col(D, t.line_c[l], a0, a1, a2);
        for (int q = 0; q < kNQ; ++q) {
            const double v = quad(a0, a1, a2, t.g[q]);
            rmx = fmax(rmx, v); rmn = fmin(rmn, v);
            bad = bad || !isfinite(v);
        }
    }
    mx = rmx; mn = rmn;
}

// The nonnegative 5-point Gauss nodes on [-1, 1].
constexpr double kG1 = 0.538469310105683091036314420700, kG2 = 0.906179845938663992797626878299;

// Running extremes of the limiter scan.
struct Extremes {
    double mx, mn;
    __device__ __forceinline__ void up(double v) { mx = v > mx ? v : mx; }
    __device__ __forceinline__ void down(double v) { mn = v < mn ? v : mn; }
    // The two Gauss pairs s = +-g1, +-g2 of a line a0 + s (a1 + s a2): the
    // larger of a pair is (a0 + a2 s^2) + |a1| s, the smaller with the minus.
    __device__ __forceinline__ void pairs(double a0, double a1, double a2) {
        const double e1 = fma(a2, kG1 * kG1, a0), e2 = fma(a2, kG2 * kG2, a0), b = fabs(a1);
        up(fma(b, kG1, e1)); up(fma(b, kG2, e2));
        down(fma(-b, kG1, e1)); down(fma(-b, kG2, e2));
    }
    // A line and its centre.
    __device__ __forceinline__ void line(double a0, double a1, double a2) {
        up(a0); down(a0);
        pairs(a0, a1, a2);
    }
    // The lines at +c and -c of the coefficient rows (p0 + c p1 + c^2 p2) of
    // the three powers along the line; the two centres again as a pair.
    __device__ __forceinline__ void line_pair(double c, const double (&p0)[3], const double (&p1)[3],
                                              const double (&p2)[3]) {
        double e[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) e[k] = fma(p2[k], c * c, p0[k]);
        up(fma(fabs(p1[0]), c, e[0]));
        down(fma(-fabs(p1[0]), c, e[0]));
        pairs(fma(p1[0], c, e[0]), fma(p1[1], c, e[1]), fma(p1[2], c, e[2]));
        pairs(fma(p1[0], -c, e[0]), fma(p1[1], -c, e[1]), fma(p1[2], -c, e[2]));
    }
};

// The limiter points of a cell of boundary class (ci, cj)
// (state_reconstruction.cpp:152-168), five Gauss points on each of: the rows
// eta = 0, +-g1, +-g2 (cell quadrature) and +-1 (edges), the columns xi = +-1,
// and the diffusion samples' lines, 0.9 and 0.3 cell sizes from an interior
// edge (+-0.8, +-0.4) and 0.9, 0.675, 0.45 and 0.225 from a wall: there the
// 0.3 line gives way to three. The lines common to every cell are scanned as
// symmetric pairs and their points as symmetric pairs (85 points in 280 FP64
// operations, 84 of them comparisons); a wall adds its lines, so that a cell
// takes the same operations whatever its neighbours in the warp are.
// mq: the largest value at the 25 points of the cell quadrature.
__device__ __forceinline__ void scan_cell(const double (&D)[9], int ci, int cj, double& mx, double& mn, double& mq) {
    Extremes x{D[0], D[0]};
    x.pairs(D[0], D[1], D[2]);
    const double r0[3] = {D[0], D[1], D[2]}, r1[3] = {D[3], D[4], D[5]}, r2[3] = {D[6], D[7], D[8]};
    x.line_pair(kG1, r0, r1, r2);
    x.line_pair(kG2, r0, r1, r2);
    mq = x.mx;
    x.line_pair(0.8, r0, r1, r2);
    x.line_pair(1.0, r0, r1, r2);
    const double c0[3] = {D[0], D[3], D[6]}, c1[3] = {D[1], D[4], D[7]}, c2[3] = {D[2], D[5], D[8]};
    x.line_pair(0.8, c0, c1, c2);
    x.line_pair(1.0, c0, c1, c2);
    auto row = [&](double c) { double a0, a1, a2; q2_row(D, c, a0, a1, a2); x.line(a0, a1, a2); };
    auto col = [&](double c) { double a0, a1, a2; q2_col(D, c, a0, a1, a2); x.line(a0, a1, a2); };
    row(cj == 0 ? 0.35 : -0.4);
    row(cj == 2 ? -0.35 : 0.4);
    col(ci == 0 ? 0.35 : -0.4);
    col(ci == 2 ? -0.35 : 0.4);
    if (cj != 1) { const double s = cj == 0 ? 1.0 : -1.0; row(-0.1 * s); row(-0.55 * s); }
    if (ci != 1) { const double s = ci == 0 ? 1.0 : -1.0; col(-0.1 * s); col(-0.55 * s); }
    mx = x.mx; mn = x.mn;
}

// theta of one field: min over points of (bound - mean)/(v - mean) for v
// outside [lo, hi] (state_reconstruction.cpp:216-224). With v = mean + D and
// rounding monotone, the minimum is reached at the extreme D, so one
// division per bound gives the reference's value.
__device__ __forceinline__ double theta_of(double m, double lo, double hi, double dmax, double dmin) {
    auto ratio = [](double a, double b) { return rcp_range(b) ? div_normal(a, b) : a / b; };
    double th = 1.0;
    const double vmax = m + dmax, vmin = m + dmin;
    if (vmax > hi) th = fmin(th, ratio(hi - m, vmax - m));
    if (vmin < lo) th = fmin(th, ratio(lo - m, vmin - m));
    return th < 1.0 ? fmax(0.0, th * (1.0 - 1e-13)) : 1.0;
}

// Averages of this magnitude or more: a limiter value could overflow.
constexpr double kScanGuard = 1e30;

// One field of one cell: gather, neighbour bounds, reconstruction, limiter
// factor th and the unlimited D. top: the field's upper bound (Xe for the
// composition).
__device__ __forceinline__ void recon_field(const StageHot& t, const double* __restrict__ F, const unsigned (&at)[3][3],
                                            int ci, int cj, double top, double (&D)[9], double& mean, double& lo,
                                            double& hi, double& th, double& mq, int& st, bool& bad) {
    double u[3][3];
#pragma unroll
    for (int dj = 0; dj < 3; ++dj)
#pragma unroll
        for (int di = 0; di < 3; ++di) u[dj][di] = MP_LD(F + at[dj][di]);
    // 3x3 neighbour bounds (state_reconstruction.cpp:189-196); the clamped
    // gather repeats in-domain values, which leaves min/max unchanged.
    mean = lo = hi = u[1][1];
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
    hi = top < hi ? top : hi;
    const int s1 = reconstruct(t, candidate_mask(ci, cj), u, D);
    st = st ? st : s1;
    double mx, mn;
    if (!small) {
        // Copies, so that the arrays of the common path stay in registers.
        double Dc[9], x, n;
        bool b = false;
#pragma unroll
        for (int m = 0; m < 9; ++m) Dc[m] = D[m];
        scan_lines_exact(t, t.line_off[cj * 3 + ci], t.line_off[cj * 3 + ci + 1], Dc, x, n, b);
        mx = mq = x; mn = n;
        bad = bad || b;
    } else {
        scan_cell(D, ci, cj, mx, mn, mq);
    }
    th = theta_of(mean, lo, hi, mx, mn);
}

// Reconstruction and limiter of both fields, one field after the other
// through the same code (18 limited coefficients live one field at a time).
__device__ __forceinline__ void recon_cell(const StageHot& t, const ReconArgs& a, const Physics& ph, int i, int j) {
    if (i >= a.nx || j >= a.ny) return;
    const int nx = a.nx, ny = a.ny;
    const long long cell = (long long)j * nx + i;
    const size_t N = (size_t)nx * ny;
    MP_CHECK_INDEX(a.status, cell, N);
    const int gj = a.gj0 + j, gny = global_ny(a);
    const int ci = i == 0 ? 0 : (i == nx - 1 ? 2 : 1), cj = gj == 0 ? 0 : (gj == gny - 1 ? 2 : 1);
    const long long key = cell + (long long)a.gj0 * nx;
    // Cells stay below 2^31 (checked on create).
    unsigned at[3][3];
#pragma unroll
    for (int dj = 0; dj < 3; ++dj)
#pragma unroll
        for (int di = 0; di < 3; ++di) {
            const int ii = min(max(i + di - 1, 0), nx - 1), jj = min(max(j + dj - 1, 0), ny - 1);
            MP_CHECK_INDEX(a.status, (long long)jj * nx + ii, N);
            at[dj][di] = (unsigned)jj * (unsigned)nx + (unsigned)ii;
        }
    int st = 0;
    bool bad = false, means = true;
    double loH = 0, hiH = 0, loC = 0, hiC = 0, topH = 0;
#pragma unroll 1
    for (int f = 0; f < 2; ++f) {
        double D[9], mean, lo, hi, th, mq;
        recon_field(t, f ? a.C : a.H, at, ci, cj, f ? ph.k.Xe : INFINITY, D, mean, lo, hi, th, mq, st, bad);
        // state_reconstruction.cpp:187-188: admissible means.
        means = means && isfinite(mean) && mean >= 0.0 && (f == 0 || mean <= ph.k.Xe);
        if (f) { loC = lo; hiC = hi; }
        else { loH = lo; hiH = hi; topH = fma(th, mq, mean); }
        if (a.theta) a.theta[f * N + cell] = th;
        double* r = a.rec + rec_at(cell) + f * 9 * kRecStride;
#pragma unroll
        for (int m = 0; m < 9; ++m) r[m * kRecStride] = D[m] * th;
    }
    const int st_lim = !means ? (int)E_OUTOFRANGE : (bad ? (int)E_FP : 0);
    // With a lithostatic pressure Tep is monotone over the cell's height.
    double t0 = ph.Tep, t1 = t0;
    if (ph.litho) {
        t0 = tep_at(ph, t.y0 + gj * t.dy);
        t1 = tep_at(ph, t.y0 + (gj + 1) * t.dy);
    }
    a.flags[cell] = st || st_lim ? (unsigned char)FLAG_CHECK
                                 : cell_flags(ph, fmin(t0, t1), fmax(t0, t1), loH, hiH, loC, hiC, topH);
    if (st) record_error(a.status, PART_UPDATE, key, st);
    if (st_lim) record_error(a.status, PART_LIMIT, key, st_lim);
}

// ---------------------------------------------------------- cell phase kernel

struct CellPhaseArgs {
    int nx, ny;
    const StageHot* tab;   // batched instances: their tables in device memory
    const double* H;
    const double* C;
    const double* rec;
    unsigned char* flags;
    double* T;
    double* phi;
    unsigned long long* status;
    int gj0 = 0, gny = 0;  // slab: global row of local row 0, global rows
    // Adiabatic source (when Physics::source): vertical solid and Darcy
    // velocities at the cell points [cell*25 + b*5 + a]; per cell the heat
    // sum w/A * source, the rate sum w/A * cooling |v_y| and sum w * source.
    const double* cvs_y = nullptr;
    const double* cud_y = nullptr;
    double* srcH = nullptr;
    double* srcR = nullptr;
    double* srcS = nullptr;
    const int* gate = nullptr;   // device flag: the launch does nothing while it is 0
};

__device__ __forceinline__ void load_rec(const double* rec, long long cell, double* DH, double* DC) {
    const double* r = rec + rec_at(cell);
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        DH[m] = MP_LD(r + m * kRecStride);
        DC[m] = MP_LD(r + (m + 9) * kRecStride);
    }
}

// Cell quadrature of T and phi (evolve.cpp:359-376) and the wet flag of the
// porosity sampling (initial_flow.cpp:56-67) on the same 5x5 points, with
// every point's admissibility test and the exact check of the diffusion
// samples: cells that are not plain. Inlined, as the other tested forms are: a
// function of its own reads the tables and constants through generic pointers
// into the kernel's parameters. Where no cell is plain (pure composition,
// 640x1280) the cell phase takes 60 us so and took 90 that way, the faces 182
// and 220, the diffusion 238 and 313; plain cells are as fast either way.
// kExt: the lithostatic pressure and the adiabatic source are compiled in
// (a launch picks the variant; the default path carries none of their code).
template <bool kExt>
__device__ __forceinline__ void cellphase_general(const StageHot& t, const CellPhaseArgs& a, const Physics& ph, long long cell) {
    const long long N = (long long)a.nx * a.ny;
    if (cell >= N) return;
    MP_CHECK_INDEX(a.status, cell, N);
    const double mH = MP_LD(a.H + cell), mC = MP_LD(a.C + cell);
    double DH[9], DC[9];
    load_rec(a.rec, cell, DH, DC);
    int st_por = 0, st_cell = 0, st_face = 0;
    double Tsum = 0.0, Psum = 0.0, Ssum = 0.0, Rsum = 0.0, Wsum = 0.0;
    bool wet = false;
    const int gjc = a.gj0 + (int)(cell / a.nx);
    for (int b = 0; b < kNQ; ++b) {
        double h0, h1, h2, c0, c1, c2;
        const double y = t.g[b];
        q2_row(DH, y, h0, h1, h2);
        q2_row(DC, y, c0, c1, c2);
        const double tep = (kExt && ph.litho) ? tep_at(ph, height(t, gjc, y)) : ph.Tep;
#pragma unroll
        for (int q = 0; q < kNQ; ++q) {
            const double x = t.g[q];
            const double h = mH + quad(h0, h1, h2, x);
            const double c = mC + quad(c0, c1, c2, x);
            PhaseLean pl;
            const int s = phase_stage_lean(ph.sk, h, c, tep, pl);
            if (s) { st_por = st_por ? st_por : s; continue; }
            if (!(pl.T >= 0.0 && pl.phil < 1.0)) st_cell = st_cell ? st_cell : E_OUTOFRANGE;
            const double w = t.cw[b * kNQ + q];
            Tsum += w * pl.T;
            Psum += w * pl.phil;
            wet = wet || pl.phil > 0.0;
            if (kExt && ph.source) {
                // evolve.cpp:359-369 with PhaseTransportVelocities at this point's porosity.
                const long long at = cell * (kNQ * kNQ) + b * kNQ + q;
                const double factor = pl.phil == 0.0 ? 0.0 : (ph.theta == 0.0 ? pl.phil : pow(pl.phil, 1.0 + ph.theta));
                const double vy = __ldg(a.cvs_y + at) + factor * __ldg(a.cud_y + at);
                const double src = -ph.cooling * pl.T * vy;
                Ssum += w * src;
                Rsum += w * ph.cooling * fabs(vy);
                Wsum += t.cwp[b * kNQ + q] * src;
            }
        }
    }
    const unsigned char fl = a.flags[cell];
    if (fl & FLAG_CHECK) {
        // Exact admissibility of the limited values at the diffusion samples.
        const int i = (int)(cell % a.nx), j = a.gj0 + (int)(cell / a.nx);
        const int ci = i == 0 ? 0 : (i == a.nx - 1 ? 2 : 1);
        const int cj = j == 0 ? 0 : (j == global_ny(a) - 1 ? 2 : 1);
        const int cls = cj * 3 + ci;
        for (int l = t.line_off[cls]; l < t.line_off[cls + 1]; ++l) {
            if (!t.line_kind[l]) continue;
            double h0, h1, h2, c0, c1, c2;
            const bool row = t.line_dir[l] == 0;
            const double lc = t.line_c[l];
            if (row) { q2_row(DH, lc, h0, h1, h2); q2_row(DC, lc, c0, c1, c2); }
            else { q2_col(DH, lc, h0, h1, h2); q2_col(DC, lc, c0, c1, c2); }
            for (int q = 0; q < kNQ; ++q) {
                const double s_ = t.g[q];
                const double h = mH + quad(h0, h1, h2, s_);
                const double c = mC + quad(c0, c1, c2, s_);
                const double tep = (kExt && ph.litho) ? tep_at(ph, height(t, j, row ? lc : t.g[q])) : ph.Tep;
                PhaseLean pl;
                const int s = phase_stage_lean(ph.sk, h, c, tep, pl);
                if (s) { st_face = st_face ? st_face : s; continue; }
                if (!(pl.T >= 0.0 && pl.phil < 1.0)) st_face = st_face ? st_face : E_OUTOFRANGE;
            }
        }
    }
    const long long key = cell + (long long)a.gj0 * a.nx;
    if (st_por) record_error(a.status, PART_POROSITY, key, st_por);
    if (st_face) record_error(a.status, PART_FACES, key, st_face);
    if (st_cell) record_error(a.status, PART_CELLS, key, st_cell);
    a.flags[cell] = (unsigned char)((fl & FLAG_CHECK) | (wet ? FLAG_WET : 0));
    a.T[cell] = Tsum;
    a.phi[cell] = Psum;
    if (kExt && ph.source) { a.srcH[cell] = Ssum; a.srcR[cell] = Rsum; a.srcS[cell] = Wsum; }
}

// The same quadrature of a plain cell: no tests, no failure. Bound by the
// FP64 pipe; with the tests, clips and library divisions of every point
// (1239 FP64 and 3187 instructions per warp) it took 100 us at 640x1280, so
// (545 and 987) 46 us.
//
// The adiabatic source's two velocities at 25 points lie cell by cell (200
// bytes apart from lane to lane): a warp first copies its cells' stretch to
// shared memory, lane by lane, where the stride of 25 doubles has no bank
// conflict. Read in place they took 938 L1 wavefronts per warp and 188 us at
// 640x1280. vy: the warp's buffer of 2 x 32 x 25 doubles (kExt, source on).
constexpr int kCellPoints = kNQ * kNQ;
constexpr size_t kSourceBufBytes = 4 * 2 * 32 * kCellPoints * sizeof(double);   // four warps

__device__ __forceinline__ void stage_source(const CellPhaseArgs& a, long long first, long long end, double* vy) {
    const int lane = threadIdx.x & 31;
    const int n = (int)min(32LL, end - first) * kCellPoints;
    const double* vs = a.cvs_y + first * kCellPoints;
    const double* ud = a.cud_y + first * kCellPoints;
    for (int k = lane; k < n; k += 32) {
        __pipeline_memcpy_async(vy + k, vs + k, sizeof(double));
        __pipeline_memcpy_async(vy + 32 * kCellPoints + k, ud + k, sizeof(double));
    }
    __pipeline_commit();
}
// The cell of this lane, [0, end) (every lane of a warp calls). averages: T
// and phi are wanted; the stages inside a step, whose averages nothing reads,
// leave out a plain cell unless its wet flag or source needs the quadrature.
template <bool kExt>
__device__ __forceinline__ void cellphase_cell(const StageHot& t, const CellPhaseArgs& a, const Physics& ph, long long cell,
                                               long long end, bool averages, const double* vy = nullptr) {
    bool valid = cell < end;
    if (valid) cell = checked_index(a.status, cell, (long long)a.nx * a.ny, valid);
    const unsigned char fl = valid ? a.flags[cell] : 0;
    if (!averages && !(kExt && (ph.litho || ph.source)) && (fl & FLAG_PLAIN)) return;
    double DH[9], DC[9];
    if (fl & FLAG_PLAIN) {
        load_rec(a.rec, cell, DH, DC);
        DH[0] += MP_LD(a.H + cell);
        DC[0] += MP_LD(a.C + cell);
    }
    if (kExt && ph.source) {
        __pipeline_wait_prior(0);
        __syncwarp();
    }
    if (!valid) return;
    if (!(fl & FLAG_PLAIN)) { cellphase_general<kExt>(t, a, ph, cell); return; }
    const int gj = a.gj0 + (int)((unsigned)cell / (unsigned)a.nx);
    double Tsum = 0.0, Psum = 0.0, Ssum = 0.0, Rsum = 0.0;
#pragma unroll 1
    for (int b = 0; b < kNQ; ++b) {
        const double y = t.g[b];
        double h0, h1, h2, c0, c1, c2;
        q2_row(DH, y, h0, h1, h2);
        q2_row(DC, y, c0, c1, c2);
        const double tep = (kExt && ph.litho) ? tep_at(ph, height(t, gj, y)) : ph.Tep;
        double Trow = 0.0, Prow = 0.0;   // by row, as the split form adds them
#pragma unroll
        for (int q = 0; q < kNQ; ++q) {
            const double x = t.g[q];
            PhaseLean pl;
            phase_plain<false>(ph.sk, quad(h0, h1, h2, x), quad(c0, c1, c2, x), tep, pl);
            const double w = t.cw[b * kNQ + q];
            Trow = fma(w, pl.T, Trow);
            Prow = fma(w, pl.phil, Prow);
            if (kExt && ph.source) {
                const int at = (int)(threadIdx.x & 31) * kCellPoints + b * kNQ + q;
                const double factor = pl.phil == 0.0 ? 0.0 : (ph.theta == 0.0 ? pl.phil : pow(pl.phil, 1.0 + ph.theta));
                const double v = fma(factor, vy[32 * kCellPoints + at], vy[at]);
                const double wv = w * v;
                Ssum = fma(wv, pl.T, Ssum);
                Rsum += fabs(wv);
            }
        }
        Tsum += Trow;
        Psum += Prow;
    }
    // Porosities are not negative: the cell is wet where their mean is not 0.
    if (kExt && ph.litho) a.flags[cell] = (unsigned char)(fl | (Psum > 0.0 ? FLAG_WET : 0));
    a.T[cell] = Tsum;
    a.phi[cell] = Psum;
    if (kExt && ph.source) {
        // The quadrature weights are per area here and absolute in srcS.
        const double heat = -ph.cooling * Ssum;
        a.srcH[cell] = heat; a.srcR[cell] = ph.cooling * Rsum; a.srcS[cell] = heat * t.area;
    }
}

// ---------------------------------------------------------------- face kernel

struct FaceArgs {
    int nx, ny;
    const StageHot* tab;   // batched instances: their tables in device memory
    const double* H;
    const double* C;
    const double* rec;
    const unsigned char* flags;
    const double* vsn;     // [edge*5 + q], canonical
    const double* udn;
    double* face;          // 4 * nedge SoA: fluxH, fluxC, rate, fluxMixture
    unsigned long long* status;
    int gj0 = 0, gny = 0;  // slab: global row of local row 0, global rows
    const int* gate = nullptr;   // device flag: the launch does nothing while it is 0
};

// Limited H and C of one side along the edge line: v(s) = m + c0 + s*(c1 + s*c2).
struct SideLine {
    double mH, mC;
    double h0, h1, h2, c0, c1, c2;
};

__device__ __forceinline__ void side_line(const FaceArgs& a, long long cell, bool row, double fixed,
                                          SideLine& s) {
    double DH[9], DC[9];
    load_rec(a.rec, cell, DH, DC);
    s.mH = MP_LD(a.H + cell);
    s.mC = MP_LD(a.C + cell);
    if (row) { q2_row(DH, fixed, s.h0, s.h1, s.h2); q2_row(DC, fixed, s.c0, s.c1, s.c2); }
    else { q2_col(DH, fixed, s.h0, s.h1, s.h2); q2_col(DC, fixed, s.c0, s.c1, s.c2); }
}

// Limited evaluation + phase + Phase()'s admissibility (evolve.cpp:270-277).
__device__ __forceinline__ int side_phase(const Physics& ph, const SideLine& s, double at, double tep, double& h,
                                          double& c, PhaseLean& pl) {
    h = s.mH + quad(s.h0, s.h1, s.h2, at);
    c = s.mC + quad(s.c0, s.c1, s.c2, at);
    int st = phase_stage(ph.sk, h, c, tep, pl);
    if (!st && !(pl.T >= 0.0 && pl.phil < 1.0)) st = E_OUTOFRANGE;
    return st;
}

// One edge Gauss point of the face fluxes from both sides' phase states:
// edge porosity, transport velocities, Lax-Friedrichs fluxes or the boundary
// policy (evolve.cpp:36-52,292-329; initial_flow.cpp:94-117), and the point's
// CFL rate term before its quadrature weight; st keeps the first failure.
struct PointFlux {
    double fh, fc, vn, speed;   // speed: (aC + aH + 2 |vs|) * sens
};
__device__ __forceinline__ PointFlux face_point(const Physics& ph, const PhaseLean& A, const PhaseLean& B, double cL,
                                                double cR, bool wetL, bool wetR, bool boundary, double vs, double ud,
                                                double tep, double LD, int& st) {
    // Edge porosity: harmonic mean of both sides, zero next to a dry cell
    // (initial_flow.cpp:94-117). PhaseTransportVelocities (evolve.cpp:36-52)
    // on normal components: bulk = ephi cl + (1 - ephi) cs, and the
    // composition velocity adds cl/bulk times the Darcy flux. With
    // S = phil_A + phil_B and Q = S bulk, ephi = 2 phil_A phil_B / S and
    // cl/bulk = cl S / Q come from one division 1/(S Q) where it is in range.
    const double cl = 0.5 * (A.cl + B.cl), cs = 0.5 * (A.cs + B.cs);
    const double S = A.phil + B.phil;
    double ephi = 0.0, clb = 0.0;   // clb = cl/bulk where bulk > 0, else 0
    if (wetL && wetR && S > 0.0) {
        const double P2 = 2.0 * A.phil * B.phil;
        const double Q = P2 * (cl - cs) + cs * S;
        const double SQ = S * Q;
        if (SQ > 1e-290 && SQ < 1e290) {
            const double x = 1.0 / SQ;
            ephi = P2 * (Q * x);
            clb = cl * (S * (S * x));
        } else {
            ephi = P2 / S;
            const double bulk = ephi * cl + (1.0 - ephi) * cs;
            clb = bulk > 0.0 ? cl / bulk : 0.0;
        }
    }
    const double factor = ephi == 0.0 ? 0.0 : (ph.theta == 0.0 ? ephi : pow(ephi, 1.0 + ph.theta));
    const double flux = factor * ud;
    const double vn = vs + flux;
    const double ve = vs + clb * flux;
    const double aH = ph.lf_global ? ph.lf_speed : fabs(vn);
    const double aC = ph.lf_global ? ph.lf_speed : fabs(ve);
    if (ph.lf_global && !(aH + 1e-14 >= fabs(vn) && aC + 1e-14 >= fabs(ve))) st = st ? st : E_OUTOFRANGE;
    double fh = 0.5 * (vn * (A.T + B.T) - aH * (B.T - A.T)) - LD * (1.0 - ephi) * vs;
    double fc = 0.5 * (ve * (cL + cR) - aC * (cR - cL));
    if (boundary) {
        // EvaluateAdvectionBoundary (initialization.cpp:469-489) per field.
        const int kh = (ph.Hpol == MP_BC_ZERO_FLUX || vn == 0.0) ? 2 : (vn < 0.0 ? 0 : 1);
        const int kc = (ph.Cpol == MP_BC_ZERO_FLUX || ve == 0.0) ? 2 : (ve < 0.0 ? 0 : 1);
        if ((kh == 0 && ph.Hpol != MP_BC_INFLOW_OUTFLOW) || (kc == 0 && ph.Cpol != MP_BC_INFLOW_OUTFLOW))
            st = st ? st : E_OUTOFRANGE;
        const double inC = kc == 0 ? ph.inflowC : cL;
        double Tb = A.T;
        if (kh == 0) {
            PhaseLean pin;
            const int s3 = phase_stage(ph.sk, ph.inflowH, inC, tep, pin);
            if (s3) st = st ? st : s3;
            Tb = pin.T;
        }
        fh = kh == 2 ? 0.0 : vn * Tb - LD * (1.0 - ephi) * vs;
        fc = kc == 2 ? 0.0 : ve * (kc == 0 ? ph.inflowC : cL);
    }
    const double sens = 1.0 + fmax(fabs(A.dTdC), fabs(B.dTdC));
    if (!isfinite(sens)) st = st ? st : E_FP;
    return PointFlux{fh, fc, vn, (aC + aH + 2.0 * fabs(vs)) * sens};
}

// A phase point checked to be plain here, else through the tested form.
__device__ __forceinline__ int inflow_temperature(const Physics& ph, double H, double C, double tep, double& T) {
    PhaseLean p;
    const double slack = 1e-12 * (1.0 + fabs(H));
    int st = 0;
    if (ph.sk.ordinary && tep >= 1e-9 && tep <= 1e100 && H >= slack && H + slack < tep + (1.0 - C * ph.sk.invXe) + ph.k.LD &&
        C >= 1e-90 && C <= ph.k.Xe * (1.0 - 1e-12))
        phase_plain<false>(ph.sk, H, C, tep, p);
    else
        st = phase_stage(ph.sk, H, C, tep, p);
    T = p.T;
    return st;
}

// Transport velocities of an edge point between plain phase states
// (face_point's, without a division): the edge porosity, the mixture velocity
// vn and the composition velocity ve.
__device__ __forceinline__ void plain_velocities(const Physics& ph, const PhaseLean& A, const PhaseLean& B, bool wet,
                                                 double vs, double ud, double& ephi, double& vn, double& ve) {
    ephi = 0.0;
    vn = ve = vs;
    const double P2 = 2.0 * A.phil * B.phil;
    if (!(wet && P2 > 0.0)) return;
    // ephi = P2/S and cl/bulk = cl S/Q as face_point forms them.
    const double S = A.phil + B.phil, cl = 0.5 * (A.cl + B.cl), cs = 0.5 * (A.cs + B.cs);
    const double Q = fma(P2, cl - cs, cs * S), SQ = S * Q;
    double clb;
    if (rcp_range(SQ)) {
        const double x = rcp(SQ);
        ephi = P2 * (Q * x);
        clb = cl * (S * (S * x));
    } else {
        ephi = P2 / S;
        const double bulk = ephi * cl + (1.0 - ephi) * cs;
        clb = bulk > 0.0 ? cl / bulk : 0.0;
    }
    const double factor = ph.theta == 0.0 || ephi == 0.0 ? ephi : pow(ephi, 1.0 + ph.theta);
    vn = fma(factor, ud, vs);
    ve = fma(clb, __dmul_rn(factor, ud), vs);
}

// face_point of an interior edge between two plain cells. With local speeds
// the Lax-Friedrichs flux is the upwind one.
__device__ __forceinline__ PointFlux face_point_plain(const Physics& ph, const PhaseLean& A, const PhaseLean& B, double cL,
                                                      double cR, bool wet, double vs, double ud, int& st) {
    double ephi, vn, ve, fh, fc;
    plain_velocities(ph, A, B, wet, vs, ud, ephi, vn, ve);
    const double latent = ph.k.LD * (1.0 - ephi) * vs;
    double aH = fabs(vn), aC = fabs(ve);
    if (ph.lf_global) {
        if (!(ph.lf_speed + 1e-14 >= aH && ph.lf_speed + 1e-14 >= aC)) st = st ? st : E_OUTOFRANGE;
        aH = aC = ph.lf_speed;
        fh = 0.5 * (vn * (A.T + B.T) - aH * (B.T - A.T)) - latent;
        fc = 0.5 * (ve * (cL + cR) - aC * (cR - cL));
    } else {
        fh = fma(vn, vn >= 0.0 ? A.T : B.T, -latent);
        fc = ve * (ve >= 0.0 ? cL : cR);
    }
    const double dA = fabs(A.dTdC), dB = fabs(B.dTdC);
    return PointFlux{fh, fc, vn, (aC + aH + 2.0 * fabs(vs)) * (1.0 + (dA > dB ? dA : dB))};
}

// face_point at the wall of a plain cell: EvaluateAdvectionBoundary
// (initialization.cpp:469-489) per field.
__device__ __forceinline__ PointFlux wall_point_plain(const Physics& ph, const PhaseLean& A, double c, bool wet, double vs,
                                                      double ud, double tep, int& st) {
    double ephi, vn, ve;
    plain_velocities(ph, A, A, wet, vs, ud, ephi, vn, ve);
    double aH = fabs(vn), aC = fabs(ve);
    if (ph.lf_global) {
        if (!(ph.lf_speed + 1e-14 >= aH && ph.lf_speed + 1e-14 >= aC)) st = st ? st : E_OUTOFRANGE;
        aH = aC = ph.lf_speed;
    }
    const bool inH = vn < 0.0 && ph.Hpol != MP_BC_ZERO_FLUX, inC = ve < 0.0 && ph.Cpol != MP_BC_ZERO_FLUX;
    if ((inH && ph.Hpol != MP_BC_INFLOW_OUTFLOW) || (inC && ph.Cpol != MP_BC_INFLOW_OUTFLOW)) st = st ? st : E_OUTOFRANGE;
    const double cb = inC ? ph.inflowC : c;
    double Tb = A.T;
    if (inH) {
        const int s = inflow_temperature(ph, ph.inflowH, cb, tep, Tb);
        st = st ? st : s;
    }
    const double fh = ph.Hpol == MP_BC_ZERO_FLUX || vn == 0.0 ? 0.0 : fma(vn, Tb, -(ph.k.LD * (1.0 - ephi) * vs));
    const double fc = ph.Cpol == MP_BC_ZERO_FLUX ? 0.0 : ve * cb;
    return PointFlux{fh, fc, vn, (aC + aH + 2.0 * fabs(vs)) * (1.0 + fabs(A.dTdC))};
}

// An edge of the mesh: the edge along i (horizontal) or j at (i, j).
struct EdgeAt {
    bool horizontal;
    int i, j;
};
// Edge k in id order (slabs, and the tested forms below).
__device__ __forceinline__ EdgeAt edge_by_id(int nx, int ny, long long e) {
    const long long nI = (long long)nx * (ny + 1);
    if (e < nI) return EdgeAt{true, (int)((unsigned)e % (unsigned)nx), (int)((unsigned)e / (unsigned)nx)};
    const unsigned k = (unsigned)(e - nI), w = (unsigned)nx + 1u;
    return EdgeAt{false, (int)(k % w), (int)(k / w)};
}
// Edge k of a whole mesh in the order interior horizontal, interior vertical,
// walls: the walls' boundary policy runs in warps of its own instead of in
// one or two lanes of every row's first and last warp.
__device__ __forceinline__ EdgeAt edge_by_kind(int nx, int ny, long long kk) {
    unsigned k = (unsigned)kk;
    const unsigned nh = (unsigned)nx * (unsigned)(ny - 1), w = (unsigned)nx - 1u, nv = w * (unsigned)ny;
    if (k < nh) return EdgeAt{true, (int)(k % (unsigned)nx), (int)(k / (unsigned)nx) + 1};
    k -= nh;
    if (k < nv) return EdgeAt{false, (int)(k % w) + 1, (int)(k / w)};
    k -= nv;
    if (k < 2u * (unsigned)nx) return EdgeAt{true, (int)(k < (unsigned)nx ? k : k - nx), k < (unsigned)nx ? 0 : ny};
    k -= 2u * (unsigned)nx;
    return EdgeAt{false, k < (unsigned)ny ? 0 : nx, (int)(k < (unsigned)ny ? k : k - ny)};
}

__device__ __forceinline__ long long edge_id(int nx, int ny, const EdgeAt& g) {
    return g.horizontal ? (long long)g.j * nx + g.i : (long long)nx * (ny + 1) + (long long)g.j * (nx + 1) + g.i;
}

// Left/right cells and orientation as the reference's Build (evolve.cpp:230-251).
struct EdgeCells {
    long long e, L, R;
    bool boundary, reverse;
};
__device__ __forceinline__ EdgeCells edge_cells(const FaceArgs& a, const EdgeAt& g) {
    const int nx = a.nx;
    EdgeCells c;
    if (g.horizontal) {
        const int gj = a.gj0 + g.j, gny = global_ny(a);
        c.e = (long long)g.j * nx + g.i;
        c.boundary = gj == 0 || gj == gny;
        c.reverse = gj == gny;
        c.L = c.reverse ? c.e - nx : c.e;
        c.R = c.boundary ? -1 : c.e - nx;
    } else {
        c.e = (long long)nx * (a.ny + 1) + (long long)g.j * (nx + 1) + g.i;
        c.boundary = g.i == 0 || g.i == nx;
        c.reverse = g.i == 0;
        const long long row = (long long)g.j * nx;
        c.L = c.reverse ? row : row + g.i - 1;
        c.R = c.boundary ? -1 : row + g.i;
    }
    return c;
}

// An edge of any cells, every point with its admissibility tests: edges with
// a cell that is not plain.
// kExt: the lithostatic pressure is compiled in.
template <bool kExt>
__device__ __forceinline__ void face_general(const StageHot& t, const FaceArgs& a, const Physics& ph, long long e) {
    const long long nE = (long long)a.nx * (a.ny + 1) + (long long)(a.nx + 1) * a.ny;
    const size_t N = (size_t)a.nx * a.ny;
    const EdgeAt at_ = edge_by_id(a.nx, a.ny, e);
    const EdgeCells g = edge_cells(a, at_);
    const double len = at_.horizontal ? t.len_h : t.len_v;
    // The edge's fixed coordinate in the left / right cell frame.
    const double lfix = at_.horizontal == g.reverse ? 1.0 : -1.0, rfix = at_.horizontal ? 1.0 : -1.0;
    SideLine sl, sr;
    side_line(a, g.L, at_.horizontal, lfix, sl);
    if (!g.boundary) side_line(a, g.R, at_.horizontal, rfix, sr);
    const bool wetL = (a.flags[g.L] & FLAG_WET) != 0, wetR = g.boundary ? true : (a.flags[g.R] & FLAG_WET) != 0;
    const double sgn = g.reverse ? -1.0 : 1.0;
    double fluxH = 0.0, fluxC = 0.0, fluxMix = 0.0, rate = 0.0;
    int st = 0;
    for (int q = 0; q < kNQ; ++q) {
        const int cq = g.reverse ? kNQ - 1 - q : q;
        const double at = t.g[cq];
        const double vs = sgn * __ldg(a.vsn + e * kNQ + cq);
        const double ud = sgn * __ldg(a.udn + e * kNQ + cq);
        double hL, cL, hR, cR;
        PhaseLean A, B;
        // Height of this Gauss point: the edge row for horizontal edges.
        const double tep = !(kExt && ph.litho) ? ph.Tep
                         : tep_at(ph, at_.horizontal ? t.y0 + (a.gj0 + at_.j) * t.dy : height(t, a.gj0 + at_.j, at));
        int s = side_phase(ph, sl, at, tep, hL, cL, A);
        if (g.boundary) { B = A; hR = hL; cR = cL; }
        else {
            const int s2 = side_phase(ph, sr, at, tep, hR, cR, B);
            s = s ? s : s2;
        }
        if (s) { st = st ? st : s; continue; }
        const PointFlux pf = face_point(ph, A, B, cL, cR, wetL, wetR, g.boundary, vs, ud, tep, ph.k.LD, st);
        const double w = 0.5 * len * t.gw[q];
        fluxH += w * pf.fh;
        fluxC += w * pf.fc;
        fluxMix += w * pf.vn;
        rate += w * pf.speed;
    }
    if (st) record_error(a.status, PART_FACES, g.L + (long long)a.gj0 * a.nx, st);
    a.face[e] = fluxH;
    a.face[nE + e] = fluxC;
    a.face[2 * nE + e] = rate;
    a.face[3 * nE + e] = fluxMix;
}

// Limited H and C of one side along an edge of a uniform mesh: the cell's
// polynomial at xi or eta = s = +-1, mean included.
__device__ __forceinline__ void edge_line(const FaceArgs& a, long long cell, bool horizontal, double s,
                                          double (&h)[3], double (&c)[3]) {
    double DH[9], DC[9];
    load_rec(a.rec, cell, DH, DC);
    DH[0] += MP_LD(a.H + cell);
    DC[0] += MP_LD(a.C + cell);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (horizontal) {
            h[k] = fma(s, DH[k + 3], DH[k] + DH[k + 6]);
            c[k] = fma(s, DC[k + 3], DC[k] + DC[k + 6]);
        } else {
            h[k] = fma(s, DH[3 * k + 1], DH[3 * k] + DH[3 * k + 2]);
            c[k] = fma(s, DC[3 * k + 1], DC[3 * k] + DC[3 * k + 2]);
        }
    }
}

__device__ __forceinline__ void store_face(const FaceArgs& a, long long e, double half, double fluxH, double fluxC,
                                           double rate, double fluxMix) {
    const long long nE = (long long)a.nx * (a.ny + 1) + (long long)(a.nx + 1) * a.ny;
    a.face[e] = half * fluxH;
    a.face[nE + e] = half * fluxC;
    a.face[2 * nE + e] = half * rate;
    a.face[3 * nE + e] = half * fluxMix;
}

// The Gauss point taken l-th: the centre, then the two pairs.
__device__ __forceinline__ int face_point_at(int l) { return l == 0 ? 2 : (l & 1 ? 2 + ((l + 1) >> 1) : 2 - (l >> 1)); }
// Eutectic temperature at the point s of an edge.
template <bool kExt>
__device__ __forceinline__ double face_tep(const StageHot& t, const FaceArgs& a, const Physics& ph, const EdgeAt& at, double s) {
    if (!(kExt && ph.litho)) return ph.Tep;
    return tep_at(ph, at.horizontal ? t.y0 + (a.gj0 + at.j) * t.dy : height(t, a.gj0 + at.j, s));
}

// A wall edge of a plain cell (in warps of their own, edge_by_kind). Out of
// line: its branches in the interior edges' loop cost that loop registers
// (147 us for them all against 130 when it was taken out).
template <bool kExt>
__device__ __noinline__ void face_wall(const StageHot& t, const FaceArgs& a, const Physics& ph, long long e) {
    const EdgeAt at = edge_by_id(a.nx, a.ny, e);
    const EdgeCells g = edge_cells(a, at);
    double h[3], c[3];
    edge_line(a, g.L, at.horizontal, at.horizontal == g.reverse ? 1.0 : -1.0, h, c);
    const bool wet = (a.flags[g.L] & FLAG_WET) != 0;
    const double sgn = g.reverse ? -1.0 : 1.0;
    double fluxH = 0.0, fluxC = 0.0, fluxMix = 0.0, rate = 0.0;
    int st = 0;
    for (int l = 0; l < kNQ; ++l) {
        const int q = face_point_at(l);
        const double x = t.g[q], x2 = x * x, w = t.gw[q];
        const double vs = sgn * __ldg(a.vsn + e * kNQ + q), ud = sgn * __ldg(a.udn + e * kNQ + q);
        const double tep = face_tep<kExt>(t, a, ph, at, x);
        const double cx = fma(c[1], x, fma(c[2], x2, c[0]));
        PhaseLean A;
        phase_plain<true>(ph.sk, fma(h[1], x, fma(h[2], x2, h[0])), cx, tep, A);
        const PointFlux pf = wall_point_plain(ph, A, cx, wet, vs, ud, tep, st);
        fluxH = fma(w, pf.fh, fluxH);
        fluxC = fma(w, pf.fc, fluxC);
        fluxMix = fma(w, pf.vn, fluxMix);
        rate = fma(w, pf.speed, rate);
    }
    if (st) record_error(a.status, PART_FACES, g.L + (long long)a.gj0 * a.nx, st);
    store_face(a, e, 0.5 * (at.horizontal ? t.len_h : t.len_v), fluxH, fluxC, rate, fluxMix);
}

// Fluxes and rate of one edge. The Gauss points are taken as the centre and
// two symmetric pairs, whose values share their even part. With every point
// tested, clipped and divided through the library, in a loop that carried the
// boundary policy, the kernel issued 2909 instructions per warp, 969 of them
// FP64, and took 219 us at 640x1280; so 1135, 482 and 121 us. Bound by the
// latency of the phase evaluation's chain and the records' loads together
// (issue 47 %, FP64 pipe 40 %, DRAM 3.7 TB/s).
template <bool kExt>
__device__ __forceinline__ void face_edge(const StageHot& t, const FaceArgs& a, const Physics& ph, const EdgeAt& at) {
    const EdgeCells g = edge_cells(a, at);
    const size_t N = (size_t)a.nx * a.ny;
    MP_CHECK_INDEX(a.status, g.L, N);
    if (!g.boundary) MP_CHECK_INDEX(a.status, g.R, N);
    const unsigned char fl = a.flags[g.L] & (g.boundary ? 0xff : a.flags[g.R]);
    if (!(fl & FLAG_PLAIN)) { face_general<kExt>(t, a, ph, g.e); return; }
    if (g.boundary) { face_wall<kExt>(t, a, ph, g.e); return; }
    const bool wet = (fl & FLAG_WET) != 0;
    double hL[3], cL[3], hR[3], cR[3];
    edge_line(a, g.L, at.horizontal, at.horizontal ? -1.0 : 1.0, hL, cL);
    edge_line(a, g.R, at.horizontal, at.horizontal ? 1.0 : -1.0, hR, cR);
    double fluxH = 0.0, fluxC = 0.0, fluxMix = 0.0, rate = 0.0;
    int st = 0;
#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
        const double x = t.g[2 + p], x2 = x * x, w = t.gw[2 + p];
        const double eHL = fma(hL[2], x2, hL[0]), eCL = fma(cL[2], x2, cL[0]);
        const double eHR = fma(hR[2], x2, hR[0]), eCR = fma(cR[2], x2, cR[0]);
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            if (m == 1 && p == 0) break;
            const double s = m ? -x : x;
            const long long v = g.e * kNQ + (m ? 2 - p : 2 + p);
            const double vs = __ldg(a.vsn + v), ud = __ldg(a.udn + v);
            const double tep = face_tep<kExt>(t, a, ph, at, s);
            const double cl = fma(cL[1], s, eCL), cr = fma(cR[1], s, eCR);
            PhaseLean A, B;
            phase_plain<true>(ph.sk, fma(hL[1], s, eHL), cl, tep, A);
            phase_plain<true>(ph.sk, fma(hR[1], s, eHR), cr, tep, B);
            const PointFlux pf = face_point_plain(ph, A, B, cl, cr, wet, vs, ud, st);
            fluxH = fma(w, pf.fh, fluxH);
            fluxC = fma(w, pf.fc, fluxC);
            fluxMix = fma(w, pf.vn, fluxMix);
            rate = fma(w, pf.speed, rate);
        }
    }
    if (st) record_error(a.status, PART_FACES, g.L + (long long)a.gj0 * a.nx, st);
    store_face(a, g.e, 0.5 * (at.horizontal ? t.len_h : t.len_v), fluxH, fluxC, rate, fluxMix);
}

// ------------------------------------------------------------- diffusion

// The diffusive part of one edge's H flux and rate (evolve.cpp:330-347 with
// IntegrateDiffusive(Boundary)FluxWithDerivatives, diffusiveflux.cpp:105-200,
// identity law): temperatures of the limited states at 4 samples per Gauss
// point on the line normal to the edge (2 per side; at a wall 4 inside and the
// wall value), gradient sum_k c_k (T_k - T_last) / ds, flux -= w kappa grad,
// and |d flux / d T_k| added to the rate sample by sample. Added to the face
// results after the advective part, as the reference adds them.
// Edges with a cell that is not plain. kLitho: the lithostatic pressure is
// compiled in.
template <bool kLitho>
__device__ __forceinline__ void diffusion_general(const StageHot& t, const FaceArgs& a, const Physics& ph, long long e) {
    const int nx = a.nx, ny = a.ny;
    const long long nI = (long long)nx * (ny + 1);
    const long long nE = nI + (long long)(nx + 1) * ny;
    if (e >= nE) return;
    const size_t N = (size_t)nx * ny;
    bool boundary, reverse, horizontal;
    long long L, Rc = -1;
    int wall = -1;
    if (e < nI) {
        horizontal = true;
        const unsigned ue = (unsigned)e;
        const int i = (int)(ue % (unsigned)nx), j = (int)(ue / (unsigned)nx);
        const int gj = a.gj0 + j, gny = global_ny(a);
        boundary = (gj == 0 || gj == gny);
        reverse = (gj == gny);
        L = reverse ? (long long)(j - 1) * nx + i : (long long)j * nx + i;
        if (!boundary) Rc = (long long)(j - 1) * nx + i;
        else wall = gj == 0 ? 0 : 1;
    } else {
        horizontal = false;
        const unsigned k = (unsigned)(e - nI);
        const int i = (int)(k % (unsigned)(nx + 1)), j = (int)(k / (unsigned)(nx + 1));
        boundary = (i == 0 || i == nx);
        reverse = (i == 0);
        L = reverse ? (long long)j * nx : (long long)j * nx + (i - 1);
        if (!boundary) Rc = (long long)j * nx + i;
        else wall = i == 0 ? 2 : 3;
    }
    const int type = boundary ? ph.wall_type[wall] : 1;
    if (boundary && type == 0) return;             // zero flux: nothing added
    MP_CHECK_INDEX(a.status, L, N);
    if (!boundary) MP_CHECK_INDEX(a.status, Rc, N);
    const int o = horizontal ? 0 : 1;
    double DL[9], CL[9], DR[9], CR[9];
    double mHL = 0, mCL = 0, mHR = 0, mCR = 0;
    if (type == 1) {
        load_rec(a.rec, L, DL, CL);
        mHL = MP_LD(a.H + L); mCL = MP_LD(a.C + L);
        if (!boundary) {
            load_rec(a.rec, Rc, DR, CR);
            mHR = MP_LD(a.H + Rc); mCR = MP_LD(a.C + Rc);
        }
    }
    double integral = 0.0, rate = a.face[2 * nE + e];
    const double kappa = ph.kappa;
    int st = 0;
    for (int q = 0; q < kNQ; ++q) {
        const double w = t.dif_w[o][q];
        if (boundary && type == 2) { integral += w * ph.wall_value[wall]; continue; }
        const int cq = reverse ? kNQ - 1 - q : q;
        const double at = t.g[cq];
        const int count = boundary ? 5 : 4;
        double v[5];
        // Temperatures at the samples: limited H, C on the line across the edge
        // through this Gauss point, in the frame of the sample's cell.
        double lh0, lh1, lh2, lc0, lc1, lc2, rh0 = 0, rh1 = 0, rh2 = 0, rc0 = 0, rc1 = 0, rc2 = 0;
        if (horizontal) { q2_col(DL, at, lh0, lh1, lh2); q2_col(CL, at, lc0, lc1, lc2); }
        else { q2_row(DL, at, lh0, lh1, lh2); q2_row(CL, at, lc0, lc1, lc2); }
        if (!boundary) {
            if (horizontal) { q2_col(DR, at, rh0, rh1, rh2); q2_col(CR, at, rc0, rc1, rc2); }
            else { q2_row(DR, at, rh0, rh1, rh2); q2_row(CR, at, rc0, rc1, rc2); }
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const bool left = boundary || k < 2;
            const double s = boundary ? t.dif_pos_bnd[wall][k] : t.dif_pos_int[o][k];
            const double h = left ? mHL + quad(lh0, lh1, lh2, s) : mHR + quad(rh0, rh1, rh2, s);
            const double c = left ? mCL + quad(lc0, lc1, lc2, s) : mCR + quad(rc0, rc1, rc2, s);
            const long long cellk = left ? L : Rc;
            const double tep = !(kLitho && ph.litho) ? ph.Tep
                             : tep_at(ph, height(t, a.gj0 + (int)(cellk / nx), horizontal ? s : at));
            PhaseLean pl;
            int s1 = phase_stage_lean(ph.sk, h, c, tep, pl);
            if (!s1 && !(pl.T >= 0.0 && pl.phil < 1.0)) s1 = E_OUTOFRANGE;
            if (s1) st = st ? st : s1;
            v[k] = s1 ? 0.0 : pl.T;
        }
        if (boundary) v[4] = ph.wall_value[wall];
        const double* c = boundary ? t.dif_c_bnd : t.dif_c_int;
        const double last = v[count - 1];
        double grad = 0.0, clast = 0.0;
        for (int k = 0; k + 1 < count; ++k) { grad += c[k] * (v[k] - last); clast -= c[k]; }
        const double ds = t.dif_ds[o][boundary ? 1 : 0];
        grad /= ds;
        if (!isfinite(grad)) st = st ? st : E_FP;
        integral -= w * kappa * grad;
        const double scale = -w * kappa / ds;
        for (int k = 0; k < count; ++k) {
            if (boundary && k + 1 == count) continue;     // the wall value: not a sample
            rate += fabs(scale * (k + 1 == count ? clast : c[k]));
        }
    }
    if (st) record_error(a.status, PART_FACES, L + (long long)a.gj0 * nx, st);
    a.face[e] += integral;
    a.face[2 * nE + e] = rate;
}

// The same part of an interior edge between plain cells or (kWall) of a plain
// cell at a wall of prescribed temperature: on each Gauss point's normal line
// the limited states are one quadratic per side, whose coefficients are taken
// for the centre and the two symmetric pairs of points. The rate's share is a
// constant of the edge. 1100 instructions and 140 us at 640x1280; with every
// sample tested and its derivative added to the rate one by one 4591 and 441.
// The derivative weights are [1/24, -9/8, 9/8, -1/24] and [1/4, -4/3, 3, -4, 25/12].
template <bool kWall, bool kLitho>
__device__ __forceinline__ void diffusion_plain(const StageHot& t, const FaceArgs& a, const Physics& ph, const EdgeAt& at,
                                                const EdgeCells& g, int wall) {
    const int o = at.horizontal ? 0 : 1;
    // Coefficients of each side by power across the edge [k] and along it [j].
    struct SideD { double h[3][3], c[3][3]; } s[kWall ? 1 : 2];
#pragma unroll
    for (int n = 0; n < (kWall ? 1 : 2); ++n) {
        const long long cell = n ? g.R : g.L;
        double DH[9], DC[9];
        load_rec(a.rec, cell, DH, DC);
        DH[0] += MP_LD(a.H + cell);
        DC[0] += MP_LD(a.C + cell);
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                s[n].h[k][j] = at.horizontal ? DH[3 * k + j] : DH[3 * j + k];
                s[n].c[k][j] = at.horizontal ? DC[3 * k + j] : DC[3 * j + k];
            }
    }
    double sum = 0.0;
#pragma unroll 1
    for (int p = 0; p < 3; ++p) {
        const double x = t.g[2 + p], x2 = x * x, w = t.gw[2 + p];
#pragma unroll 1
        for (int m = 0; m < (p ? 2 : 1); ++m) {
            const double xs = m ? -x : x;
            double v[4];
#pragma unroll
            for (int n = 0; n < (kWall ? 1 : 2); ++n) {
                double h[3], c[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    h[k] = fma(s[n].h[k][1], xs, fma(s[n].h[k][2], x2, s[n].h[k][0]));
                    c[k] = fma(s[n].c[k][1], xs, fma(s[n].c[k][2], x2, s[n].c[k][0]));
                }
                const int row = a.gj0 + (at.horizontal ? (g.reverse || n ? at.j - 1 : at.j) : at.j);
#pragma unroll
                for (int q = 0; q < (kWall ? 4 : 2); ++q) {
                    const double y = kWall ? t.dif_pos_bnd[wall][q] : t.dif_pos_int[o][2 * n + q];
                    const double tep = !(kLitho && ph.litho) ? ph.Tep : tep_at(ph, height(t, row, at.horizontal ? y : xs));
                    PhaseLean pl;
                    phase_plain<false>(ph.sk, quad(h[0], h[1], h[2], y), quad(c[0], c[1], c[2], y), tep, pl);
                    v[2 * n + q] = pl.T;
                }
            }
            if (kWall) {
                const double last = ph.wall_value[wall];
                double grad = 0.0;
#pragma unroll
                for (int q = 0; q < 4; ++q) grad = fma(t.dif_c_bnd[q], v[q] - last, grad);
                sum = fma(w, grad, sum);
            } else {
                sum = fma(w, fma(t.dif_c_int[0], v[0] - v[3], t.dif_c_int[2] * (v[2] - v[1])), sum);
            }
        }
    }
    // flux -= sum_q (len w_q / 2) kappa grad_q / ds; the rate gets the same
    // sum of |d flux / d T_k|, whose Gauss weights add up to 2.
    const double len = at.horizontal ? t.len_h : t.len_v;
    const double scale = 0.5 * len * ph.kappa / t.dif_ds[o][kWall ? 1 : 0];
    double weights = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) weights += fabs(kWall ? t.dif_c_bnd[q] : t.dif_c_int[q]);
    const long long nE = (long long)a.nx * (a.ny + 1) + (long long)(a.nx + 1) * a.ny;
    a.face[g.e] = fma(-scale, sum, a.face[g.e]);
    a.face[2 * nE + g.e] = fma(2.0 * scale, weights, a.face[2 * nE + g.e]);
}
template <bool kLitho>
__device__ __noinline__ void diffusion_wall(const StageHot& t, const FaceArgs& a, const Physics& ph, long long e, int wall) {
    const EdgeAt at = edge_by_id(a.nx, a.ny, e);
    diffusion_plain<true, kLitho>(t, a, ph, at, edge_cells(a, at), wall);
}
// With the pressure compiled in, the tested form beside the plain one spills
// (155 us against 151 at 640x1280 with plain cells): out of line there.
__device__ __noinline__ void diffusion_general_litho(const StageHot& t, const FaceArgs& a, const Physics& ph, long long e) {
    diffusion_general<true>(t, a, ph, e);
}

template <bool kLitho>
__device__ __forceinline__ void diffusion_edge(const StageHot& t, const FaceArgs& a, const Physics& ph, const EdgeAt& at) {
    const EdgeCells g = edge_cells(a, at);
    const size_t N = (size_t)a.nx * a.ny;
    const int wall = at.horizontal ? (g.reverse ? 1 : 0) : (g.reverse ? 2 : 3);
    if (g.boundary && ph.wall_type[wall] == MP_THERMAL_ZERO_FLUX) return;
    MP_CHECK_INDEX(a.status, g.L, N);
    if (!g.boundary) MP_CHECK_INDEX(a.status, g.R, N);
    const unsigned char fl = a.flags[g.L] & (g.boundary ? 0xff : a.flags[g.R]);
    // A wall temperature beyond 1e100 takes the form that tests the gradient
    // for overflow; a plain cell's temperatures stay below.
    const bool tested = !(fl & FLAG_PLAIN) ||
                        (g.boundary && (ph.wall_type[wall] == MP_THERMAL_FLUX || !(fabs(ph.wall_value[wall]) <= 1e100)));
    if (tested) {
        if constexpr (kLitho) diffusion_general_litho(t, a, ph, g.e);
        else diffusion_general<false>(t, a, ph, g.e);
    }
    else if (g.boundary) diffusion_wall<kLitho>(t, a, ph, g.e, wall);
    else diffusion_plain<false, kLitho>(t, a, ph, at, g, 0);
}

// ----------------------------------------------------------------- sum kernel

// Where a block of the accumulation (or axpy) kernels leaves its share, and
// who adds the shares up: the block that finishes last, in share order.
struct Shares {
    Partial* partial;      // `count` shares
    Totals* totals;
    unsigned* ticket;      // blocks finished; 0 between launches
    int count;
};

enum SumMode : int { SUM_STORE_L = 0, SUM_RK = 1 };

struct SumArgs {
    int nx, ny;
    double area;           // cell area
    double inv_area;       // 1 / area
    const double* face;
    const double* H;       // stage state
    const double* C;
    const double* H0;      // U^n
    const double* C0;
    double* outH;          // RK: next state; STORE_L: rhs
    double* outC;
    double* rate;          // optional per-cell rate
    int mode;
    double a0, a1, dt;     // next = a0*U^n + a1*(U + dt*L)
    Shares shares;
    const double* dtp;     // when set, dt is read from device memory (batched instances)
    int gj0 = 0, gny = 0;  // slab: global row of local row 0, global rows
    long long cbeg = 0;    // cells [cbeg, cend) are accumulated (cend < 0: all)
    long long cend = -1;
    // Adiabatic source per cell (cell phase kernel): heat, rate, integral.
    const double* srcH = nullptr;
    const double* srcR = nullptr;
    const double* srcS = nullptr;
    // General quad meshes: the area of every cell (else `area` for all).
    const double* cell_area = nullptr;
    const int* gate = nullptr;   // device flag: the launch does nothing while it is 0
    unsigned long long* status = nullptr;   // status word of the index checks (MP_CHECKED)
};

__device__ __forceinline__ bool gated_off(const int* gate) { return gate && *gate == 0; }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_min(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Deterministic reduction of one Partial per thread over the first kRedBlock
// threads of a block (every thread of the block calls; valid in thread 0).
// The 11 fields lie in shared memory as rows: a warp folds whole rows, lane l
// the entries l, l + 32, ... in order, then its shuffle tree. Reducing all
// fields in every warp and again over the warps took two thirds of a small
// block's time (55 dependent shuffle steps twice).
constexpr int kFields = 11;
__device__ __forceinline__ Partial block_reduce(const Partial& v) {
    __shared__ double sh[kFields][kRedBlock];
    __shared__ double out[kFields];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __syncthreads();
    if (tid < kRedBlock) {
        const double r[kFields] = {v.maxRate, v.divergence, v.Cmax, v.nonfinite, v.Hmin, v.Cmin, v.bH, v.bC, v.HI, v.CI, v.sH};
#pragma unroll
        for (int k = 0; k < kFields; ++k) sh[k][tid] = r[k];
    }
    __syncthreads();
    // Rows 0-3: maxima, 4-5: minima, 6-10: sums.
    for (int k = warp; k < kFields; k += (int)(blockDim.x >> 5)) {
        double x = sh[k][lane];
        auto fold = [&](double y) { x = k < 4 ? fmax(x, y) : k < 6 ? fmin(x, y) : x + y; };
#pragma unroll
        for (int n = 32; n < kRedBlock; n += 32) fold(sh[k][lane + n]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) fold(__shfl_down_sync(0xffffffffu, x, o));
        if (lane == 0) out[k] = x;
    }
    __syncthreads();
    return Partial{out[0], out[1], out[6], out[7], out[8], out[9], out[4], out[5], out[2], out[3], out[10]};
}

// This block's share, and by the last block the totals.
__device__ __forceinline__ void finish_block(const Partial& v, const Shares& s, int index) {
    __shared__ bool last;
    const Partial b = block_reduce(v);
    if (threadIdx.x == 0) {
        s.partial[index] = b;
        __threadfence();
        last = atomicAdd(s.ticket, 1u) == (unsigned)s.count - 1u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    Partial w = partial_identity();
    for (int k = threadIdx.x; k < s.count; k += kRedBlock) {
        const double* f = reinterpret_cast<const double*>(s.partial + k);
        Partial q;
        double* d = reinterpret_cast<double*>(&q);
#pragma unroll
        for (int n = 0; n < kFields; ++n) d[n] = __ldcg(f + n);
        fold_partial(w, q);
    }
    w = block_reduce(w);
    if (threadIdx.x == 0) {
        *s.totals = Totals{w.maxRate, w.divergence, w.bH, w.bC, w.HI, w.CI, w.Hmin, w.Cmin, w.Cmax, w.nonfinite, w.sH};
        *s.ticket = 0;
    }
}

// Per-cell accumulation + RK combination; folds the cell's contribution to
// the stage reductions into v.
// kSrc: the adiabatic source terms are added. kArea: per-cell areas.
template <bool kSrc = false, bool kArea = false>
__device__ __forceinline__ void sum_cell(const SumArgs& a, unsigned cell, const double* dtp, Partial& v) {
    const int nx = a.nx, ny = a.ny;
    const long long nI = (long long)nx * (ny + 1);
    const long long nE = nI + (long long)(nx + 1) * ny;
    const int i = (int)(cell % (unsigned)nx), j = (int)(cell / (unsigned)nx);
    MP_CHECK_INDEX(a.status, cell, (long long)nx * ny);
    const double A = kArea ? __ldg(a.cell_area + cell) : a.area, invA = kArea ? 1.0 / A : a.inv_area;
    // Faces of this cell in the reference's id order: bottom, top, left, right,
    // each with the sign of its side (evolve.cpp:350-354).
    const unsigned eb = cell, et = cell + (unsigned)nx;
    const unsigned el = (unsigned)nI + cell + (unsigned)j, er = el + 1u;    // below 2^31 (mesh_too_large)
    MP_CHECK_INDEX(a.status, et, nI);
    MP_CHECK_INDEX(a.status, er, nE);
    const int gj = a.gj0 + j, gny = global_ny(a);
    const double sb = -1.0, stp = (gj == gny - 1) ? -1.0 : 1.0, sl = (i == 0) ? -1.0 : 1.0, sr = -1.0;
    const unsigned ids[4] = {eb, et, el, er};
    const double sg[4] = {sb, stp, sl, sr};
    const double *fH = a.face, *fC = fH + nE, *fR = fC + nE, *fM = fR + nE;
    // The reference divides each face term by the area; here the signed sums
    // are scaled once by 1/A (a few ulp apart).
    double rH = 0.0, rC = 0.0, rr = 0.0, dv = 0.0, bH = 0.0, bC = 0.0;
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const double FH = MP_LD(fH + ids[f]), FC = MP_LD(fC + ids[f]), FR = MP_LD(fR + ids[f]), FM = MP_LD(fM + ids[f]);
        rH += sg[f] * FH;
        rC += sg[f] * FC;
        rr += FR;
        dv -= sg[f] * FM;
    }
    rH *= invA; rC *= invA; rr *= invA; dv *= invA;
    double sH = 0.0;
    if (kSrc) {
        // The source terms follow the face terms, as the reference adds them.
        rH += MP_LD(a.srcH + cell); rr += MP_LD(a.srcR + cell); sH = MP_LD(a.srcS + cell);
    }
    if (gj == 0) { bH += MP_LD(fH + eb); bC += MP_LD(fC + eb); }
    if (gj == gny - 1) { bH += MP_LD(fH + et); bC += MP_LD(fC + et); }
    if (i == 0) { bH += MP_LD(fH + el); bC += MP_LD(fC + el); }
    if (i == nx - 1) { bH += MP_LD(fH + er); bC += MP_LD(fC + er); }
    double nh, nc;
    if (a.mode == SUM_RK) {
        const double dt_ = dtp ? *dtp : a.dt;
        const double h = MP_LD(a.H + cell), c = MP_LD(a.C + cell);
        const double sh_ = __dadd_rn(h, __dmul_rn(dt_, rH));
        const double sc_ = __dadd_rn(c, __dmul_rn(dt_, rC));
        nh = __dadd_rn(__dmul_rn(a.a0, MP_LD(a.H0 + cell)), __dmul_rn(a.a1, sh_));
        nc = __dadd_rn(__dmul_rn(a.a0, MP_LD(a.C0 + cell)), __dmul_rn(a.a1, sc_));
    } else {
        nh = MP_LD(a.H + cell); nc = MP_LD(a.C + cell);
    }
    a.outH[cell] = a.mode == SUM_RK ? nh : rH;
    a.outC[cell] = a.mode == SUM_RK ? nc : rC;
    if (a.rate) a.rate[cell] = rr;
    v.maxRate = fmax(v.maxRate, rr);
    v.divergence = fmax(v.divergence, fabs(dv));
    v.bH += bH; v.bC += bC;
    v.HI += nh * A; v.CI += nc * A;
    v.Hmin = fmin(v.Hmin, nh); v.Cmin = fmin(v.Cmin, nc); v.Cmax = fmax(v.Cmax, nc);
    v.nonfinite = fmax(v.nonfinite, (isfinite(nh) && isfinite(nc) && isfinite(rr)) ? 0.0 : 1.0);
    v.sH += sH;
}

// This thread's cells in the sum block starting at first.
// `first` counts from the start of the accumulated range [cbeg, cend); dtp:
// where the step size is (null: in the arguments).
template <bool kSrc = false, bool kArea = false>
__device__ __forceinline__ Partial sum_cells(const SumArgs& a, long long first, const double* dtp) {
    const long long end = a.cend >= 0 ? a.cend : (long long)a.nx * a.ny;
    const int per = sum_per(end - a.cbeg);
    Partial v = partial_identity();
    auto add = [&](int k) {
        const long long c = a.cbeg + first + k * kRedBlock + threadIdx.x;
        if (c < end) sum_cell<kSrc, kArea>(a, (unsigned)c, dtp, v);
    };
    // A known count lets the cells' loads overlap (1 - 2 % of a step at 321x643).
    if (per <= kSumPer) {
#pragma unroll
        for (int k = 0; k < kSumPer; ++k) {
            if (k >= per) break;
            add(k);
        }
    } else {
#pragma unroll 1
        for (int k = 0; k < per; ++k) add(k);
    }
    return v;
}

// U1 = U^n + dt*L^n over this thread's cells, with the
// admissibility/integral partials of U1 (cell_area: per-cell areas, or null
// for `area` everywhere).
__device__ __forceinline__ Partial axpy_cells(long long n, const double* H0, const double* C0, const double* LH,
                                              const double* LC, double dt, double area, double* H1, double* C1,
                                              long long first, const double* cell_area = nullptr) {
    const int per = sum_per(n);
    Partial v = partial_identity();
#pragma unroll 4
    for (int q = 0; q < per; ++q) {
        const long long k = first + q * kRedBlock + threadIdx.x;
        if (k >= n) continue;
        const double h = __dadd_rn(H0[k], __dmul_rn(dt, LH[k]));
        const double c = __dadd_rn(C0[k], __dmul_rn(dt, LC[k]));
        H1[k] = h; C1[k] = c;
        const double A = cell_area ? __ldg(cell_area + k) : area;
        v.HI += h * A; v.CI += c * A;
        v.Hmin = fmin(v.Hmin, h); v.Cmin = fmin(v.Cmin, c); v.Cmax = fmax(v.Cmax, c);
        v.nonfinite = fmax(v.nonfinite, (isfinite(h) && isfinite(c)) ? 0.0 : 1.0);
    }
    return v;
}


}  // namespace
}  // namespace mp

#endif
