// Coupled H/C transport on B200: FP64 stage kernels, the SSPRK2/SSPRK3 time
// loop and the mp_transport_* entry points.
//
// One stage L(U) (RHS, src/couple/evolve.cpp:279-384) is four kernels, the
// last of which also reduces its totals in a fixed order:
//   recon_kernel      per cell: candidate smoothness + weights, limiter theta,
//                     limited deviation polynomials;
//   cellphase_kernel  per cell: 5x5 cell quadrature of the phase (T, phi, wet
//                     flag), diffusion-sample admissibility;
//   face_kernel       per edge: limited evaluations on both sides at the 5
//                     Gauss points, phase, edge porosity, transport
//                     velocities, local Lax-Friedrichs fluxes, boundary
//                     policy, CFL rate;
//   sum_kernel        per cell: conservative accumulation in the reference's
//                     face order, the Runge-Kutta combination, block partials.
// The time loop (evolve.cpp:428-511) runs on the device (graph_steps: a CUDA
// graph of the stage kernels and the step controller, one host wait per 64
// steps; uniform and general quad meshes) or, for row slabs and profiling
// runs, on the host (do_step: one small device->host read per stage).
#include "common.hpp"
#include "phase_math.cuh"
#include "stage_device.cuh"
#include "stage_kernels.cuh"
#include "step_ctl.cuh"
#include "tables.hpp"
#include "quad_kernels.cuh"
#include "quad_tables.hpp"
#include "small_steps.hpp"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

namespace mp {

PhaseConst phase_const(const mp_material& p, const mp_derived& d);
mp_status derive_checked(const mp_material& p, mp_derived& d);

namespace {

// Rows of one launch: global position of the local rows and the ranges the
// kernels cover (a whole mesh: gj0 = gny = 0, rec and own = [0, ny)).
struct StageRange {
    int gj0 = 0, gny = 0;
    int rec0 = 0, rec1 = 0;    // reconstruction and cell phase rows
    int own0 = 0, own1 = 0;    // rows advanced (faces of their cells, accumulation)
};

StageRange whole(int ny) { StageRange r; r.rec1 = r.own1 = ny; return r; }

// Adiabatic-source buffers of one transport (all null when alpha0 = 0).
struct SourceBufs {
    const double* cvs_y = nullptr;
    const double* cud_y = nullptr;
    double* srcH = nullptr;
    double* srcR = nullptr;
    double* srcS = nullptr;
};

// Single-instance kernels: one thread per cell / edge.
// The stage tables arrive by value as a __grid_constant__ parameter, so the
// unrolled table coefficients are constant-bank operands. Minimum resident
// blocks per SM (register caps) as measured fastest on B200 at 640x1280, each
// against its neighbours in one build: cell phase 6 (48 us; 8: 55, 5: 51; with
// the source's buffers 4: 118, 5: 135, 6: 139), faces 5 (127; 4: 133, 6: 129);
// the reconstruction keeps its natural register count (5 and 6 blocks the
// same). As built now they take 46, 121 and 85 us.
// Cells [c0, c1) are reconstructed (all rows, or a slab's owned rows +- 1), in
// id order: with 32x4 tiles a mesh of 321 columns idles a tenth of the lanes.
__global__ void __launch_bounds__(128) recon_kernel(const __grid_constant__ ReconArgs a,
                                                    const __grid_constant__ Physics ph,
                                                    const __grid_constant__ ParamTables p, unsigned c0, unsigned c1) {
    if (gated_off(a.gate)) return;
    const unsigned cell = c0 + blockIdx.x * blockDim.x + threadIdx.x, nx = (unsigned)a.nx;
    if (cell < c1) recon_cell(p.d, a, ph, (int)(cell % nx), (int)(cell / nx));
}
template <bool kExt>
__global__ void __launch_bounds__(128, kExt ? 4 : 6) cellphase_kernel(const __grid_constant__ CellPhaseArgs a,
                                                           const __grid_constant__ Physics ph,
                                                           const __grid_constant__ ParamTables p, long long c0,
                                                           long long c1, int averages) {
    if (gated_off(a.gate)) return;
    const long long cell = c0 + (long long)blockIdx.x * blockDim.x + threadIdx.x;
    extern __shared__ double source_buf[];
    double* vy = kExt ? source_buf + (threadIdx.x >> 5) * (2 * 32 * kCellPoints) : nullptr;
    const long long first = cell - (threadIdx.x & 31);
    if (kExt && ph.source && first < c1) stage_source(a, first, c1, vy);
    cellphase_cell<kExt>(p.d, a, ph, cell, c1, averages != 0, vy);
}
// Edges [h0, h0 + nh) (horizontal) then [v0, v0 + nv) (vertical): every edge
// of the mesh, or of a slab's owned cells.
// kRange: the edges of a slab's owned rows (two ranges, in id order);
// otherwise every edge of the mesh, the walls last.
template <bool kExt, bool kRange>
__global__ void __launch_bounds__(128, 5) face_kernel(const __grid_constant__ FaceArgs a,
                                                      const __grid_constant__ Physics ph,
                                                      const __grid_constant__ ParamTables p, long long h0, long long nh,
                                                      long long v0, long long nv) {
    if (gated_off(a.gate)) return;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nh + nv) return;
    // One call site: the edge body is inlined once.
    face_edge<kExt>(p.d, a, ph, kRange ? edge_by_id(a.nx, a.ny, k < nh ? h0 + k : v0 + (k - nh))
                                       : edge_by_kind(a.nx, a.ny, k));
}
// The diffusive part of the same edges (only launched when diffusion is on).
// 4 resident blocks: 151 us at 640x1280 against 152 with 5 and 171 with 3
// (unbounded); as built now 140. kLitho: the pressure model is compiled in.
template <bool kLitho>
__global__ void __launch_bounds__(128, 4) diffusion_kernel(const __grid_constant__ FaceArgs a,
                                                        const __grid_constant__ Physics ph,
                                                        const __grid_constant__ ParamTables p, long long h0,
                                                        long long nh, long long v0, long long nv) {
    if (gated_off(a.gate)) return;
    const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= nh + nv) return;
    const bool all = nh == (long long)a.nx * (a.ny + 1) && nv == (long long)(a.nx + 1) * a.ny;
    diffusion_edge<kLitho>(p.d, a, ph, all ? edge_by_kind(a.nx, a.ny, k) : edge_by_id(a.nx, a.ny, k < nh ? h0 + k : v0 + (k - nh)));
}

// Four resident blocks; with the source three (of 79 registers: a step of the
// product physics at 256x512 takes 2 % less).
template <bool kSrc, bool kArea = false>
__global__ void __launch_bounds__(kRedBlock, kSrc ? 3 : 4) sum_kernel(SumArgs a) {
    if (gated_off(a.gate)) return;
    const Partial v = sum_cells<kSrc, kArea>(a, (long long)blockIdx.x * sum_cells_per_block(a.cend - a.cbeg), a.dtp);
    finish_block(v, a.shares, (int)blockIdx.x);
}

// U1 = U^n + dt*L^n with the admissibility/integral partials of U1 (dtp:
// dt read from device memory; gate: see ReconArgs).
__global__ void __launch_bounds__(kRedBlock, 4) axpy_kernel(int n, const double* H0, const double* C0, const double* LH,
                                                         const double* LC, double dt, double area, double* H1,
                                                         double* C1, Shares shares, const double* cell_area,
                                                         const double* dtp = nullptr, const int* gate = nullptr) {
    if (gated_off(gate)) return;
    const Partial v = axpy_cells(n, H0, C0, LH, LC, dtp ? *dtp : dt, area, H1, C1, (long long)blockIdx.x * sum_cells_per_block(n),
                                 cell_area);
    finish_block(v, shares, (int)blockIdx.x);
}

// Commit of an accepted step on the device: U^{n+1} (a stage buffer) into U^n.
__global__ void __launch_bounds__(kRedBlock) commit_kernel(long long n, const double* sH, const double* sC, double* H,
                                                           double* C, const int* gate) {
    if (gated_off(gate)) return;
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
        H[k] = sH[k];
        C[k] = sC[k];
    }
}

}  // namespace
}  // namespace mp

// -------------------------------------------------------------------- handle

struct mp_transport {
    mp_mesh_desc mesh;
    mp_transport_opts opts;
    mp_derived der;
    mp::Physics ph;
    cudaStream_t stream = nullptr;
    int nx = 0, ny = 0;
    size_t N = 0, NE = 0;
    mp::StageTables host_tab;
    mp::ParamTables ptab;                   // kernel-parameter copy of the tables
    // State and stage buffers (device).
    double *H = nullptr, *C = nullptr;      // accepted state U^n
    double *S1H = nullptr, *S1C = nullptr;  // stage states
    double *S2H = nullptr, *S2C = nullptr;
    double *LH = nullptr, *LC = nullptr;    // L(U^n)
    double *T = nullptr, *phi = nullptr;
    void* rec = nullptr;                    // 18 * N doubles (limited deviation polynomials)
    unsigned char* flags = nullptr;         // wet | exact-check flags per cell
    double *vsn = nullptr, *udn = nullptr;
    double* face = nullptr;
    double* rate = nullptr;
    mp::Partial* partial = nullptr;
    mp::Totals* d_tot = nullptr;
    unsigned* d_ticket = nullptr;          // finished blocks of the running reduction
    mp::Totals* h_tot = nullptr;           // pinned, several slots
    unsigned long long* d_status = nullptr;
    unsigned long long* h_status = nullptr;
    int sum_blocks = 0;
    double time = 0.0;
    int accepted = 0;
    bool have_L = false;
    // Time controls (evolve.cpp:449-457, input TimeInput): end time the last
    // step is shortened to land on, and the "fixed" control.
    double t_end = INFINITY;
    bool fixed = false;
    // Row slab of a decomposed mesh (mp_transport_create_slab): local rows
    // hold global rows range.gj0.. of range.gny; rows [own0, own1) are
    // advanced. A whole mesh has range = whole(ny). Between stages the hooks
    // fill the halo rows and combine the stage totals across slabs.
    mp::StageRange range;
    mp_halo_fn halo = nullptr;
    mp_combine_fn combine = nullptr;
    void* hook_user = nullptr;
    // Adiabatic source: cell-point vertical velocities (25 per cell) and the
    // per-cell source sums of a stage.
    double *cvs_y = nullptr, *cud_y = nullptr, *srcH = nullptr, *srcR = nullptr, *srcS = nullptr;
    mp::Totals curTot{};                   // totals of L(U^n)
    // General quad mesh (mp_transport_create_quads): per-cell tables in HBM;
    // cell_area points into them (null on a uniform mesh).
    bool quad = false;
    mp::QuadDev qdev{};
    double* qbuf = nullptr;                // one allocation holding every table
    const double* cell_area = nullptr;
    // Device-resident stepping (uniform meshes without hooks; not while
    // profiling): mp_transport_step runs up to kGraphSteps steps per CUDA
    // graph launch, decisions by the step controller; the graph is captured
    // again when a setter changes what it captured (gen).
    bool use_graph = true;
    unsigned long long gen = 1, graph_gen = 0, small_gen = 0;
    int small_blocks = 0;                  // steps in one kernel of so many blocks (small_steps.cu), or 0: the graph
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t graph_exec = nullptr;
    mp::InstCtl *d_ctl = nullptr, *h_ctl = nullptr;
    mp::CtlHeader *d_hdr = nullptr, *h_hdr = nullptr;
    mp_step_report *d_rep = nullptr, *h_rep = nullptr;
    int* d_gate = nullptr;
    double* d_dt = nullptr;
    unsigned long long host_syncs = 0;     // host waits for device results in stepping calls
    // Optional per-kernel timing (CUDA events on this handle's stream).
    bool profile = false;
    std::vector<cudaEvent_t> ev_pool;
    std::vector<int> ev_kind;              // pending pairs: kind of kernel
    size_t ev_used = 0;
    double kern_ms[6] = {0, 0, 0, 0, 0, 0};
    unsigned long long kern_n[6] = {0, 0, 0, 0, 0, 0};
};

namespace mp {
namespace {


// Event pair around one kernel when profiling
// (kind: 0 reconstruction/limiter, 1 cell phase, 2 face, 3 sum, 4 axpy/reductions).
cudaEvent_t prof_event(mp_transport* t) {
    if (t->ev_used == t->ev_pool.size()) {
        cudaEvent_t e;
        cudaEventCreate(&e);
        t->ev_pool.push_back(e);
    }
    return t->ev_pool[t->ev_used++];
}
template <class F>
void timed(mp_transport* t, int kind, F&& launch) {
    if (!t->profile) { launch(); return; }
    cudaEventRecord(prof_event(t), t->stream);
    launch();
    cudaEventRecord(prof_event(t), t->stream);
    t->ev_kind.push_back(kind);
}
// Called after a stream synchronisation: fold pending pairs into the totals.
void harvest(mp_transport* t) {
    for (size_t k = 0; k < t->ev_kind.size(); ++k) {
        float ms = 0.f;
        if (cudaEventElapsedTime(&ms, t->ev_pool[2 * k], t->ev_pool[2 * k + 1]) == cudaSuccess) {
            t->kern_ms[t->ev_kind[k]] += ms;
            t->kern_n[t->ev_kind[k]] += 1;
        }
    }
    t->ev_kind.clear();
    t->ev_used = 0;
}

void free_all(mp_transport* t) {
    if (t->graph_exec) cudaGraphExecDestroy(t->graph_exec);
    if (t->graph) cudaGraphDestroy(t->graph);
    for (void* p : {(void*)t->d_ctl, (void*)t->d_hdr, (void*)t->d_rep, (void*)t->d_gate, (void*)t->d_dt}) if (p) cudaFree(p);
    for (void* p : {(void*)t->h_ctl, (void*)t->h_hdr, (void*)t->h_rep}) if (p) cudaFreeHost(p);
    for (cudaEvent_t e : t->ev_pool) cudaEventDestroy(e);
    void* bufs[] = {t->H, t->C, t->S1H, t->S1C, t->S2H, t->S2C, t->LH, t->LC, t->T, t->phi,
                    t->rec, t->flags, t->vsn, t->udn, t->face, t->rate, t->partial, t->d_tot, t->d_ticket, t->d_status,
                    t->cvs_y, t->cud_y, t->srcH, t->srcR, t->srcS};
    for (void* b : bufs) if (b) cudaFree(b);
    if (t->qbuf) cudaFree(t->qbuf);
    if (t->h_tot) cudaFreeHost(t->h_tot);
    if (t->h_status) cudaFreeHost(t->h_status);
}

mp_status check_status(mp_transport* t, const char* where) {
    const unsigned long long v = *t->h_status;
    if (v == ~0ULL) return MP_OK;
    const long long cell = (long long)((v >> 8) & ((1ULL << 48) - 1));
    const int code = (int)(v & 0xff);
    if ((int)(v >> 56) == PART_CHECK) {
        set_error("%s: index check: index %lld outside its array (bounds-checked build)", where, cell);
        return (mp_status)code;
    }
    const char* what = code == MP_ERR_ARG_OUTOFRANGE ? "inadmissible state (T < 0, porosity >= 1, C outside [0,Xe] or backflow)"
                     : code == MP_ERR_FP ? "non-finite value in reconstruction, smoothness or CFL rate"
                     : code == MP_ERR_PHASE_INVALID ? "phase input outside [0, Xe] or non-finite"
                     : code == MP_ERR_PHASE_RUNTIME ? "computed phase fraction outside [0, 1]"
                     : code == MP_ERR_PHASE_OVERFLOW ? "phase temperature not representable" : "stage failure";
    set_error("%s: cell %lld: %s", where, cell, what);
    return (mp_status)code;
}

// Launch the stage kernels of state (H, C).
void launch_stage_kernels(int nx, int ny, const StageRange& rg, const ParamTables& pt, const Physics& ph, const double* H, const double* C, double* rec,
                          unsigned char* flags, double* T, double* phi, const double* vsn, const double* udn,
                          double* face, unsigned long long* status, double* theta, bool averages, cudaStream_t s,
                          mp_transport* prof, const SourceBufs& src = SourceBufs{}, const int* gate = nullptr) {
    const size_t NE = (size_t)nx * (ny + 1) + (size_t)(nx + 1) * ny;
    auto run = [&](int kind, auto&& f) { if (prof) timed(prof, kind, f); else f(); };
    {
        ReconArgs a{nx, ny, nullptr, H, C, rec, flags, status, theta, rg.gj0, rg.gny, gate};
        const unsigned c0 = (unsigned)rg.rec0 * nx, c1 = (unsigned)rg.rec1 * nx;
        run(0, [&] { recon_kernel<<<(c1 - c0 + 127) / 128, 128, 0, s>>>(a, ph, pt, c0, c1); });
    }
    {
        CellPhaseArgs a{nx, ny, nullptr, H, C, rec, flags, T, phi, status, rg.gj0, rg.gny,
                           src.cvs_y, src.cud_y, src.srcH, src.srcR, src.srcS, gate};
        const long long c0 = (long long)rg.rec0 * nx, c1 = (long long)rg.rec1 * nx;
        const unsigned g = (unsigned)((c1 - c0 + 127) / 128);
        if (ph.litho || ph.source) run(1, [&] { cellphase_kernel<true><<<g, 128, ph.source ? kSourceBufBytes : 0, s>>>(a, ph, pt, c0, c1, averages); });
        else run(1, [&] { cellphase_kernel<false><<<g, 128, 0, s>>>(a, ph, pt, c0, c1, averages); });
    }
    {
        FaceArgs a{nx, ny, nullptr, H, C, rec, flags, vsn, udn, face, status, rg.gj0, rg.gny, gate};
        const long long nI = (long long)nx * (ny + 1);
        const long long h0 = (long long)rg.own0 * nx, nh = (long long)(rg.own1 - rg.own0 + 1) * nx;
        const long long v0 = nI + (long long)rg.own0 * (nx + 1), nv = (long long)(rg.own1 - rg.own0) * (nx + 1);
        (void)NE;
        const unsigned g = (unsigned)((nh + nv + 127) / 128);
        const bool ranged = !(rg.own0 == 0 && rg.own1 == ny);
        if (ranged) {
            if (ph.litho) run(2, [&] { face_kernel<true, true><<<g, 128, 0, s>>>(a, ph, pt, h0, nh, v0, nv); });
            else run(2, [&] { face_kernel<false, true><<<g, 128, 0, s>>>(a, ph, pt, h0, nh, v0, nv); });
        } else {
            if (ph.litho) run(2, [&] { face_kernel<true, false><<<g, 128, 0, s>>>(a, ph, pt, h0, nh, v0, nv); });
            else run(2, [&] { face_kernel<false, false><<<g, 128, 0, s>>>(a, ph, pt, h0, nh, v0, nv); });
        }
        if (ph.diffusion)
            run(2, [&] {
                if (ph.litho) diffusion_kernel<true><<<g, 128, 0, s>>>(a, ph, pt, h0, nh, v0, nv);
                else diffusion_kernel<false><<<g, 128, 0, s>>>(a, ph, pt, h0, nh, v0, nv);
            });
    }
}

// The shares of a launch of `count` blocks of the accumulation or axpy kernel.
Shares shares_of(const mp_transport* t, int count) { return Shares{t->partial, t->d_tot, t->d_ticket, count}; }

// Launch one stage evaluation of state (H, C). mode SUM_STORE_L writes L to
// (outH, outC); SUM_RK writes a0*U^n + a1*(U + dt*L). Totals land in *d_tot.
// gate / dtp (device-resident steps): a device flag that switches the whole
// launch off, and dt read from device memory.
mp_status launch_stage(mp_transport* t, const double* H, const double* C, int mode, double a0, double a1, double dt,
                       double* outH, double* outC, double* theta = nullptr, const int* gate = nullptr,
                       const double* dtp = nullptr) {
    NvtxRange range("mp_transport stage");
    cudaStream_t s = t->stream;
    if (t->halo) {
        // A slab: its neighbours' owned rows into this stage input's halo rows.
        MP_CUDA(cudaStreamSynchronize(s));
        const int rc = t->halo(t->hook_user, const_cast<double*>(H), const_cast<double*>(C));
        if (rc) { set_error("halo exchange failed (%d)", rc); return rc > 0 ? (mp_status)rc : MP_ERR_CUDA; }
    }
    mp_transport* prof = t->profile ? t : nullptr;
    // The averages T and phi that get_state returns are those of the latest
    // evaluation: in a device-resident step that is L(U^{n+1}), or after a
    // failure the stage that complete_averages then finishes.
    const bool averages = mode == SUM_STORE_L || !gate;
    SourceBufs sb;
    if (t->ph.source) {
        if (!t->cvs_y) {
            set_error("the adiabatic source (alpha0 != 0) needs the flow velocities at the cell quadrature points "
                      "(mp_transport_set_cell_velocity)");
            return MP_ERR_ARG_WRONGSTATE;
        }
        sb = SourceBufs{t->cvs_y, t->cud_y, t->srcH, t->srcR, t->srcS};
    }
    if (t->quad) {
        const StageRange& rg = t->range;
        const int gny = rg.gny > 0 ? rg.gny : t->ny;
        const long long nI = (long long)t->nx * (t->ny + 1);
        const long long h0 = (long long)rg.own0 * t->nx, nh = (long long)(rg.own1 - rg.own0 + 1) * t->nx;
        const long long v0 = nI + (long long)rg.own0 * (t->nx + 1), nv = (long long)(rg.own1 - rg.own0) * (t->nx + 1);
        timed(t, 0, [&] {
            launch_quad_stage(t->qdev, t->nx, t->ny, rg.gj0, gny, rg.rec0, rg.rec1, h0, nh, v0, nv, t->ph, H, C,
                              static_cast<double*>(t->rec), t->flags, t->T, t->phi, t->vsn, t->udn, t->face,
                              t->d_status, theta, SourcePtrs{sb.cvs_y, sb.cud_y, sb.srcH, sb.srcR, sb.srcS}, averages, s, gate);
        });
    } else {
        launch_stage_kernels(t->nx, t->ny, t->range, t->ptab, t->ph, H, C, static_cast<double*>(t->rec), t->flags, t->T,
                                     t->phi, t->vsn, t->udn, t->face, t->d_status, theta, averages, s, prof, sb, gate);
    }
    {
        SumArgs a{t->nx, t->ny, t->host_tab.area, 1.0 / t->host_tab.area, t->face, H, C, t->H, t->C, outH, outC, t->rate, mode, a0, a1, dt,
                  shares_of(t, t->sum_blocks), dtp, t->range.gj0, t->range.gny, (long long)t->range.own0 * t->nx,
                  (long long)t->range.own1 * t->nx, sb.srcH, sb.srcR, sb.srcS, t->cell_area, gate, t->d_status};
        if (t->quad) {
            if (sb.srcH) timed(t, 3, [&] { sum_kernel<true, true><<<t->sum_blocks, kRedBlock, 0, s>>>(a); });
            else timed(t, 3, [&] { sum_kernel<false, true><<<t->sum_blocks, kRedBlock, 0, s>>>(a); });
        } else {
            if (sb.srcH) timed(t, 3, [&] { sum_kernel<true><<<t->sum_blocks, kRedBlock, 0, s>>>(a); });
            else timed(t, 3, [&] { sum_kernel<false><<<t->sum_blocks, kRedBlock, 0, s>>>(a); });
        }
    }
    count_launch(t->quad ? 1 : 4);
    if (!t->quad && t->ph.diffusion) count_launch();
    MP_CUDA(cudaGetLastError());
    return MP_OK;
}

mp_status read_totals(mp_transport* t, Totals& out, bool& failed, const char* where) {
    cudaStream_t s = t->stream;
    MP_CUDA(cudaMemcpyAsync(t->h_tot, t->d_tot, sizeof(Totals), cudaMemcpyDeviceToHost, s));
    MP_CUDA(cudaMemcpyAsync(t->h_status, t->d_status, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    MP_CUDA(cudaStreamSynchronize(s));
    t->host_syncs += 1;
    harvest(t);
    if (t->combine) {
        // A slab: totals and the first failure across all slabs.
        static_assert(sizeof(Totals) == sizeof(mp_stage_partials), "Totals layout");
        const int rc = t->combine(t->hook_user, reinterpret_cast<mp_stage_partials*>(t->h_tot), t->h_status);
        if (rc) { set_error("%s: totals combine failed (%d)", where, rc); return rc > 0 ? (mp_status)rc : MP_ERR_CUDA; }
    }
    out = *t->h_tot;
    failed = *t->h_status != ~0ULL;
    (void)where;
    return MP_OK;
}

mp_status reset_status(mp_transport* t) {
    MP_CUDA(cudaMemsetAsync(t->d_status, 0xff, sizeof(unsigned long long), t->stream));
    return MP_OK;
}

// RHS at the accepted state: L(U^n) -> (LH, LC), totals -> curTot.
mp_status eval_current(mp_transport* t, double* theta = nullptr) {
    MP_TRY(reset_status(t));
    MP_TRY(launch_stage(t, t->H, t->C, SUM_STORE_L, 0, 0, 0, t->LH, t->LC, theta));
    bool failed;
    Totals tot;
    MP_TRY(read_totals(t, tot, failed, "RHS"));
    if (failed) return check_status(t, "RHS");
    if (!std::isfinite(tot.maxRate)) { set_error("RHS: nonfinite coupled stage rate"); return MP_ERR_FP; }
    t->curTot = tot;
    t->have_L = true;
    return MP_OK;
}

size_t own_begin(const mp_transport* t) { return (size_t)t->range.own0 * t->nx; }
size_t own_count(const mp_transport* t) { return (size_t)(t->range.own1 - t->range.own0) * t->nx; }

bool admissible(const Totals& tot, double Xe) {
    return tot.nonfinite == 0.0 && tot.Hmin >= 0.0 && tot.Cmin >= 0.0 && tot.Cmax <= Xe;
}

// One accepted step (evolve.cpp:449-507), SSPRK2 or Shu-Osher SSPRK3.
mp_status do_step(mp_transport* t, mp_step_report& rep) {
    NvtxRange range("mp_transport step (host loop)");
    cudaStream_t s = t->stream;
    if (!t->have_L) MP_TRY(eval_current(t));
    const mp_transport_opts& o = t->opts;
    const double Xe = o.material.Xe;
    const Totals first = t->curTot;
    const double oldHI = first.HI, oldCI = first.CI;
    const double remaining = t->t_end - t->time;
    const double cap = t->fixed ? o.dt_initial : (t->accepted == 0 ? o.dt_initial : o.dt_max);
    const double limit = first.maxRate > 0 ? o.cfl / first.maxRate : o.dt_max;
    double dt = std::min(remaining, cap);
    if (t->fixed && !(dt <= limit * (1 + 1e-12))) {
        set_error("Fixed time step exceeds the phase-coupled CFL bound; use control: cfl");
        return MP_ERR_ARG_OUTOFRANGE;
    }
    if (!t->fixed) dt = std::min(dt, limit);
    const double start = t->time;
    int retries = 0;
    double courant = 0.0;
    Totals second{}, third{}, fin{};
    const size_t o0 = own_begin(t), on = own_count(t);
    const int per_block = sum_cells_per_block((long long)on), nblk_axpy = (int)((on + per_block - 1) / per_block);
    for (;;) {
        if (!(dt >= std::min(remaining, o.dt_min) && retries < 40)) {
            set_error("Coupled step cannot satisfy admissibility/CFL above minimum step");
            return MP_ERR_NOT_CONVERGED;
        }
        bool valid, failed;
        Totals adm;
        timed(t, 4, [&] {
            axpy_kernel<<<nblk_axpy, kRedBlock, 0, s>>>((int)on, t->H + o0, t->C + o0, t->LH + o0, t->LC + o0, dt,
                                                         t->host_tab.area,
                                                         t->S1H + o0, t->S1C + o0, shares_of(t, nblk_axpy),
                                                         t->cell_area ? t->cell_area + o0 : nullptr);
        });
        count_launch();
        MP_CUDA(cudaGetLastError());
        MP_TRY(read_totals(t, adm, failed, "stage 1"));
        valid = admissible(adm, Xe);
        if (valid) {
            MP_TRY(reset_status(t));
            if (o.integrator == MP_SSPRK3)
                MP_TRY(launch_stage(t, t->S1H, t->S1C, SUM_RK, 0.75, 0.25, dt, t->S2H, t->S2C));
            else
                MP_TRY(launch_stage(t, t->S1H, t->S1C, SUM_RK, 0.5, 0.5, dt, t->S2H, t->S2C));
            MP_TRY(read_totals(t, second, failed, "stage 2"));
            if (failed) return check_status(t, "RHS");
            if (!std::isfinite(second.maxRate)) { set_error("RHS: nonfinite coupled stage rate"); return MP_ERR_FP; }
            courant = dt * std::max(first.maxRate, second.maxRate);
            valid = courant <= o.cfl * (1 + 1e-12);
            if (valid) valid = admissible(second, Xe);   // totals of the combined state
        }
        if (valid && o.integrator == MP_SSPRK3) {
            MP_TRY(reset_status(t));
            MP_TRY(launch_stage(t, t->S2H, t->S2C, SUM_RK, 1.0 / 3.0, 2.0 / 3.0, dt, t->S1H, t->S1C));
            MP_TRY(read_totals(t, third, failed, "stage 3"));
            if (failed) return check_status(t, "RHS");
            if (!std::isfinite(third.maxRate)) { set_error("RHS: nonfinite coupled stage rate"); return MP_ERR_FP; }
            courant = dt * std::max(std::max(first.maxRate, second.maxRate), third.maxRate);
            valid = courant <= o.cfl * (1 + 1e-12);
            if (valid) valid = admissible(third, Xe);
            fin = third;
        } else {
            fin = second;
        }
        if (valid) break;
        if (t->fixed) {
            set_error("Fixed coupled step failed stage admissibility/CFL");
            return MP_ERR_ARG_OUTOFRANGE;
        }
        dt *= 0.5;
        ++retries;
    }
    // Balance (evolve.cpp:486-490) from the integrals of the new state.
    const double HI = fin.HI, CI = fin.CI;
    double bH, bC, repH, repC;
    double repS;
    if (o.integrator == MP_SSPRK3) {
        repH = (first.bH + second.bH) / 6 + third.bH * (2.0 / 3.0);
        repC = (first.bC + second.bC) / 6 + third.bC * (2.0 / 3.0);
        repS = (first.sH + second.sH) / 6 + third.sH * (2.0 / 3.0);
        bH = HI - oldHI + dt * (repH - repS);
        bC = CI - oldCI + dt * repC;
    } else {
        repH = .5 * (first.bH + second.bH);
        repC = .5 * (first.bC + second.bC);
        repS = .5 * (first.sH + second.sH);
        bH = HI - oldHI + .5 * dt * (first.bH + second.bH - first.sH - second.sH);
        bC = CI - oldCI + .5 * dt * (first.bC + second.bC);
    }
    if (!(std::fabs(bH) < 1e-10 * std::max(1.0, std::fabs(oldHI)) && std::fabs(bC) < 1e-10)) {
        set_error("Coupled finite-volume conservation balance failed (H %.3e, C %.3e)", bH, bC);
        return MP_ERR_PLIB;
    }
    // Commit: the new state becomes U^n, then its RHS for the next step.
    double* nH = o.integrator == MP_SSPRK3 ? t->S1H : t->S2H;
    double* nC = o.integrator == MP_SSPRK3 ? t->S1C : t->S2C;
    MP_CUDA(cudaMemcpyAsync(t->H, nH, t->N * sizeof(double), cudaMemcpyDeviceToDevice, s));
    MP_CUDA(cudaMemcpyAsync(t->C, nC, t->N * sizeof(double), cudaMemcpyDeviceToDevice, s));
    t->time = start + dt;
    t->have_L = false;
    MP_TRY(eval_current(t));
    ++t->accepted;
    rep = mp_step_report{};
    rep.status = 0; rep.retries = retries; rep.dt = dt; rep.time = t->time; rep.courant = courant;
    rep.boundaryH = repH; rep.boundaryC = repC; rep.sourceH = repS;
    rep.maxRate = t->curTot.maxRate; rep.divergence = t->curTot.divergence;
    rep.balanceH = bH; rep.balanceC = bC; rep.H_integral = HI; rep.C_integral = CI;
    return MP_OK;
}

// ------------------------------------------------------- device-resident steps

constexpr int kGraphSteps = 64;        // steps per graph launch (report rows)

bool graph_usable(const mp_transport* t) {
    return t->use_graph && !t->profile && !t->halo && !t->combine && !(t->ph.source && !t->cvs_y);
}

StepOpts single_step_opts(const mp_transport* t) {
    const mp_transport_opts& o = t->opts;
    StepOpts so{};
    so.cfl = o.cfl; so.dt_initial = o.dt_initial; so.dt_max = o.dt_max; so.dt_min = o.dt_min; so.Xe = o.material.Xe;
    so.rk3 = o.integrator == MP_SSPRK3;
    so.fixed = t->fixed ? 1 : 0;
    so.snap_end = 0; so.end_reports = 1; so.restore_time = 1;
    return so;
}

mp_status capture_leaves(cudaStream_t s, std::vector<cudaGraphNode_t>& out) {
    cudaStreamCaptureStatus cs;
    const cudaGraphNode_t* deps = nullptr;
    size_t nd = 0;
    MP_CUDA(cudaStreamGetCaptureInfo(s, &cs, nullptr, nullptr, &deps, &nd));
    out.assign(deps, deps + nd);
    return MP_OK;
}

mp_status add_while(cudaGraph_t g, const std::vector<cudaGraphNode_t>& deps, cudaGraphConditionalHandle h,
                    cudaGraphNode_t* node, cudaGraph_t* body) {
    cudaGraphNodeParams p{};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = cudaGraphCondTypeWhile;
    p.conditional.size = 1;
    MP_CUDA(cudaGraphAddNode(node, g, deps.empty() ? nullptr : deps.data(), deps.size(), &p));
    *body = p.conditional.phGraph_out[0];
    return MP_OK;
}

// The graph of up to kGraphSteps steps, the same kernels as do_step:
//   WHILE run:  begin -> WHILE attempt: {attempt, axpy, gate, stage 2,
//               control [, stage 3, control]} -> commit, copy, L(U^{n+1}),
//               control (run condition).
mp_status capture_steps(mp_transport* t, cudaGraph_t g) {
    cudaStream_t s = t->stream;
    const StepOpts so = single_step_opts(t);
    const bool rk3 = so.rk3 != 0;
    cudaGraphConditionalHandle run, attempt;
    MP_CUDA(cudaGraphConditionalHandleCreate(&run, g, 1, cudaGraphCondAssignDefault));
    cudaGraphNode_t run_node, attempt_node;
    cudaGraph_t step_body, attempt_body, tmp;
    MP_TRY(add_while(g, {}, run, &run_node, &step_body));
    MP_CUDA(cudaGraphConditionalHandleCreate(&attempt, step_body, 0, 0));
    const cudaStreamCaptureMode mode = cudaStreamCaptureModeThreadLocal;
    MP_CUDA(cudaStreamBeginCaptureToGraph(s, step_body, nullptr, nullptr, 0, mode));
    ctl_begin_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_hdr, t->d_rep, attempt);
    std::vector<cudaGraphNode_t> leaves;
    MP_TRY(capture_leaves(s, leaves));
    MP_CUDA(cudaStreamEndCapture(s, &tmp));
    MP_TRY(add_while(step_body, leaves, attempt, &attempt_node, &attempt_body));
    const size_t o0 = own_begin(t), on = own_count(t);
    const int per_block = sum_cells_per_block((long long)on), nblk_axpy = (int)((on + per_block - 1) / per_block);
    MP_CUDA(cudaStreamBeginCaptureToGraph(s, attempt_body, nullptr, nullptr, 0, mode));
    ctl_attempt_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_hdr, t->d_gate, t->d_dt);
    axpy_kernel<<<nblk_axpy, kRedBlock, 0, s>>>((int)on, t->H + o0, t->C + o0, t->LH + o0, t->LC + o0, 0.0,
                                                 t->host_tab.area, t->S1H + o0, t->S1C + o0, shares_of(t, nblk_axpy),
                                                 t->cell_area ? t->cell_area + o0 : nullptr, t->d_dt, t->d_gate);
    ctl_after_axpy_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_tot, t->d_status, t->d_gate);
    MP_TRY(launch_stage(t, t->S1H, t->S1C, SUM_RK, rk3 ? 0.75 : 0.5, rk3 ? 0.25 : 0.5, 0.0, t->S2H, t->S2C, nullptr,
                        t->d_gate, t->d_dt));
    ctl_after_stage_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_tot, t->d_status, t->d_gate, 2, rk3 ? 0 : 1,
                                                      t->d_hdr, attempt);
    if (rk3) {
        MP_TRY(launch_stage(t, t->S2H, t->S2C, SUM_RK, 1.0 / 3.0, 2.0 / 3.0, 0.0, t->S1H, t->S1C, nullptr, t->d_gate,
                            t->d_dt));
        ctl_after_stage_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_tot, t->d_status, t->d_gate, 3, 1,
                                                          t->d_hdr, attempt);
    }
    MP_CUDA(cudaStreamEndCapture(s, &tmp));
    MP_CUDA(cudaStreamBeginCaptureToGraph(s, step_body, &attempt_node, nullptr, 1, mode));
    ctl_commit_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_hdr, t->d_rep, t->d_status, t->d_gate);
    const unsigned cgrid = (unsigned)std::min<size_t>((t->N + kRedBlock - 1) / kRedBlock, 148 * 8);
    commit_kernel<<<cgrid, kRedBlock, 0, s>>>((long long)t->N, rk3 ? t->S1H : t->S2H, rk3 ? t->S1C : t->S2C, t->H,
                                              t->C, t->d_gate);
    MP_TRY(launch_stage(t, t->H, t->C, SUM_STORE_L, 0, 0, 0, t->LH, t->LC, nullptr, t->d_gate, nullptr));
    ctl_after_rhs_kernel<<<1, kCtlThreads, 0, s>>>(t->d_ctl, 1, so, t->d_tot, t->d_status, t->d_rep, t->d_hdr, 1, run);
    MP_CUDA(cudaStreamEndCapture(s, &tmp));
    MP_CUDA(cudaGetLastError());
    return MP_OK;
}

void release_graph(mp_transport* t) {
    if (t->graph_exec) cudaGraphExecDestroy(t->graph_exec);
    if (t->graph) cudaGraphDestroy(t->graph);
    t->graph_exec = nullptr;
    t->graph = nullptr;
    t->graph_gen = 0;
}

// Control records of the device-resident steps.
mp_status ensure_ctl(mp_transport* t) {
    if (!t->d_ctl) {
        MP_CUDA(cudaMalloc((void**)&t->d_ctl, sizeof(InstCtl)));
        MP_CUDA(cudaMalloc((void**)&t->d_hdr, sizeof(CtlHeader)));
        MP_CUDA(cudaMalloc((void**)&t->d_rep, kGraphSteps * sizeof(mp_step_report)));
        MP_CUDA(cudaMalloc((void**)&t->d_gate, sizeof(int)));
        MP_CUDA(cudaMalloc((void**)&t->d_dt, sizeof(double)));
        MP_CUDA(cudaMallocHost((void**)&t->h_ctl, sizeof(InstCtl)));
        MP_CUDA(cudaMallocHost((void**)&t->h_hdr, sizeof(CtlHeader)));
        MP_CUDA(cudaMallocHost((void**)&t->h_rep, kGraphSteps * sizeof(mp_step_report)));
    }
    return MP_OK;
}

// The handle as the one-kernel form of the steps takes it.
SmallMesh small_mesh(mp_transport* t) {
    SmallMesh m{};
    m.nx = t->nx; m.ny = t->ny; m.tab = &t->host_tab; m.ph = &t->ph; m.quad = t->quad; m.q = t->qdev;
    m.cell_area = t->cell_area;
    m.H = t->H; m.C = t->C; m.S1H = t->S1H; m.S1C = t->S1C; m.S2H = t->S2H; m.S2C = t->S2C; m.LH = t->LH; m.LC = t->LC;
    m.T = t->T; m.phi = t->phi; m.rec = static_cast<double*>(t->rec); m.face = t->face; m.rate = t->rate;
    m.flags = t->flags; m.vsn = t->vsn; m.udn = t->udn; m.partial = t->partial; m.status = t->d_status;
    m.ctl = t->d_ctl; m.hdr = t->d_hdr; m.reports = t->d_rep; m.opts = single_step_opts(t);
    return m;
}

mp_status ensure_graph(mp_transport* t) {
    if (t->graph_exec && t->graph_gen == t->gen) return MP_OK;
    release_graph(t);
    MP_CUDA(cudaGraphCreate(&t->graph, 0));
    // Capture on a private stream (the caller's may be the legacy default
    // stream, which cannot be captured); the graph runs on the caller's.
    cudaStream_t cap = nullptr;
    MP_CUDA(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
    cudaStream_t user = t->stream;
    t->stream = cap;
    g_capturing = true;
    const mp_status st = capture_steps(t, t->graph);
    g_capturing = false;
    cudaStreamCaptureStatus cs;
    if (cudaStreamIsCapturing(cap, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) {
        cudaGraph_t tmp;
        cudaStreamEndCapture(cap, &tmp);
    }
    t->stream = user;
    cudaStreamDestroy(cap);
    if (st != MP_OK) {
        release_graph(t);
        return st;
    }
    MP_CUDA(cudaGraphInstantiate(&t->graph_exec, t->graph, 0));
    t->graph_gen = t->gen;
    return MP_OK;
}

// T and phi of stage `which` (2, 3) of a failed step, from the records that
// the stage left: the latest evaluation, whose averages the step left out.
mp_status complete_averages(mp_transport* t, int which) {
    const double* H = which == 2 ? t->S1H : t->S2H;
    const double* C = which == 2 ? t->S1C : t->S2C;
    const long long N = (long long)t->N;
    const unsigned g = (unsigned)((N + 127) / 128);
    if (t->quad) {
        QuadStageArgs a;
        a.nx = t->nx; a.ny = t->ny; a.gj0 = 0; a.gny = t->ny;
        a.H = H; a.C = C; a.rec = static_cast<double*>(t->rec); a.flags = t->flags; a.T = t->T; a.phi = t->phi;
        a.status = t->d_status; a.q = t->qdev;
        a.src = SourcePtrs{t->cvs_y, t->cud_y, t->srcH, t->srcR, t->srcS};
        quad_cellphase_kernel<<<g, 128, 0, t->stream>>>(a, t->ph, 0, N, 1, nullptr);
    } else {
        CellPhaseArgs a{t->nx, t->ny, nullptr, H, C, static_cast<double*>(t->rec), t->flags, t->T, t->phi, t->d_status, 0, 0,
                        t->cvs_y, t->cud_y, t->srcH, t->srcR, t->srcS};
        if (t->ph.litho || t->ph.source)
            cellphase_kernel<true><<<g, 128, t->ph.source ? kSourceBufBytes : 0, t->stream>>>(a, t->ph, t->ptab, 0, N, 1);
        else
            cellphase_kernel<false><<<g, 128, 0, t->stream>>>(a, t->ph, t->ptab, 0, N, 1);
    }
    count_launch();
    MP_CUDA(cudaGetLastError());
    return reset_status(t);
}

// The host loop's message for the failure the controller recorded.
mp_status graph_failure(mp_transport* t, const InstCtl& c) {
    switch (c.fail) {
    case FAIL_STAGE:
        *t->h_status = c.word;
        return check_status(t, "RHS");
    case FAIL_RATE: set_error("RHS: nonfinite coupled stage rate"); return MP_ERR_FP;
    case FAIL_RETRIES: set_error("Coupled step cannot satisfy admissibility/CFL above minimum step"); return MP_ERR_NOT_CONVERGED;
    case FAIL_FIXED_LIMIT: set_error("Fixed time step exceeds the phase-coupled CFL bound; use control: cfl"); return MP_ERR_ARG_OUTOFRANGE;
    case FAIL_FIXED_STAGE: set_error("Fixed coupled step failed stage admissibility/CFL"); return MP_ERR_ARG_OUTOFRANGE;
    case FAIL_BALANCE:
        set_error("Coupled finite-volume conservation balance failed (H %.3e, C %.3e)", c.bal_H, c.bal_C);
        return MP_ERR_PLIB;
    default: set_error("step failed"); return (mp_status)c.status;
    }
}

// nsteps accepted steps on the device: one graph launch and one host wait
// per kGraphSteps steps. Same decisions, results and reports as the host
// loop of mp_transport_step.
mp_status graph_steps(mp_transport* t, int nsteps, mp_step_report* reports) {
    NvtxRange range("mp_transport steps (device-resident graph)");
    if (!t->have_L) MP_TRY(eval_current(t));
    MP_TRY(ensure_ctl(t));
    const SmallMesh sm = small_mesh(t);
    if (t->small_gen != t->gen) {
        t->small_blocks = t->range.gny == 0 ? small_steps_blocks(sm) : 0;
        t->small_gen = t->gen;
    }
    const bool small = t->small_blocks > 0;
    if (!small) MP_TRY(ensure_graph(t));
    cudaStream_t s = t->stream;
    // Kernels of one stage evaluation: reconstruction, cell phase, faces,
    // sums (a quad mesh: WENO and limiter apart, one more).
    const int sk = (t->quad ? 5 : 4) + (t->ph.diffusion ? 1 : 0);
    const bool rk3 = t->opts.integrator == MP_SSPRK3;
    for (int done = 0; done < nsteps; done += kGraphSteps) {
        const int chunk = std::min(kGraphSteps, nsteps - done);
        InstCtl& c = *t->h_ctl;
        c = InstCtl{};
        c.used = 1; c.time = t->time; c.t_end = t->t_end; c.accepted = t->accepted; c.have_L = 1; c.cur = t->curTot;
        *t->h_hdr = CtlHeader{0, chunk, 0, 0, 0};
        MP_CUDA(cudaMemcpyAsync(t->d_ctl, t->h_ctl, sizeof(InstCtl), cudaMemcpyHostToDevice, s));
        MP_CUDA(cudaMemcpyAsync(t->d_hdr, t->h_hdr, sizeof(CtlHeader), cudaMemcpyHostToDevice, s));
        if (small) MP_TRY(launch_small_steps(sm, t->small_blocks, s));
        else MP_CUDA(cudaGraphLaunch(t->graph_exec, s));
        MP_CUDA(cudaMemcpyAsync(t->h_ctl, t->d_ctl, sizeof(InstCtl), cudaMemcpyDeviceToHost, s));
        MP_CUDA(cudaMemcpyAsync(t->h_hdr, t->d_hdr, sizeof(CtlHeader), cudaMemcpyDeviceToHost, s));
        MP_CUDA(cudaMemcpyAsync(t->h_rep, t->d_rep, (size_t)chunk * sizeof(mp_step_report), cudaMemcpyDeviceToHost, s));
        MP_CUDA(cudaStreamSynchronize(s));
        t->host_syncs += 1;
        const CtlHeader h = *t->h_hdr;
        if (small) count_launch();
        else count_launch((unsigned long long)h.step * (4 + sk) + (unsigned long long)h.total_attempts * (3 + (sk + 1) * (rk3 ? 2 : 1)));
        t->time = c.time;
        t->accepted = c.accepted;
        t->curTot = c.cur;
        t->have_L = c.have_L != 0 && c.status == 0;
        if (c.status) {
            int k = 0;
            while (k < h.step - 1 && t->h_rep[k].status == 0) ++k;
            if (reports) {
                std::memcpy(reports + done, t->h_rep, (size_t)k * sizeof(mp_step_report));
                reports[done + k] = mp_step_report{};
                reports[done + k].status = c.status;
            }
            t->have_L = false;
            if (c.evaluated) MP_TRY(complete_averages(t, c.evaluated));
            return graph_failure(t, c);
        }
        if (reports) std::memcpy(reports + done, t->h_rep, (size_t)chunk * sizeof(mp_step_report));
    }
    return MP_OK;
}

}  // namespace
}  // namespace mp

// -------------------------------------------------------------------- C ABI

namespace mp {
// The option checks every transport entry point makes before any device work
// (time controls, integrator, diffusivity, precision, boundary policies, the
// material's derived scales and the inflow composition), so one options
// struct is accepted or rejected alike by all of them.
mp_status validate_opts(const mp_transport_opts& o, mp_derived* der_out) {
    if (!(o.cfl > 0 && o.cfl <= 1)) { set_error("Coupled CFL must be in (0,1]"); return MP_ERR_ARG_OUTOFRANGE; }
    if (o.integrator != MP_SSPRK2 && o.integrator != MP_SSPRK3) { set_error("integrator must be 2 or 3"); return MP_ERR_ARG_OUTOFRANGE; }
    if (!(std::isfinite(o.diffusivity) && o.diffusivity >= 0.0)) { set_error("Diffusivity must be finite and nonnegative"); return MP_ERR_ARG_OUTOFRANGE; }
    if (o.precision != MP_PRECISION_FP64 && o.precision != MP_PRECISION_MIXED) { set_error("unknown precision"); return MP_ERR_ARG_OUTOFRANGE; }
    if (o.H_policy < 0 || o.H_policy > 2 || o.C_policy < 0 || o.C_policy > 2) { set_error("unknown boundary policy"); return MP_ERR_ARG_OUTOFRANGE; }
    mp_derived der;
    MP_TRY(derive_checked(o.material, der));
    if (!(o.inflow_C >= 0 && o.inflow_C <= o.material.Xe)) { set_error("Composition must lie in [0, phase.parameters.Xe]"); return MP_ERR_ARG_OUTOFRANGE; }
    if (der_out) *der_out = der;
    return MP_OK;
}
}  // namespace mp

namespace {
// A whole mesh (slab = false) or the row slab [row_begin, row_end) of `mesh`.
mp_status create_impl(const mp_mesh_desc* mesh, bool slab, int row_begin, int row_end, const mp_transport_opts* opts,
                      mp_stream_t stream, mp_transport** out, const double* xy = nullptr) {
    using namespace mp;
    if (!mesh || !opts || !out) { set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (mesh->nx < 2 || mesh->ny < 2) { set_error("Transport requires at least 2x2 cells"); return MP_ERR_ARG_SIZ; }
    if (mesh_too_large(mesh->nx, mesh->ny)) { set_error("mesh has 2^31 edges or more"); return MP_ERR_ARG_SIZ; }
    mp_derived der;
    MP_TRY(validate_opts(*opts, &der));
    QuadTables qt;
    if (xy) {
        long long bad = -1;
        if (validate_quads(mesh->nx, mesh->ny, xy, &bad)) {
            set_error("Mesh has non-real/non-finite coordinates or an inverted, degenerate, or nearly singular "
                      "quadrilateral (cell %lld)", bad);
            return MP_ERR_ARG_WRONG;
        }
    }
    if (slab && !(row_begin >= 0 && row_begin < row_end && row_end <= mesh->ny)) {
        set_error("slab rows [%d, %d) outside [0, %d)", row_begin, row_end, mesh->ny);
        return MP_ERR_ARG_OUTOFRANGE;
    }
    mp_transport* t = new mp_transport;
    t->mesh = *mesh; t->opts = *opts; t->der = der;
    t->stream = (cudaStream_t)stream;
    t->nx = mesh->nx; t->ny = mesh->ny;
    if (slab) {
        // Two halo rows where the global mesh continues (3x3 gathers of the
        // reconstructed halo row reach the second one).
        const int hb = std::min(2, row_begin), ht = std::min(2, mesh->ny - row_end);
        t->ny = (row_end - row_begin) + hb + ht;
        t->range.gj0 = row_begin - hb;
        t->range.gny = mesh->ny;
        t->range.own0 = hb;
        t->range.own1 = hb + (row_end - row_begin);
        t->range.rec0 = hb > 0 ? hb - 1 : 0;
        t->range.rec1 = ht > 0 ? t->range.own1 + 1 : t->range.own1;
    } else {
        t->range = whole(mesh->ny);
    }
    if (xy) {
        // Vertices and edge spacing of the local rows on the host; the
        // per-cell tables are built on the GPU below.
        const int qs = build_quad_tables(mesh->nx, mesh->ny, xy, 0, qt, t->range.gj0, t->ny, false);
        if (qs) { delete t; set_error("per-cell stencil table construction failed"); return (mp_status)qs; }
    }
    t->N = (size_t)t->nx * t->ny;
    t->NE = (size_t)t->nx * (t->ny + 1) + (size_t)(t->nx + 1) * t->ny;
    t->ph.k = phase_const(opts->material, der);
    t->ph.sk = stage_const(t->ph.k);
    double Tep;
    if (eutectic_temperature(t->ph.k, opts->pressure, Tep)) { delete t; set_error("pressure must be finite"); return MP_ERR_ARG_OUTOFRANGE; }
    t->ph.Tep = Tep; t->ph.theta = opts->theta;
    t->ph.inflowH = opts->inflow_H; t->ph.inflowC = opts->inflow_C;
    t->ph.Hpol = opts->H_policy; t->ph.Cpol = opts->C_policy;
    t->ph.lf_global = opts->lf_global; t->ph.lf_speed = opts->lf_global_speed;
    t->ph.kappa = opts->diffusivity;
    for (int w = 0; w < 4; ++w) { t->ph.wall_type[w] = 0; t->ph.wall_value[w] = 0.0; }
    t->ph.diffusion = opts->diffusivity > 0.0;
    t->ph.litho = 0; t->ph.tep_a = t->ph.tep_b = t->ph.surface = 0.0;
    t->ph.source = opts->material.alpha0 != 0.0;
    t->ph.cooling = opts->material.alpha0 * der.l0 * opts->material.g / opts->material.cp;
    const int tb = build_stage_tables(mesh->nx, mesh->ny, mesh->x0, mesh->x1, mesh->y0, mesh->y1, t->host_tab);
    if (tb) { delete t; set_error("stencil table construction failed"); return (mp_status)tb; }
    make_param_tables(t->host_tab, t->ptab);
    const int per_block = sum_cells_per_block((long long)own_count(t));
    t->sum_blocks = (int)((own_count(t) + per_block - 1) / per_block);
    const size_t N = t->N, NE = t->NE;
    cudaError_t e = cudaSuccess;
    if (t->ph.source)
        e = cudaFuncSetAttribute(cellphase_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSourceBufBytes);
    auto alloc = [&](void** p, size_t bytes) { if (e == cudaSuccess) e = cudaMalloc(p, bytes); };
    for (double** p : {&t->H, &t->C, &t->S1H, &t->S1C, &t->S2H, &t->S2C, &t->LH, &t->LC, &t->T, &t->phi, &t->rate})
        alloc((void**)p, N * sizeof(double));
    alloc((void**)&t->rec, rec_doubles(N) * sizeof(double));
    alloc((void**)&t->flags, N);
    alloc((void**)&t->vsn, NE * kNQ * sizeof(double));
    alloc((void**)&t->udn, NE * kNQ * sizeof(double));
    alloc((void**)&t->face, 4 * NE * sizeof(double));
    alloc((void**)&t->partial, (size_t)std::max(t->sum_blocks, 1) * sizeof(Partial));
    alloc((void**)&t->d_tot, sizeof(Totals));
    alloc((void**)&t->d_ticket, sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemsetAsync(t->d_ticket, 0, sizeof(unsigned), t->stream);
    alloc((void**)&t->d_status, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMallocHost((void**)&t->h_tot, sizeof(Totals));
    if (e == cudaSuccess) e = cudaMallocHost((void**)&t->h_status, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemsetAsync(t->vsn, 0, NE * kNQ * sizeof(double), t->stream);
    if (e == cudaSuccess) e = cudaMemsetAsync(t->udn, 0, NE * kNQ * sizeof(double), t->stream);
    if (xy && e == cudaSuccess) {
        // Per-cell tables of a general quad mesh, one allocation: vertices of
        // the local rows and edge spacing from the host, the cell tables
        // built on the GPU from the whole mesh's vertices.
        const int gs = upload_quad_tables(mesh->nx, mesh->ny, xy, qt, t->range.gj0, t->ny, t->stream, &t->qbuf, t->qdev,
                                          &e);
        t->cell_area = t->qdev.geo + 3 * N;
        t->quad = true;
        if (gs == MP_ERR_ARG_WRONG) {
            free_all(t); delete t;
            set_error("per-cell stencil table construction failed (singular stencil or degenerate cell)");
            return (mp_status)gs;
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    if (e != cudaSuccess) { free_all(t); delete t; return cuda_status(e, "mp_transport_create"); }
    *out = t;
    return MP_OK;
}
}  // namespace

extern "C" mp_status mp_transport_create(const mp_mesh_desc* mesh, const mp_transport_opts* opts, mp_stream_t stream,
                                         mp_transport** out) {
    return create_impl(mesh, false, 0, 0, opts, stream, out);
}

extern "C" mp_status mp_transport_create_quads(const mp_mesh_desc* mesh, const double* xy, const mp_transport_opts* opts,
                                               mp_stream_t stream, mp_transport** out) {
    if (!xy) { mp::set_error("null vertex array"); return MP_ERR_ARG_WRONG; }
    return create_impl(mesh, false, 0, 0, opts, stream, out, xy);
}

extern "C" size_t mp_transport_instance_bytes(const mp_mesh_desc* mesh, int quads) {
    using namespace mp;
    if (!mesh || mesh->nx < 2 || mesh->ny < 2 || mesh_too_large(mesh->nx, mesh->ny)) return 0;
    const size_t nx = (size_t)mesh->nx, ny = (size_t)mesh->ny, N = nx * ny;
    const size_t NE = nx * (ny + 1) + (nx + 1) * ny;
    // Each array is its own cudaMalloc, which takes whole 2 MiB pages; the
    // small control and reduction buffers share one more page.
    const size_t page = (size_t)2 << 20;
    auto pages = [&](size_t bytes) { return (bytes + page - 1) / page * page; };
    size_t b = 11 * pages(N * sizeof(double))                   // state, stage buffers, L, T, phi, rate
             + pages(rec_doubles(N) * sizeof(double)) + pages(N)   // records, flags
             + 2 * pages(NE * kNQ * sizeof(double)) + pages(4 * NE * sizeof(double))   // velocities, face values
             + pages((N / sum_cells_per_block((long long)N) + 1) * sizeof(Partial)) + page;
    if (quads) {
        const size_t V = 2 * (nx + 1) * (ny + 1);
        // Per-cell tables and geometry (an upper bound, kQBudget), vertices
        // and edge spacing in one allocation; the builder's copy of the
        // vertices is held while the tables are built.
        b += pages(((size_t)kQBudget * N + V + NE * kNQ) * sizeof(double)) +
             pages(V * sizeof(double) + sizeof(int));
    }
    return b;
}

extern "C" mp_status mp_transport_create_quads_slab(const mp_mesh_desc* global_mesh, const double* xy, int row_begin,
                                                    int row_end, const mp_transport_opts* opts, mp_stream_t stream,
                                                    mp_transport** out) {
    if (!xy) { mp::set_error("null vertex array"); return MP_ERR_ARG_WRONG; }
    return create_impl(global_mesh, true, row_begin, row_end, opts, stream, out, xy);
}

extern "C" mp_status mp_mesh_vertices(const mp_mesh_desc* mesh, int family, double perturbation, unsigned long long seed,
                                      double* xy) {
    if (!mesh || !xy) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    const int st = mp::mesh_vertices(mesh->nx, mesh->ny, mesh->x0, mesh->x1, mesh->y0, mesh->y1, family, perturbation,
                                     seed, xy);
    if (st) mp::set_error("mesh: unknown family, non-finite or empty domain, or perturbation outside [0, 0.25)");
    return (mp_status)st;
}

extern "C" mp_status mp_transport_create_slab(const mp_mesh_desc* global_mesh, int row_begin, int row_end,
                                              const mp_transport_opts* opts, mp_stream_t stream, mp_transport** out) {
    return create_impl(global_mesh, true, row_begin, row_end, opts, stream, out);
}

extern "C" mp_status mp_transport_slab_layout(const mp_transport* t, int* local_rows, int* row0, int* own_begin,
                                              int* own_end) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (local_rows) *local_rows = t->ny;
    if (row0) *row0 = t->range.gj0;
    if (own_begin) *own_begin = t->range.own0;
    if (own_end) *own_end = t->range.own1;
    return MP_OK;
}

extern "C" mp_status mp_transport_set_hooks(mp_transport* t, mp_halo_fn halo, mp_combine_fn combine, void* user) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    t->halo = halo;
    t->combine = combine;
    t->hook_user = user;
    t->have_L = false;
    t->gen += 1;
    return MP_OK;
}

extern "C" void mp_transport_destroy(mp_transport* t) {
    if (!t) return;
    cudaStreamSynchronize(t->stream);
    mp::free_all(t);
    delete t;
}

extern "C" mp_status mp_transport_set_face_velocity(mp_transport* t, const double* vs_n, const double* ud_n) {
    if (!t || !vs_n || !ud_n) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    const size_t bytes = t->NE * mp::kNQ * sizeof(double);
    MP_CUDA(cudaMemcpyAsync(t->vsn, vs_n, bytes, cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaMemcpyAsync(t->udn, ud_n, bytes, cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaStreamSynchronize(t->stream));
    t->have_L = false;
    return MP_OK;
}

extern "C" mp_status mp_transport_set_state(mp_transport* t, const double* H, const double* C, double time) {
    if (!t || !H || !C) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (!std::isfinite(time)) { mp::set_error("Nonfinite source time"); return MP_ERR_ARG_OUTOFRANGE; }
    const size_t o0 = mp::own_begin(t), ob = mp::own_count(t) * sizeof(double);
    MP_CUDA(cudaMemcpyAsync(t->H + o0, H, ob, cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaMemcpyAsync(t->C + o0, C, ob, cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaStreamSynchronize(t->stream));
    t->time = time;
    t->accepted = 0;
    t->have_L = false;
    return MP_OK;
}

extern "C" mp_status mp_transport_get_state(mp_transport* t, double* H, double* C, double* T, double* phi) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    const size_t o0 = mp::own_begin(t), b = mp::own_count(t) * sizeof(double);
    if (H) MP_CUDA(cudaMemcpyAsync(H, t->H + o0, b, cudaMemcpyDefault, t->stream));
    if (C) MP_CUDA(cudaMemcpyAsync(C, t->C + o0, b, cudaMemcpyDefault, t->stream));
    if (T) MP_CUDA(cudaMemcpyAsync(T, t->T + o0, b, cudaMemcpyDefault, t->stream));
    if (phi) MP_CUDA(cudaMemcpyAsync(phi, t->phi + o0, b, cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaStreamSynchronize(t->stream));
    return MP_OK;
}

extern "C" mp_status mp_transport_rhs(mp_transport* t, double* rhsH, double* rhsC, double* T, double* phi, double* rate,
                                      mp_stage_totals* totals) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    MP_TRY(mp::eval_current(t));
    const size_t o0 = mp::own_begin(t), b = mp::own_count(t) * sizeof(double);
    if (rhsH) MP_CUDA(cudaMemcpyAsync(rhsH, t->LH + o0, b, cudaMemcpyDefault, t->stream));
    if (rhsC) MP_CUDA(cudaMemcpyAsync(rhsC, t->LC + o0, b, cudaMemcpyDefault, t->stream));
    if (T) MP_CUDA(cudaMemcpyAsync(T, t->T + o0, b, cudaMemcpyDefault, t->stream));
    if (phi) MP_CUDA(cudaMemcpyAsync(phi, t->phi + o0, b, cudaMemcpyDefault, t->stream));
    if (rate) MP_CUDA(cudaMemcpyAsync(rate, t->rate + o0, b, cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaStreamSynchronize(t->stream));
    if (totals) {
        totals->boundaryH = t->curTot.bH; totals->boundaryC = t->curTot.bC; totals->sourceH = t->curTot.sH;
        totals->maxRate = t->curTot.maxRate; totals->divergence = t->curTot.divergence;
    }
    return MP_OK;
}

extern "C" mp_status mp_transport_step(mp_transport* t, int nsteps, mp_step_report* reports) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (nsteps < 0) { mp::set_error("nsteps must be nonnegative"); return MP_ERR_ARG_OUTOFRANGE; }
    if (nsteps > 0 && mp::graph_usable(t)) return mp::graph_steps(t, nsteps, reports);
    for (int k = 0; k < nsteps; ++k) {
        // At the end time (within 32 ulp of it, evolve.cpp:450-451) stepping stops;
        // the remaining reports keep dt = 0 and the end time.
        if (std::isfinite(t->t_end) &&
            t->t_end - t->time <= 32 * std::numeric_limits<double>::epsilon() * std::max(1.0, std::fabs(t->t_end))) {
            t->time = t->t_end;
            if (reports)
                for (int r = k; r < nsteps; ++r) { reports[r] = mp_step_report{}; reports[r].time = t->time; }
            return MP_OK;
        }
        mp_step_report rep{};
        const double t0 = t->time;
        const mp_status s = mp::do_step(t, rep);
        if (s != MP_OK) {
            // The accepted state (t->H, t->C) is untouched until commit; restore the clock.
            t->time = t0;
            t->have_L = false;
            if (reports) { reports[k] = mp_step_report{}; reports[k].status = s; }
            return s;
        }
        if (reports) reports[k] = rep;
    }
    return MP_OK;
}

extern "C" mp_status mp_transport_set_time_control(mp_transport* t, int control, double t_end) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (control != MP_TIME_CFL && control != MP_TIME_FIXED) { mp::set_error("unknown time control %d", control); return MP_ERR_ARG_OUTOFRANGE; }
    if (std::isnan(t_end)) { mp::set_error("end time must not be NaN"); return MP_ERR_ARG_OUTOFRANGE; }
    if (control == MP_TIME_FIXED && !(t->opts.dt_initial > 0 && std::isfinite(t->opts.dt_initial))) {
        mp::set_error("fixed control needs a positive finite dt_initial");
        return MP_ERR_ARG_OUTOFRANGE;
    }
    t->fixed = control == MP_TIME_FIXED;
    t->t_end = t_end;
    t->gen += 1;
    return MP_OK;
}

extern "C" mp_status mp_transport_set_thermal_bc(mp_transport* t, const int* type, const double* value) {
    if (!t || !type || !value) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    for (int w = 0; w < 4; ++w) {
        if (type[w] < MP_THERMAL_ZERO_FLUX || type[w] > MP_THERMAL_FLUX) { mp::set_error("unknown thermal condition %d", type[w]); return MP_ERR_ARG_WRONG; }
        if (type[w] != MP_THERMAL_ZERO_FLUX && !std::isfinite(value[w])) { mp::set_error("Boundary data must be finite"); return MP_ERR_ARG_OUTOFRANGE; }
    }
    bool flux = false;
    for (int w = 0; w < 4; ++w) {
        t->ph.wall_type[w] = type[w];
        t->ph.wall_value[w] = type[w] == MP_THERMAL_ZERO_FLUX ? 0.0 : value[w];
        flux = flux || type[w] == MP_THERMAL_FLUX;
    }
    t->ph.diffusion = t->ph.kappa > 0.0 || flux;
    t->have_L = false;
    t->gen += 1;
    return MP_OK;
}

extern "C" mp_status mp_transport_set_pressure_model(mp_transport* t, int model, double value) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (!std::isfinite(value)) { mp::set_error("pressure model value must be finite"); return MP_ERR_ARG_OUTOFRANGE; }
    if (model == MP_PRESSURE_CONSTANT) {
        if (value < 0) { mp::set_error("pressure must be nonnegative Pa"); return MP_ERR_ARG_OUTOFRANGE; }
        double Tep;
        if (mp::eutectic_temperature(t->ph.k, value, Tep)) { mp::set_error("pressure-corrected temperature is not representable"); return MP_ERR_PHASE_OVERFLOW; }
        t->opts.pressure = value;
        t->ph.Tep = Tep;
        t->ph.litho = 0;
    } else if (model == MP_PRESSURE_LITHOSTATIC) {
        const double top = t->range.gny > 0 ? t->mesh.y1 : t->mesh.y1;
        if (value < top) { mp::set_error("surface_y must be at or above the mesh top"); return MP_ERR_ARG_OUTOFRANGE; }
        // Tep(y) = TDe0 + rho g l0 (surface - y) / nu / dT (eutectic_rescaled.cpp:143-161).
        const long double b = (long double)t->opts.material.rho * t->opts.material.g * t->der.l0 /
                              t->opts.material.nu / t->der.dT;
        t->ph.litho = 1;
        t->ph.tep_a = t->der.TDe0;
        t->ph.tep_b = (double)b;
        t->ph.surface = value;
    } else {
        mp::set_error("unknown pressure model %d", model);
        return MP_ERR_ARG_OUTOFRANGE;
    }
    t->have_L = false;
    t->gen += 1;
    return MP_OK;
}

extern "C" mp_status mp_transport_set_cell_velocity(mp_transport* t, const double* vs_y, const double* ud_y) {
    if (!t || !vs_y || !ud_y) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    const size_t n = t->N * mp::kNQ * mp::kNQ;
    cudaError_t e = cudaSuccess;
    for (double** p : {&t->cvs_y, &t->cud_y})
        if (!*p && e == cudaSuccess) e = cudaMalloc(p, n * sizeof(double));
    for (double** p : {&t->srcH, &t->srcR, &t->srcS})
        if (!*p && e == cudaSuccess) e = cudaMalloc(p, t->N * sizeof(double));
    if (e != cudaSuccess) return mp::cuda_status(e, "mp_transport_set_cell_velocity");
    MP_CUDA(cudaMemcpyAsync(t->cvs_y, vs_y, n * sizeof(double), cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaMemcpyAsync(t->cud_y, ud_y, n * sizeof(double), cudaMemcpyDefault, t->stream));
    MP_CUDA(cudaMemsetAsync(t->srcH, 0, t->N * sizeof(double), t->stream));
    MP_CUDA(cudaMemsetAsync(t->srcR, 0, t->N * sizeof(double), t->stream));
    MP_CUDA(cudaMemsetAsync(t->srcS, 0, t->N * sizeof(double), t->stream));
    MP_CUDA(cudaStreamSynchronize(t->stream));
    t->have_L = false;
    t->gen += 1;
    return MP_OK;
}

extern "C" mp_status mp_transport_get_time(const mp_transport* t, double* time, int* accepted) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    if (time) *time = t->time;
    if (accepted) *accepted = t->accepted;
    return MP_OK;
}

extern "C" mp_status mp_transport_limiter(mp_transport* t, double* thetaH, double* thetaC) {
    if (!t || !thetaH || !thetaC) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    double* theta = nullptr;
    MP_CUDA(cudaMalloc(&theta, 2 * t->N * sizeof(double)));
    const mp_status s = mp::eval_current(t, theta);
    cudaError_t e = cudaSuccess;
    const size_t o0 = mp::own_begin(t), ob = mp::own_count(t) * sizeof(double);
    if (s == MP_OK) e = cudaMemcpyAsync(thetaH, theta + o0, ob, cudaMemcpyDefault, t->stream);
    if (s == MP_OK && e == cudaSuccess) e = cudaMemcpyAsync(thetaC, theta + t->N + o0, ob, cudaMemcpyDefault, t->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(t->stream);
    cudaFree(theta);
    if (s != MP_OK) return s;
    return mp::cuda_status(e, "mp_transport_limiter");
}

extern "C" mp_status mp_transport_profile(mp_transport* t, int enable) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    MP_CUDA(cudaStreamSynchronize(t->stream));
    mp::harvest(t);
    t->profile = enable != 0;
    for (int k = 0; k < 6; ++k) { t->kern_ms[k] = 0; t->kern_n[k] = 0; }
    return MP_OK;
}

extern "C" mp_status mp_transport_kernel_times(mp_transport* t, double* ms, unsigned long long* launches) {
    if (!t || !ms || !launches) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    MP_CUDA(cudaStreamSynchronize(t->stream));
    mp::harvest(t);
    for (int k = 0; k < 6; ++k) { ms[k] = t->kern_ms[k]; launches[k] = t->kern_n[k]; }
    return MP_OK;
}

namespace mp {
namespace {
// Independent FP64 FMA chains: 8 per thread, unrolled.
__global__ void fp64_probe_kernel(double* out, int iters, double a, double b) {
    double x[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) x[k] = threadIdx.x * 1e-9 + k;
    for (int it = 0; it < iters; ++it) {
#pragma unroll
        for (int k = 0; k < 8; ++k) x[k] = fma(x[k], a, b);
    }
    double s = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) s += x[k];
    if (s == 12345.678) out[0] = s;   // keep the chains live
}
}  // namespace
}  // namespace mp

extern "C" mp_status mp_probe_fp64_peak(mp_stream_t stream, double* tflops) {
    if (!tflops) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    cudaStream_t s = (cudaStream_t)stream;
    int dev = 0, sms = 0;
    MP_CUDA(cudaGetDevice(&dev));
    MP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    double* out = nullptr;
    MP_CUDA(cudaMalloc(&out, sizeof(double)));
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0); cudaEventCreate(&e1);
    const int threads = 256, blocks = sms * 8, iters = 4096;
    mp::fp64_probe_kernel<<<blocks, threads, 0, s>>>(out, 64, 0.999999, 1e-7);   // warm-up
    cudaEventRecord(e0, s);
    mp::fp64_probe_kernel<<<blocks, threads, 0, s>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e1, s);
    mp::count_launch(2);
    cudaError_t e = cudaEventSynchronize(e1);
    float ms = 0.f;
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0); cudaEventDestroy(e1); cudaFree(out);
    if (e != cudaSuccess) return mp::cuda_status(e, "mp_probe_fp64_peak");
    *tflops = 2.0 * 8.0 * iters * (double)threads * blocks / (ms * 1e-3) / 1e12;
    return MP_OK;
}

// ------------------------------------------------ stage on caller buffers

namespace mp {

size_t raw_partial_bytes(size_t ncell) {
    const size_t per = (size_t)sum_cells_per_block((long long)ncell);
    return (ncell + per - 1) / per * sizeof(Partial);
}
size_t raw_totals_bytes() { return sizeof(Totals) + sizeof(unsigned); }

// One stage evaluation L(U) (STORE_L mode) on buffers the caller provides:
// tab (host StageTables, passed to the kernels by value), rec (18 doubles per
// cell, cells rounded up to 32), wet (ncell bytes), face
// (4*nedge doubles), partial (raw_partial_bytes), totals (raw_totals_bytes),
// status (one unsigned long long). Used by entry points that cannot allocate.
mp_status stage_rhs_raw(int nx, int ny, const mp_transport_opts& o, const double* H, const double* C,
                        const double* vsn, const double* udn, double* rhsH, double* rhsC, double* T, double* phi,
                        double* rate, const StageTables& tab, double* rec, unsigned char* wet, double* face, void* partial,
                        void* totals, unsigned long long* status, mp_stage_totals* out, cudaStream_t s) {
    mp_derived der;
    MP_TRY(derive_checked(o.material, der));
    Physics ph;
    ph.k = phase_const(o.material, der);
    ph.sk = stage_const(ph.k);
    if (eutectic_temperature(ph.k, o.pressure, ph.Tep)) { set_error("pressure must be finite"); return MP_ERR_ARG_OUTOFRANGE; }
    ph.theta = o.theta; ph.inflowH = o.inflow_H; ph.inflowC = o.inflow_C;
    ph.Hpol = o.H_policy; ph.Cpol = o.C_policy; ph.lf_global = o.lf_global; ph.lf_speed = o.lf_global_speed;
    ph.diffusion = 0; ph.kappa = 0.0;
    ph.litho = 0; ph.tep_a = ph.tep_b = ph.surface = 0.0;
    ph.source = 0; ph.cooling = 0.0;
    for (int w = 0; w < 4; ++w) { ph.wall_type[w] = 0; ph.wall_value[w] = 0.0; }
    const size_t N = (size_t)nx * ny;
    const size_t NE = (size_t)nx * (ny + 1) + (size_t)(nx + 1) * ny;
    const int per_block = sum_cells_per_block((long long)N), sum_blocks = (int)((N + per_block - 1) / per_block);
    Partial* part = static_cast<Partial*>(partial);
    Totals* tot = static_cast<Totals*>(totals);
    unsigned* ticket = reinterpret_cast<unsigned*>(tot + 1);
    MP_CUDA(cudaMemsetAsync(ticket, 0, sizeof(unsigned), s));
    MP_CUDA(cudaMemsetAsync(status, 0xff, sizeof(unsigned long long), s));
    (void)NE;
    ParamTables pt;
    make_param_tables(tab, pt);
    launch_stage_kernels(nx, ny, whole(ny), pt, ph, H, C, rec, wet, T, phi, vsn, udn, face, status, nullptr, true, s,
                                 nullptr);
    {
        SumArgs a{nx, ny, tab.area, 1.0 / tab.area, face, H, C, H, C, rhsH, rhsC, rate, SUM_STORE_L, 0.0, 0.0, 0.0,
                  Shares{part, tot, ticket, sum_blocks}, nullptr, 0, 0, 0, (long long)N};
        sum_kernel<false><<<sum_blocks, kRedBlock, 0, s>>>(a);
    }
    count_launch(4);
    MP_CUDA(cudaGetLastError());
    Totals host_tot;
    unsigned long long host_status = 0;
    MP_CUDA(cudaMemcpyAsync(&host_tot, tot, sizeof(Totals), cudaMemcpyDeviceToHost, s));
    MP_CUDA(cudaMemcpyAsync(&host_status, status, sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    MP_CUDA(cudaStreamSynchronize(s));
    if (host_status != ~0ULL) {
        const long long cell = (long long)((host_status >> 8) & ((1ULL << 48) - 1));
        set_error("RHS: cell %lld: stage failure (class %d)", cell, (int)(host_status & 0xff));
        return (mp_status)(host_status & 0xff);
    }
    if (!std::isfinite(host_tot.maxRate)) { set_error("RHS: nonfinite coupled stage rate"); return MP_ERR_FP; }
    if (out) {
        out->boundaryH = host_tot.bH; out->boundaryC = host_tot.bC; out->sourceH = 0.0;
        out->maxRate = host_tot.maxRate; out->divergence = host_tot.divergence;
    }
    return MP_OK;
}

}  // namespace mp

extern "C" mp_status mp_transport_set_device_steps(mp_transport* t, int enable) {
    if (!t) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    t->use_graph = enable != 0;
    return MP_OK;
}

extern "C" mp_status mp_transport_run_stats(const mp_transport* t, unsigned long long* host_syncs) {
    if (!t || !host_syncs) { mp::set_error("null argument"); return MP_ERR_ARG_WRONG; }
    *host_syncs = t->host_syncs;
    return MP_OK;
}
