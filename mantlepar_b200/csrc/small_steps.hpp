// Device-resident steps of a small mesh in one kernel (small_steps.cu): what
// the transport handle passes to it.
#ifndef MP_SMALL_STEPS_HPP
#define MP_SMALL_STEPS_HPP

#include "quad_tables.hpp"
#include "stage_kernels.cuh"
#include "step_ctl.cuh"
#include "tables.hpp"

namespace mp {

struct SmallMesh {
    int nx, ny;
    const StageTables* tab;             // host tables of a uniform mesh
    const Physics* ph;                  // host
    bool quad;
    QuadDev q;
    const double* cell_area;            // quad mesh
    // Device buffers of the handle (transport.cu).
    double *H, *C, *S1H, *S1C, *S2H, *S2C, *LH, *LC, *T, *phi, *rec, *face, *rate;
    unsigned char* flags;
    const double *vsn, *udn;
    Partial* partial;
    unsigned long long* status;
    InstCtl* ctl;
    CtlHeader* hdr;
    mp_step_report* reports;
    StepOpts opts;
};

// Blocks of the cluster in which steps of this mesh run as one kernel; 0
// where they do not (too many cells, adiabatic source, no cluster of 8 blocks
// fits the GPU).
int small_steps_blocks(const SmallMesh& m);
// Up to hdr->nsteps steps (ctl and hdr set as for the step graph); one launch.
mp_status launch_small_steps(const SmallMesh& m, int blocks, cudaStream_t stream);

}  // namespace mp

#endif
