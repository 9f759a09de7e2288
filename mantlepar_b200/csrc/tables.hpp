// Per-mesh tables of the uniform-mesh ML-WENO stage (host-built; the
// kernels read them as a kernel parameter or from global memory).
//
// On a uniform rectangular mesh every interior cell has the same stencil
// geometry up to a translation, so the reference's per-cell setup
// (TensorStencilPoly::Initialize, src/mlweno/tensorstencilpoly.cpp:146-231;
// SetTargetSmoothness :383-398; Reconstruction::Initialize,
// src/mlweno/reconstruction.cpp:109-210; the limiter point set,
// src/couple/state_reconstruction.cpp:152-168; diffusion sample geometry,
// src/mlweno/diffusiveflux.cpp:255-334) collapses to one table set per
// mesh, with nine boundary classes (left/interior/right x bottom/interior/top)
// for the candidate mask and the limiter points. All coordinates are in the
// target cell's own frame xi = (x - x_c)/(dx/2), eta = (y - y_c)/(dy/2), in
// which every cell is [-1, 1]^2 and the candidates' coefficients are plain
// difference quotients of the stencil.
#ifndef MP_TABLES_HPP
#define MP_TABLES_HPP

namespace mp {

constexpr int kNQ = 5;             // Gauss points per edge / per cell axis
constexpr int kMaxLines = 256;     // limiter point lines over all 9 classes

// The fields the stage kernels read, small enough to travel as a kernel
// parameter (constant-bank operands instead of loads).
struct StageHot {
    // Smoothness indicators in the cell's frame, as sigma / epsA. With the
    // half extents in units of h = sqrt(area) Xh = dx/(2h), Yh = dy/(2h)
    // (Xh Yh = 1/4), the order-2 candidate's sigma (the derivatives of orders
    // 1 and 2 over the unit reference square, tensorstencilpoly.cpp:318-398)
    // is a sum of eight squares of its coefficients q_ij:
    //   sg[0] (q10 + cy q12)^2 + sg[1] (q01 + cx q21)^2 + sg[2] (q20 + cy q22)^2
    // + sg[3] (q02 + cx q22)^2 + sg[4] q11^2 + sg[5] q12^2 + sg[6] q21^2 + sg[7] q22^2
    // with cx = 1/(12 Xh^2), cy = 1/(12 Yh^2), and an order-1 candidate's
    // (over the target cell) is gx dE^2 + gy dN^2 + gb (dNE - dE - dN)^2 on
    // the differences to the target.
    double cx, cy, sg[8], gx2, gy2, gb;
    double epsA;            // epsilon * cell area of the weight regulariser
    double epsA2;           // its square
    double area;            // cell area (1-point rule, as MeshInfo::CacheAreas)
    double len_h, len_v;    // lengths of AlongI (horizontal) / AlongJ edges
    double gw[kNQ];         // Gauss weights
    double cw[kNQ * kNQ];   // cell-quadrature weight / area, q = b*5 + a
    double g[kNQ];          // Gauss points: the cell is [-1, 1]^2 in its frame
    // Thermal diffusion by normal-line sampling (diffusiveflux.cpp:203-334)
    // with 4 samples per Gauss point and extent fraction 0.9, for this mesh:
    // derivative weights (interior: middle of 4 nodes; wall: end of 5 nodes),
    // physical spacing [horizontal/vertical edges][interior/wall], physical
    // Gauss weights len*w_q/2 [horizontal/vertical][q], and the coordinate
    // across the edge of each sample in its cell's frame: interior
    // samples k = 0, 1 lie in the left cell, 2, 3 in the right one
    // [horizontal/vertical][k]; wall samples k = 0..3 lie in the wall cell,
    // farthest first [wall: bottom, top, left, right][k].
    double dif_c_int[4];
    double dif_c_bnd[5];
    double dif_ds[2][2];
    double dif_w[2][kNQ];
    double dif_pos_int[2][4];
    double dif_pos_bnd[4][4];
    // Physical height of a point: y = y0 + (row + 0.5) * dy + eta * hn (global
    // row; hn = dy / 2), and the physical cell-quadrature weights w_a w_b |J|
    // (q = b*5 + a).
    double y0, dy, hn;
    double cwp[kNQ * kNQ];
    // Limiter points grouped into 5-point lines: apart from the cell centre,
    // every limiter point lies on a row eta = line_c with xi = g_q, or on a
    // column xi = line_c with eta = g_q (q = 0..4). Class c owns lines
    // [line_off[c], line_off[c+1]); line_dir 0 = row, 1 = column; line_kind
    // 1 = diffusion samples.
    int line_off[10];
    double line_c[kMaxLines];
    unsigned char line_dir[kMaxLines];
    unsigned char line_kind[kMaxLines];
};

using StageTables = StageHot;

// Build the tables of an nx x ny uniform mesh on [x0,x1] x [y0,y1].
// Returns 0 or an mp_status code (mesh extents outside the range of doubles).
int build_stage_tables(int nx, int ny, double x0, double x1, double y0, double y1, StageTables& t);

}  // namespace mp

#endif
