// Device helpers of the general (logically rectangular) quad mesh kernels,
// shared by the transport stage and the preheat: vertex reads, the
// reference's edge and bilinear maps (src/core/integral.cpp:62-121), the
// cell frame, the normal-line diffusion samples, the table-driven
// reconstruction of one field, and the edge orientation of the flux loops.
#ifndef MP_QUAD_DEVICE_CUH
#define MP_QUAD_DEVICE_CUH

#include "common.hpp"
#include "quad_tables.hpp"
#include "stage_device.cuh"

namespace mp {
namespace {

struct P2 {
    double x, y;
};

__device__ __forceinline__ P2 vtx(const QuadDev& q, int nx, int I, int J) {
    const size_t k = (size_t)J * (nx + 1) + I;
    return P2{__ldg(q.xy + 2 * k), __ldg(q.xy + 2 * k + 1)};
}
// integral.cpp:91-121: edge interpolation, bilinear map, Jacobian on [-1,1]^2.
__device__ __forceinline__ P2 lerp_edge(double r, P2 a, P2 b) {
    const double s = 0.5 * (1.0 - r), t = 0.5 * (1.0 + r);
    return P2{s * a.x + t * b.x, s * a.y + t * b.y};
}
__device__ __forceinline__ P2 bilinear(double rx, double ry, const P2* c) {
    return lerp_edge(ry, lerp_edge(rx, c[0], c[1]), lerp_edge(rx, c[3], c[2]));
}
__device__ __forceinline__ double jacobian(double rx, double ry, const P2* c) {
    const double s = 0.5 * (1.0 + rx), t = 0.5 * (1.0 + ry);
    const double xi_x = 0.5 * ((1.0 - t) * (c[1].x - c[0].x) + t * (c[2].x - c[3].x));
    const double xi_y = 0.5 * ((1.0 - t) * (c[1].y - c[0].y) + t * (c[2].y - c[3].y));
    const double et_x = 0.5 * ((1.0 - s) * (c[3].x - c[0].x) + s * (c[2].x - c[1].x));
    const double et_y = 0.5 * ((1.0 - s) * (c[3].y - c[0].y) + s * (c[2].y - c[1].y));
    return xi_x * et_y - xi_y * et_x;
}
// integral.cpp:62-89: length and unit normal (dy, -dx)/length of a -> b.
__device__ __forceinline__ void edge_geometry(P2 a, P2 b, double& len, P2& n) {
    const double dx = b.x - a.x, dy = b.y - a.y;
    const double scale = fmax(fabs(dx), fabs(dy));
    const double ux = dx / scale, uy = dy / scale;
    const double norm = sqrt(fma(ux, ux, __dmul_rn(uy, uy)));
    len = scale * norm;
    n = P2{uy / norm, -ux / norm};
}
// Full Q2 form, monomial m = j*3 + i of xi^i eta^j.
__device__ __forceinline__ double q2v(const double* D, double x, double y) {
    return quad(quad(D[0], D[1], D[2], x), quad(D[3], D[4], D[5], x), quad(D[6], D[7], D[8], x), y);
}

// The cell's frame: centre, 1/h, and corners.
struct CellFrame {
    double cx, cy, inv_h, area;
    P2 c[4];
};
__device__ __forceinline__ CellFrame cell_frame(const QuadDev& q, int nx, size_t N, long long cell) {
    const int i = (int)(cell % nx), j = (int)(cell / nx);
    CellFrame f;
    f.cx = __ldg(q.geo + cell);
    f.cy = __ldg(q.geo + N + cell);
    f.inv_h = 1.0 / __ldg(q.geo + 2 * N + cell);
    f.area = __ldg(q.geo + 3 * N + cell);
    f.c[0] = vtx(q, nx, i, j); f.c[1] = vtx(q, nx, i + 1, j);
    f.c[2] = vtx(q, nx, i + 1, j + 1); f.c[3] = vtx(q, nx, i, j + 1);
    return f;
}

// A point in a cell's frame. Rounded products (no contraction with what
// follows), so that every kernel forms the same point.
__device__ __forceinline__ P2 normalised(P2 p, double cx, double cy, double inv_h) {
    return P2{__dmul_rn(p.x - cx, inv_h), __dmul_rn(p.y - cy, inv_h)};
}

// The bilinear map of a cell in its own frame: x(r, s) = m + b r + c s + d r s.
struct NormalCell {
    P2 n[4];               // corners
    P2 m, b, c, d;
    // Jacobian j0 + jr r + js s of the map (d x d vanishes).
    __device__ __forceinline__ static double cross(P2 u, P2 v) { return fma(u.x, v.y, -__dmul_rn(u.y, v.x)); }
    // The same over four times j0, the map's area: Gauss weights times it add
    // up to one, whatever the corners' roundings.
    __device__ __forceinline__ void mean_jacobian(double& j0, double& jr, double& js) const {
        const double g = __dmul_rn(0.25, rcp(cross(b, c)));
        j0 = 0.25;
        jr = __dmul_rn(cross(b, d), g);
        js = __dmul_rn(cross(d, c), g);
    }
};
__device__ __forceinline__ NormalCell normal_cell(const CellFrame& f) {
    NormalCell k;
#pragma unroll
    for (int v = 0; v < 4; ++v) k.n[v] = normalised(f.c[v], f.cx, f.cy, f.inv_h);
    auto quarter = [&](double s1, double s2, double s3) {
        return P2{0.25 * (k.n[0].x + s1 * k.n[1].x + s2 * k.n[2].x + s3 * k.n[3].x),
                  0.25 * (k.n[0].y + s1 * k.n[1].y + s2 * k.n[2].y + s3 * k.n[3].y)};
    };
    k.m = quarter(1.0, 1.0, 1.0);
    k.d = quarter(-1.0, 1.0, -1.0);
    const P2 b = quarter(-1.0, -1.0, 1.0), c = quarter(1.0, -1.0, -1.0);
    k.b = P2{-b.x, -b.y};
    k.c = P2{-c.x, -c.y};
    return k;
}

// Edge e of cell (i, j) in counter-clockwise order (0 bottom, 1 right, 2 top,
// 3 left): its local edge id, whether it is a wall, and whether the cell's
// point order runs against the canonical one. Local rows j of a mesh whose
// local row 0 is global row gj0 of gny global rows.
__device__ __forceinline__ void cell_edge(int nx, int ny, int i, int j, int gj0, int gny, int e, long long& id,
                                          bool& wall, bool& rev) {
    const long long nI = (long long)nx * (ny + 1);
    const int gj = gj0 + j;
    if (e == 0) { id = (long long)j * nx + i; wall = gj == 0; rev = false; }
    else if (e == 1) { id = nI + (long long)j * (nx + 1) + i + 1; wall = i == nx - 1; rev = false; }
    else if (e == 2) { id = (long long)(j + 1) * nx + i; wall = gj == gny - 1; rev = true; }
    else { id = nI + (long long)j * (nx + 1) + i; wall = i == 0; rev = true; }
}

// Visit every normal-line diffusion sample on this cell's side of its four
// edges (diffusiveflux.cpp:255-334, 4 samples; interior edges 2 on each side
// at offsets -1.5, -0.5 spacings from the edge, wall edges 4 at -4..-1).
template <class F>
__device__ __forceinline__ void visit_samples(const QuadDev& q, int nx, int ny, int gj0, int gny, int i, int j,
                                              const CellFrame& f, F&& visit) {
    for (int e = 0; e < 4; ++e) {
        long long id;
        bool wall, rev;
        cell_edge(nx, ny, i, j, gj0, gny, e, id, wall, rev);
        const P2 a = f.c[e], b = f.c[(e + 1) & 3];
        double len;
        P2 n;
        edge_geometry(a, b, len, n);
        for (int k = 0; k < kNQ; ++k) {
            const P2 p = lerp_edge(q.gq[k], a, b);
            const double sp = __ldg(q.sp + id * kNQ + (rev ? kNQ - 1 - k : k));
            const int ns = wall ? 4 : 2;
            for (int s = 0; s < ns; ++s) {
                const double d = (wall ? (double)(s - 4) : (double)s - 1.5) * sp;
                visit(P2{p.x + d * n.x, p.y + d * n.y});
            }
        }
    }
}

// The deviation polynomials D[f] of F fields from their 3x3 neighbourhoods
// u[f] with the cell's own tables (same candidate set and weights as
// reconstruct() of the uniform path). The fields share the cell's stencils
// and so its tables: every entry is read once and applied to each field, and
// per field the operations run in the same order whatever F is, so a field's
// result does not depend on the fields reconstructed with it. The kernel is
// bound by the bytes of the tables: the coefficients of each candidate are
// formed once, the smoothness indicators as sums of squares from them and the
// cell's six moments (quad_tables.hpp; 115 doubles per cell), and a 2x2
// candidate's constant from its zero mean over the target; reading the folded
// smoothness matrices and the constants as well (181 doubles) took 278 us at
// 640x1280, so it takes 155 (two resident blocks of 255 registers, every
// table load of a cell in flight; three blocks 176, four 228). Tables of
// candidates that are off are zero. Returns the first failure in field order.
template <int F>
__device__ __forceinline__ int reconstruct_quad(const QuadDev& q, size_t N, long long cell, int ci, int cj,
                                                double eA, const double (&u)[F][3][3], double (&D)[F][9]) {
    double d[F][3][3];
#pragma unroll
    for (int f = 0; f < F; ++f)
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < 3; ++b) d[f][a][b] = u[f][a][b] - u[f][1][1];
    auto mom = [&](int k) { return __ldg(q.mom + (size_t)k * N + cell); };
    const unsigned on = candidate_mask(ci, cj);
    const double ie = 1.0 / eA;
    // 3x3 candidate in the target's frame.
#pragma unroll
    for (int f = 0; f < F; ++f) {
        D[f][0] = d[f][0][0];
#pragma unroll
        for (int m = 1; m < 9; ++m) D[f][m] = 0.0;
    }
#pragma unroll
    for (int c = 1; c < 9; ++c) {
        double x[F];
#pragma unroll
        for (int f = 0; f < F; ++f) x[f] = d[f][c / 3][c % 3] - d[f][0][0];
#pragma unroll
        for (int m = 0; m < 9; ++m) {
            const double g = __ldg(q.G0 + (size_t)((c - 1) * 9 + m) * N + cell);
#pragma unroll
            for (int f = 0; f < F; ++f) D[f][m] = fma(x[f], g, D[f][m]);
        }
    }
    double s[F][5];
    {
        // Its sigma over the unit square of the stencil's frame, whose
        // coordinates are the target's plus (dx, dy): the coefficients moved
        // back (monomial j*3 + i; the constant is not needed), then the
        // closed form of tables.hpp with Xh = Yh = 1.
        const double dx = mom(0), dy = mom(1);
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const double* p = D[f];
            // Along x: c1 = p1 - 2 dx p2, c0 = p0 - dx p1 + dx^2 p2.
            const double r01 = fma(-2.0 * dx, p[2], p[1]);
            const double r11 = fma(-2.0 * dx, p[5], p[4]), r10 = fma(-dx, fma(-dx, p[5], p[4]), p[3]);
            const double r21 = fma(-2.0 * dx, p[8], p[7]), r20 = fma(-dx, fma(-dx, p[8], p[7]), p[6]);
            // Along y, per power of x.
            const double q01 = fma(-2.0 * dy, r20, r10), q02 = r20;
            const double q10 = fma(-dy, fma(-dy, r21, r11), r01), q11 = fma(-2.0 * dy, r21, r11), q12 = r21;
            const double q20 = fma(-dy, fma(-dy, p[8], p[5]), p[2]), q21 = fma(-2.0 * dy, p[8], p[5]), q22 = p[8];
            const double c = 1.0 / 12.0;
            const double t1 = fma(c, q12, q10), t2 = fma(c, q21, q01), t3 = fma(c, q22, q20), t4 = fma(c, q22, q02);
            double a = t1 * t1, b = t2 * t2;
            a = fma((13.0 / 3.0) * t3, t3, a);
            b = fma((13.0 / 3.0) * t4, t4, b);
            a = fma((7.0 / 6.0) * q11, q11, a);
            b = fma(0.7 * q12, q12, b);
            a = fma(0.7 * q21, q21, a);
            b = fma((43.0 / 270.0) * q22, q22, b);
            s[f][0] = fma(a + b, ie, 1.0);
        }
    }
    // 2x2 candidates: slopes b1, b2 and mixed coefficient b3; sigma is the
    // mean over the target of (b1 + b3 y)^2 + (b2 + b3 x)^2.
    const double mx = mom(2), my = mom(3), mxy = mom(4), var = mom(5);
    const int offi[4] = {0, 0, -1, -1}, offj[4] = {-1, 0, -1, 0};
    double b[F][4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int oi = offi[k], oj = offj[k];
#pragma unroll
        for (int f = 0; f < F; ++f)
#pragma unroll
            for (int m = 0; m < 3; ++m) b[f][k][m] = 0.0;
#pragma unroll
        for (int c = 1; c < 4; ++c) {
            double x[F];
#pragma unroll
            for (int f = 0; f < F; ++f) x[f] = d[f][1 + oj + c / 2][1 + oi + c % 2] - d[f][1 + oj][1 + oi];
#pragma unroll
            for (int m = 0; m < 3; ++m) {
                const double tv = __ldg(q.T4 + (size_t)(k * 12 + (c - 1) * 4 + m + 1) * N + cell);
#pragma unroll
                for (int f = 0; f < F; ++f) b[f][k][m] = fma(x[f], tv, b[f][k][m]);
            }
        }
#pragma unroll
        for (int f = 0; f < F; ++f) {
            const double gx = fma(b[f][k][2], my, b[f][k][0]), gy = fma(b[f][k][2], mx, b[f][k][1]);
            s[f][k + 1] = fma(fma(var * b[f][k][2], b[f][k][2], fma(gy, gy, gx * gx)), ie, 1.0);
        }
    }
    int st = 0;
#pragma unroll
    for (int f = 0; f < F; ++f) {
        if (on != 31u) {
#pragma unroll
            for (int k = 0; k < 5; ++k) s[f][k] = (on >> k) & 1u ? s[f][k] : 1.0;
        }
        double w[5];
        const int s1 = weno_weights(s[f], on, eA * eA, w);
        st = st ? st : s1;
#pragma unroll
        for (int m = 0; m < 9; ++m) D[f][m] = on & 1u ? D[f][m] * w[0] : 0.0;
        double g[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
            for (int m = 0; m < 3; ++m) g[m] = fma(w[k + 1], b[f][k][m], g[m]);
        D[f][0] -= fma(g[0], mx, fma(g[1], my, g[2] * mxy));
        D[f][1] += g[0];
        D[f][3] += g[1];
        D[f][4] += g[2];
    }
    return st;
}

// Left/right cells and oriented vertices of edge e (evolve.cpp:230-251).
struct QuadEdge {
    bool horizontal, boundary, reverse;
    long long e, L, R;
    int wall;
    P2 a, b;
};
__device__ __forceinline__ QuadEdge quad_edge(const QuadDev& q, int nx, int ny, int gj0, int gny, bool horizontal, int i,
                                              int j) {
    QuadEdge g;
    g.R = -1;
    g.wall = -1;
    g.horizontal = horizontal;
    P2 v0, v1;
    if (horizontal) {
        const int gj = gj0 + j;
        g.e = (long long)j * nx + i;
        g.boundary = gj == 0 || gj == gny;
        g.reverse = gj == gny;
        g.L = g.reverse ? g.e - nx : g.e;
        if (!g.boundary) g.R = g.e - nx;
        else g.wall = gj == 0 ? 0 : 1;
        v0 = vtx(q, nx, i, j); v1 = vtx(q, nx, i + 1, j);
    } else {
        const long long row = (long long)j * nx;
        g.e = (long long)nx * (ny + 1) + row + j + i;
        g.boundary = i == 0 || i == nx;
        g.reverse = i == 0;
        g.L = g.reverse ? row : row + (i - 1);
        if (!g.boundary) g.R = row + i;
        else g.wall = i == 0 ? 2 : 3;
        v0 = vtx(q, nx, i, j); v1 = vtx(q, nx, i, j + 1);
    }
    g.a = g.reverse ? v1 : v0;
    g.b = g.reverse ? v0 : v1;
    return g;
}
// Edge e in id order.
__device__ __forceinline__ QuadEdge quad_edge(const QuadDev& q, int nx, int ny, int gj0, int gny, long long e) {
    const long long nI = (long long)nx * (ny + 1);
    const bool horizontal = e < nI;
    const unsigned k = (unsigned)(horizontal ? e : e - nI), w = (unsigned)(horizontal ? nx : nx + 1);
    return quad_edge(q, nx, ny, gj0, gny, horizontal, (int)(k % w), (int)(k / w));
}

}  // namespace
}  // namespace mp

#endif
