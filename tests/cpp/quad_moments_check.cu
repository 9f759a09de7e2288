// The moments of the cells of a general quad mesh (build_quad_moments_gpu)
// against the same integrals in extended precision on the host, by a rule of
// more points: the largest difference in units of 2^-53 / h, the rounding of a
// coordinate of the unit domain in a cell's frame. A whole mesh and a slab.
#include "quad_tables.hpp"

#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <vector>

typedef long double ld;

static void check(cudaError_t e) {
    if (e != cudaSuccess) { std::printf("CUDA %s\n", cudaGetErrorString(e)); std::exit(1); }
}

int main() {
    const int nx = 13, ny = 9;
    std::vector<double> xy(2 * (nx + 1) * (ny + 1));
    unsigned long long s = 12345;
    auto noise = [&] { s = s * 6364136223846793005ULL + 1442695040888963407ULL; return (double)(s >> 11) * 0x1p-53 - 0.5; };
    for (int j = 0; j <= ny; ++j)
        for (int i = 0; i <= nx; ++i) {
            const bool in = i > 0 && i < nx && j > 0 && j < ny;
            xy[2 * (j * (nx + 1) + i)] = 0.5 * (i + (in ? 0.4 * noise() : 0.0)) / nx;
            xy[2 * (j * (nx + 1) + i) + 1] = (j + (in ? 0.4 * noise() : 0.0)) / ny;
        }
    mp::QuadTables t;
    if (mp::build_quad_tables(nx, ny, xy.data(), 1, t, 0, ny, false)) { std::printf("tables\n"); return 1; }
    double *d_xy, *d_mom;
    check(cudaMalloc((void**)&d_xy, xy.size() * 8));
    check(cudaMemcpy(d_xy, xy.data(), xy.size() * 8, cudaMemcpyHostToDevice));
    check(cudaMalloc((void**)&d_mom, (size_t)mp::kQMom * nx * ny * 8));
    const ld g[3] = {0.0L, 0.538469310105683091036314420700208805L, 0.906179845938663992797626878299392965L};
    const ld gw[3] = {128.0L / 225.0L, 0.478628670499366468041291514835638193L, 0.236926885056189087514264040719917363L};
    ld worst = 0;
    for (int part = 0; part < 2; ++part) {
        const int row0 = part ? 3 : 0, rows = part ? 4 : ny;
        const size_t N = (size_t)nx * rows;
        if (mp::build_quad_moments_gpu(nx, ny, d_xy, row0, rows, t.gq3, t.gw3, t.gq1, t.gw1, d_mom, 0)) { std::printf("launch\n"); return 1; }
        std::vector<double> mom(mp::kQMom * N);
        check(cudaMemcpy(mom.data(), d_mom, mom.size() * 8, cudaMemcpyDeviceToHost));
        for (size_t cell = 0; cell < N; ++cell) {
            const int i = (int)(cell % nx), j = row0 + (int)(cell / nx);
            auto v = [&](int I, int J, int k) { return (ld)xy[2 * (J * (nx + 1) + I) + k]; };
            const int ci[4] = {0, 1, 1, 0}, cj[4] = {0, 0, 1, 1};
            ld x[4], y[4], cx = 0, cy = 0;
            for (int k = 0; k < 4; ++k) { x[k] = v(i + ci[k], j + cj[k], 0); y[k] = v(i + ci[k], j + cj[k], 1); cx += x[k] / 4; cy += y[k] / 4; }
            auto jac = [&](ld r, ld q) {
                const ld xr = ((1 - q) * (x[1] - x[0]) + (1 + q) * (x[2] - x[3])) / 4, yr = ((1 - q) * (y[1] - y[0]) + (1 + q) * (y[2] - y[3])) / 4;
                const ld xq = ((1 - r) * (x[3] - x[0]) + (1 + r) * (x[2] - x[1])) / 4, yq = ((1 - r) * (y[3] - y[0]) + (1 + r) * (y[2] - y[1])) / 4;
                return xr * yq - yr * xq;
            };
            const ld h = sqrtl(4 * jac(0, 0));
            ld area = 0, m[5] = {0, 0, 0, 0, 0};   // x, y, xy, x^2, y^2
            for (int a = -2; a <= 2; ++a)
                for (int b = -2; b <= 2; ++b) {
                    const ld r = (a < 0 ? -1 : 1) * g[std::abs(a)], q = (b < 0 ? -1 : 1) * g[std::abs(b)];
                    const ld w = gw[std::abs(a)] * gw[std::abs(b)] * jac(r, q);
                    const ld f[4] = {(1 - r) * (1 - q) / 4, (1 + r) * (1 - q) / 4, (1 + r) * (1 + q) / 4, (1 - r) * (1 + q) / 4};
                    ld px = 0, py = 0;
                    for (int k = 0; k < 4; ++k) { px += f[k] * (x[k] - cx) / h; py += f[k] * (y[k] - cy) / h; }
                    area += w;
                    const ld e[5] = {px, py, px * py, px * px, py * py};
                    for (int k = 0; k < 5; ++k) m[k] += w * e[k];
                }
            for (ld& e : m) e /= area;
            ld want[6] = {0, 0, m[0], m[1], m[2], m[3] - m[0] * m[0] + m[4] - m[1] * m[1]};
            if (i > 0 && i < nx - 1 && j > 0 && j < ny - 1) {
                const int oi[4] = {-1, 2, 2, -1}, oj[4] = {-1, -1, 2, 2};
                ld ox = 0, oy = 0;
                for (int k = 0; k < 4; ++k) { ox += v(i + oi[k], j + oj[k], 0) / 4; oy += v(i + oi[k], j + oj[k], 1) / 4; }
                want[0] = (cx - ox) / h;
                want[1] = (cy - oy) / h;
            }
            for (int k = 0; k < mp::kQMom; ++k) worst = std::max(worst, fabsl(mom[k * N + cell] - want[k]) * h * 0x1p53L);
        }
    }
    std::printf("%.3Lf\n", worst);
    return 0;
}
