// Checks of the device arithmetic that the stage kernels build on, one line
// of results per check (read by test_gpu_stage_math.py):
//   rcp, div, sqrt, rsqrt: the short reciprocal, quotient, square root and
//     inverse square root of stage_device.cuh against 1.0 / x, a / b, sqrt and
//     1 / sqrt in extended precision on the host: arguments, those that round
//     to another double, the largest distance in representable doubles, and
//     the largest relative error of the hardware's seed (as its log2);
//   plain: cells flagged plain, and those among them whose bounds come closer
//     than 1e-13 (relative to the field's largest value) to the end of a range
//     that the plain phase evaluation needs.
#include "stage_kernels.cuh"

#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

namespace mp {
namespace {

constexpr int kOut = 5;   // rcp, div, sqrt, inverse, seeds' errors
__global__ void math_kernel(int n, const double* x, const double* a, double* out, double* seed) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    double inv, none, y, r;
    out[i] = rcp(v);
    out[n + i] = div_normal(a[i], v);
    out[2 * n + i] = sqrt_normal<true>(v, inv);
    out[3 * n + i] = inv;
    out[4 * n + i] = sqrt_normal<false>(v, none);
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(v));
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
    seed[i] = y;
    seed[n + i] = r;
}

__global__ void flags_kernel(int n, Physics ph, const double* b, unsigned char* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = cell_flags(ph, b[7 * i], b[7 * i + 1], b[7 * i + 2], b[7 * i + 3], b[7 * i + 4], b[7 * i + 5], b[7 * i + 6]);
}

unsigned long long state = 88172645463325252ULL;
unsigned long long bits() {
    state ^= state << 13; state ^= state >> 7; state ^= state << 17;
    return state;
}
double uniform() { return (double)(bits() >> 11) * 0x1p-53; }

long long distance(double a, double b) {
    long long x, y;
    std::memcpy(&x, &a, 8); std::memcpy(&y, &b, 8);
    return std::llabs(x - y);
}

void check(cudaError_t e) {
    if (e != cudaSuccess) { std::printf("CUDA %s\n", cudaGetErrorString(e)); std::exit(1); }
}
template <class T>
T* device(const std::vector<T>& v) {
    T* p;
    check(cudaMalloc((void**)&p, v.size() * sizeof(T)));
    check(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return p;
}

void math() {
    std::vector<double> x, a;
    // Random mantissas over the whole range and near 1; powers of two and
    // their neighbours; both ends of the range.
    for (int k = 0; k < 2000000; ++k) x.push_back(std::ldexp(1.0 + uniform(), k % 2 ? 0 : (int)(bits() % 1919) - 960));
    for (int e = -959; e < 960; ++e)
        for (int s = -3; s <= 3; ++s) {
            double v = std::ldexp(1.0, e);
            for (int m = 0; m < std::abs(s); ++m) v = std::nextafter(v, s < 0 ? 0.0 : INFINITY);
            x.push_back(v);
        }
    for (int s = 0; s < 1000; ++s) {
        double lo = 0x1p-960 * (1.0 + s * 0x1p-52), hi = 0x1p960 * (1.0 - (s + 1) * 0x1p-53);
        x.push_back(lo);
        x.push_back(hi);
    }
    const int n = (int)x.size();
    // Numerators with the quotient and the remainder (2^-53 of it) in range.
    for (int k = 0; k < n; ++k) {
        const int e = std::ilogb(x[k]), lo = std::max(-900, -900 + e), hi = std::min(960, 960 + e);
        a.push_back(std::ldexp(1.0 + uniform(), lo + (int)(bits() % (unsigned)(hi - lo))) * (bits() & 1 ? 1.0 : -1.0));
    }
    std::vector<double> out((size_t)kOut * n), seed(2 * (size_t)n);
    double *dx = device(x), *da = device(a), *dout = device(out), *dseed = device(seed);
    math_kernel<<<(n + 255) / 256, 256>>>(n, dx, da, dout, dseed);
    check(cudaGetLastError());
    check(cudaMemcpy(out.data(), dout, out.size() * 8, cudaMemcpyDeviceToHost));
    check(cudaMemcpy(seed.data(), dseed, seed.size() * 8, cudaMemcpyDeviceToHost));
    const char* name[4] = {"rcp", "div", "sqrt", "rsqrt"};
    for (int f = 0; f < 4; ++f) {
        long long other = 0, worst = 0;
        double err = 0.0;
        for (int i = 0; i < n; ++i) {
            const long double v = x[i];
            const double want = f == 0 ? 1.0 / x[i] : f == 1 ? a[i] / x[i] : f == 2 ? std::sqrt(x[i]) : (double)(1.0L / sqrtl(v));
            const long long d = distance(out[(size_t)f * n + i], want);
            other += d != 0;
            worst = std::max(worst, d);
            const long double s = f < 2 ? seed[i] * v : seed[(size_t)n + i] * sqrtl(v);
            err = std::max(err, (double)fabsl(s - 1.0L));
            if (f == 2 && out[4 * (size_t)n + i] != out[2 * (size_t)n + i]) worst = 99;
        }
        std::printf("%s %d %lld %lld %.3f\n", name[f], n, other, worst, std::log2(err));
    }
}

void plain() {
    Physics ph{};
    ph.k.Xe = 0.5; ph.k.LD = 0.4;
    ph.sk = stage_const(ph.k);
    ph.Tep = 0.3;
    const double hliq = ph.Tep + 1.0 + ph.k.LD;
    const double low[] = {0.0, 1e-300, 1e-95, 1e-89, 1e-60, 1e-30, 1e-18, 1e-17, 1e-16, 1e-13, 1e-12, 1e-11, 1e-6, 0.1, 0.3};
    const double high[] = {1e-95, 1e-60, 1e-20, 1e-12, 1e-5, 0.1, 0.3, 0.5 - 1e-13, 0.5 - 1e-11, 0.5, 0.6};
    std::vector<double> b;
    for (double lC : low)
        for (double hC : high)
            for (double lH : {0.0, 1e-18, 1e-13, 1e-11, 0.2})
                for (double hH : {1e-6, 0.4, 0.99, 1.39, 1.69, 1.71, 2.0})
                    if (lC <= hC && lH <= hH)
                        for (double v : {ph.Tep, ph.Tep, lH, hH, lC, hC, hH}) b.push_back(v);
    const int n = (int)(b.size() / 7);
    std::vector<unsigned char> fl(n);
    double* db = device(b);
    unsigned char* df = device(fl);
    flags_kernel<<<(n + 255) / 256, 256>>>(n, ph, db, df);
    check(cudaGetLastError());
    check(cudaMemcpy(fl.data(), df, n, cudaMemcpyDeviceToHost));
    int flagged = 0, close = 0;
    for (int i = 0; i < n; ++i) {
        if (!(fl[i] & FLAG_PLAIN)) continue;
        ++flagged;
        const double lH = b[7 * i + 2], hH = b[7 * i + 3], lC = b[7 * i + 4], hC = b[7 * i + 5];
        const double hl = hliq - hC / ph.k.Xe;
        if (!(lC >= 1e-13 * hC && hC <= ph.k.Xe * (1.0 - 1e-13) && lH >= 1e-13 * hH && hH <= hl - 1e-13 * (1.0 + hH))) ++close;
    }
    std::printf("plain %d %d\n", flagged, close);
}

}  // namespace
}  // namespace mp

int main() {
    mp::math();
    mp::plain();
    return 0;
}
