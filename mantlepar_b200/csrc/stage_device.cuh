// Device building blocks of the ML-WENO H/C transport stage.
//
// Per cell, the reference's reconstruction (Reconstruction::Update +
// TensorStencilPoly::Smoothness, src/mlweno/reconstruction.cpp:275-355 and
// tensorstencilpoly.cpp:400-459) is collapsed into one Q2 "deviation"
// polynomial D(xi, eta) in the target cell's normalised frame:
//   R(x) = u_t + sum_k w_k P_k(x)  ==  u_t + D(xi, eta),
// the 2x2 candidates being re-expanded about the target centre. The limiter
// (state_reconstruction.cpp:136-192) then scales D by theta, so each limited
// evaluation at a point is one 9-term polynomial. Smoothness indicators,
// weights and coefficients are FP64 in every form: the weights are
// (sigma + epsA)^-7 ratios, so an FP32 sigma moves them by several FP32 ulps,
// and the limited values handed to the phase inversion would carry that
// error (about 3e-9 absolute on a deviation of 0.05, more than the porosity
// of a cell near the solidus tolerates at 1e-6 relative).
#ifndef MP_STAGE_DEVICE_CUH
#define MP_STAGE_DEVICE_CUH

#include <cmath>

#include "phase_math.cuh"
#include "tables.hpp"

namespace mp {

// The tables a single-instance launch passes by value (__grid_constant__).
struct ParamTables {
    StageHot d;
};

inline void make_param_tables(const StageTables& t, ParamTables& p) { p.d = t; }

// 1/x for normal x with a normal reciprocal. The hardware's approximation y
// has 20 bits (relative error below 2^-19.9 over 2 million arguments); with
// e = 1 - x y, exact but for one rounding, 1/x = y / (1 - e) = y (1 + e + e^2 +
// ...), and cutting the series after e^2 leaves e^3 < 2^-57: with the final
// rounding off by at most one representable double, for 3 in 10^4 random
// arguments (and beside powers of two, where 1/x is nearly a tie). Three FP64
// operations, no branch and no call, where the division's range tests and
// slow path end a basic block.
__device__ __forceinline__ double rcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    e = fma(e, e, e);
    return fma(y, e, y);
}
// a/b through rcp with the remainder's correction (Markstein, IBM J. Res.
// Dev. 34, 1990: with a faithful reciprocal the last step's result is faithful,
// and correctly rounded in every one of 2 million random quotients).
__device__ __forceinline__ double div_normal(double a, double b) {
    const double y = rcp(b), q = a * y;
    return fma(fma(-b, q, a), y, q);
}
// Magnitude within [2^-960, 2^960]: rcp and div_normal apply.
__device__ __forceinline__ bool rcp_range(double x) {
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - 0x03f00000u <= 0x78000000u;
}

// Square root of a normal q in rcp's range and, with kInverse, its
// reciprocal. The hardware's reciprocal square root y = (1 + d)/sqrt(q) has 20
// bits as well; Newton's step s + (q - s^2) y/2, the residual an FMA, takes
// s = q y from d to -1.5 d^2 and from there to 1.5 d^3 < 2^-56, so with the
// last rounding s is off by at most one double (3 in 10^4 arguments). The
// reciprocal is the third-order step of rcp from y on the rounded s, off by at
// most two. Six and three FP64 operations, no branch and no call.
template <bool kInverse>
__device__ __forceinline__ double sqrt_normal(double q, double& inv) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q));
    const double h = 0.5 * y;
    double s = q * y;
    s = fma(fma(-s, s, q), h, s);
    s = fma(fma(-s, s, q), h, s);
    if (kInverse) {
        double e = fma(-s, y, 1.0);
        e = fma(e, e, e);
        inv = fma(y, e, y);
    }
    return s;
}

// The phase evaluation of phase_stage_t for a point known to be plain: H in
// [0, Hliq) and C in [1e-100, Xe] with a margin, Tep in [1e-9, 1e100] and
// ordinary scales (the flag a cell's neighbour bounds give it, plain_cell
// below). Every admissibility test of phase_stage_t then holds, and the
// solid + liquid quadratic LD melt^2 - a melt - C/Xe = 0 needs one square
// root and one reciprocal for both roots: with disc = sqrt(a^2 + 4 LD C/Xe),
// big = disc + |a| and small = disc - |a| = (4 LD C/Xe) / big, melt is the
// one of its sign over 2 LD, the other (oth) gives T = Tmp - oth/2 and
// cl = C/melt = Xe oth/2. No division, no call, no clip.
template <bool kFull>
__device__ __forceinline__ void phase_plain(const StageConst& k, double H, double C, double Tep, PhaseLean& s) {
    if (H <= Tep) {
        s.T = H; s.phil = 0.0;
        if (kFull) { s.cl = 0.0; s.cs = C; s.dTdC = 0.0; }
        return;
    }
    if (H <= fma(C, k.LDoverXe, Tep)) {
        const double r = C * k.invXe, m = (H - Tep) * k.invLD, melt = r < m ? r : m;
        s.T = Tep; s.phil = melt;
        if (kFull) {
            const double second = fma(-melt, k.Xe, C);
            s.cl = k.Xe;
            s.cs = second > 0.0 ? second * rcp(1.0 - melt) : 0.0;
            s.dTdC = 0.0;
        }
        return;
    }
    const double Tmp = Tep + 1.0, a = H - Tmp, b = C * k.fourLDoverXe;
    double inv;
    const double disc = sqrt_normal<kFull>(fma(a, a, b), inv);
    const double big = disc + fabs(a), small = b * rcp(big);
    const bool below = a < 0.0;
    const double same = below ? small : big, oth = below ? big : small;
    s.phil = same * k.halfInvLD;
    s.T = fma(-0.5, oth, Tmp);
    if (kFull) { s.cl = k.halfXe * oth; s.cs = 0.0; s.dTdC = -k.LDoverXe * inv; }
}

// Row / column coefficients of a Q2 polynomial (coefficient m = j*3 + i of
// xi^i eta^j): along the row eta = y, p(xi) = a0 + xi*(a1 + xi*a2). Written
// as FMAs, so that kernels that split a cell over lanes round alike.
__device__ __forceinline__ double quad(double c0, double c1, double c2, double s) { return fma(s, fma(s, c2, c1), c0); }
__device__ __forceinline__ void q2_row(const double* D, double y, double& a0, double& a1, double& a2) {
    a0 = quad(D[0], D[3], D[6], y);
    a1 = quad(D[1], D[4], D[7], y);
    a2 = quad(D[2], D[5], D[8], y);
}
// Along the column xi = x, p(eta) = b0 + eta*(b1 + eta*b2).
__device__ __forceinline__ void q2_col(const double* D, double x, double& b0, double& b1, double& b2) {
    b0 = quad(D[0], D[1], D[2], x);
    b1 = quad(D[3], D[4], D[5], x);
    b2 = quad(D[6], D[7], D[8], x);
}

// Nonlinear weights alpha_k = (sigma_k + epsA)^-(s*r_k + eta(r_k)): exponent
// 7 for the 3x3 order-2 candidate, 5 for the 2x2 order-1 candidates
// (reconstruction.cpp:43-54,212-265), normalised to sum 1, from
// s_k = 1 + sigma_k / epsA >= 1 (s_k = 1 for a candidate that is off).
// Multiplying every alpha by epsA^7 s_0^7 (s_1 s_2 s_3 s_4)^5 leaves products
// only: w_0 ~ (s_1 s_2 s_3 s_4)^5 and w_k ~ epsA^2 s_0^7 (the other three)^5,
// one reciprocal for the five weights. Q = s_0^2 s_1 s_2 s_3 s_4 < 1e59 keeps
// every product below 1e296 (s_0^7 t^5 <= Q^5 as s_0 >= 1); it is false for a
// non-finite s_k, so only the general form below has to test for one.
static __device__ __noinline__ int weights_general(const double* s, unsigned on, double epsA2, double* w) {
    // Ratios r = epsA/(sigma + epsA) = 1/s in (0, 1]: nothing overflows.
    double sum = 0;
    int st = 0;
    for (int k = 0; k < 5; ++k) {
        if (!((on >> k) & 1u)) { w[k] = 0; continue; }
        if (!(s[k] < INFINITY)) st = MP_ERR_FP;
        const double r = 1.0 / s[k], r2 = r * r;
        w[k] = k == 0 ? r2 * r2 * r2 * r : ((on & 1u) ? epsA2 : 1.0) * (r2 * r2 * r);
        sum += w[k];
    }
    for (int k = 0; k < 5; ++k) w[k] /= sum;
    // A sum so small that its reciprocal overflows cannot be normalised.
    if (!isfinite(w[0] + w[1] + w[2] + w[3] + w[4]) || !isfinite(1.0 / sum)) st = MP_ERR_FP;
    return st;
}
__device__ __forceinline__ int weno_weights(const double (&s)[5], unsigned on, double epsA2, double (&w)[5]) {
    const double s12 = s[1] * s[2], s34 = s[3] * s[4], P = s12 * s34, s02 = s[0] * s[0];
    if (!(P * s02 < 1e59)) {
        // Copies, so that the arrays of the common path stay in registers.
        double sc[5], wc[5];
#pragma unroll
        for (int k = 0; k < 5; ++k) sc[k] = s[k];
        const int st = weights_general(sc, on, epsA2, wc);
#pragma unroll
        for (int k = 0; k < 5; ++k) w[k] = wc[k];
        return st;
    }
    auto p5 = [](double x) { const double x2 = x * x; return __dmul_rn(x2 * x2, x); };
    const double f = (on & 1u ? epsA2 : 1.0) * (s02 * s02 * (s02 * s[0]));
    w[0] = p5(P);
    // Rounded products: the sum below adds the weights themselves.
    w[1] = __dmul_rn(f, p5(s[2] * s34));
    w[2] = __dmul_rn(f, p5(s[1] * s34));
    w[3] = __dmul_rn(f, p5(s12 * s[4]));
    w[4] = __dmul_rn(f, p5(s12 * s[3]));
    if (on != 31u) {
#pragma unroll
        for (int k = 0; k < 5; ++k) w[k] = (on >> k) & 1u ? w[k] : 0.0;
    }
    const double sum = (w[0] + (w[1] + w[2])) + (w[3] + w[4]);
    const double inv = rcp_range(sum) ? rcp(sum) : 1.0 / sum;
#pragma unroll
    for (int k = 0; k < 5; ++k) w[k] *= inv;
    return 0;
}

// Candidates kept at a boundary class (ci, cj): stencils that leave the
// domain are dropped (reconstruction.cpp:150-153). Bit 0: the 3x3 stencil;
// bits 1-4: the 2x2 stencils with lower-left cell (0,-1), (0,0), (-1,-1),
// (-1,0) relative to the target, i.e. towards SE, NE, SW, NW.
__device__ __forceinline__ unsigned candidate_mask(int ci, int cj) {
    const bool e = ci != 2, w = ci != 0, n = cj != 2, s = cj != 0;
    return (e && w && n && s ? 1u : 0u) | (e && s ? 2u : 0u) | (e && n ? 4u : 0u) | (w && s ? 8u : 0u) |
           (w && n ? 16u : 0u);
}

// Build D (9 coefficients) for one field from the 3x3 neighbourhood
// u[dj][di] (index 1,1 = target) on a uniform mesh. In the cell's frame the
// candidates have closed forms: with d the differences to the target,
//   order 1 towards NE: dE/2 xi + dN/2 eta + (dNE - dE - dN)/4 xi eta
// (mean over the target zero), and the order-2 candidate is the tensor
// product of the 1D averages' inverse (a1 = (u+ - u-)/4, a2 = (u+ - 2 u0 +
// u-)/8, a0 = u0 - a2/3). Their smoothness forms are sums of squares
// (tables.hpp), so no sigma is negative. The kernel is bound by the FP64
// pipe (one warp instruction per two cycles): with the general basis and
// smoothness matrices of the mesh (64 + 44 FMAs and 4 x 21 per field) and the
// limiter scan line by line it issued 1680 FP64 instructions per warp and took
// 160 us at 640x1280; with these forms and scan_cell 1018 and 85 us.
// on: candidate_mask of the cell. Returns MP_ERR_FP when the weights cannot
// be normalised (non-finite data).
__device__ __forceinline__ int reconstruct(const StageHot& t, unsigned on, const double (&u)[3][3], double (&D)[9]) {
    const double c = u[1][1];
    const double dSW = u[0][0] - c, dS = u[0][1] - c, dSE = u[0][2] - c, dW = u[1][0] - c, dE = u[1][2] - c,
                 dNW = u[2][0] - c, dN = u[2][1] - c, dNE = u[2][2] - c;
    // Order 2: x differences of each row (A first, B second), then along y.
    const double AS = dSE - dSW, A0 = dE - dW, AN = dNE - dNW;
    const double BS = fma(-2.0, dS, dSE + dSW), B0 = dE + dW, BN = fma(-2.0, dN, dNE + dNW);
    const double q11 = (AN - AS) * 0.0625, q12 = fma(-2.0, A0, AN + AS) * 0.03125;
    const double q21 = (BN - BS) * 0.03125, q22 = fma(-2.0, B0, BN + BS) * 0.015625;
    const double q10 = fma(-1.0 / 3.0, q12, 0.25 * A0), q01 = fma(-1.0 / 3.0, q21, 0.25 * (dN - dS));
    const double q20 = fma(-1.0 / 3.0, q22, 0.125 * B0), q02 = fma(-1.0 / 3.0, q22, 0.125 * (dN + dS));
    const double q00 = fma(-1.0 / 3.0, q20 + q02, (-1.0 / 9.0) * q22);
    double s[5];
    {
        const double t1 = fma(t.cy, q12, q10), t2 = fma(t.cx, q21, q01), t3 = fma(t.cy, q22, q20),
                     t4 = fma(t.cx, q22, q02);
        const double a = fma(t.sg[0] * t1, t1, 1.0), b = (t.sg[1] * t2) * t2;
        double x = fma(t.sg[2] * t3, t3, a), y = fma(t.sg[3] * t4, t4, b);
        x = fma(t.sg[4] * q11, q11, x);
        y = fma(t.sg[5] * q12, q12, y);
        x = fma(t.sg[6] * q21, q21, x);
        y = fma(t.sg[7] * q22, q22, y);
        s[0] = x + y;
    }
    // Order 1: mixed differences and sigma of the four quadrants.
    const double bSE = (dSE - dE) - dS, bNE = (dNE - dE) - dN, bSW = (dSW - dW) - dS, bNW = (dNW - dW) - dN;
    {
        const double e = fma(t.gx2 * dE, dE, 1.0), w = fma(t.gx2 * dW, dW, 1.0);
        const double n = __dmul_rn(t.gy2 * dN, dN), o = __dmul_rn(t.gy2 * dS, dS);
        s[1] = fma(t.gb * bSE, bSE, e + o);
        s[2] = fma(t.gb * bNE, bNE, e + n);
        s[3] = fma(t.gb * bSW, bSW, w + o);
        s[4] = fma(t.gb * bNW, bNW, w + n);
    }
    if (on != 31u) {
#pragma unroll
        for (int k = 0; k < 5; ++k) s[k] = (on >> k) & 1u ? s[k] : 1.0;
    }
    double w[5];
    const int st = weno_weights(s, on, t.epsA2, w);
    D[0] = w[0] * q00;
    D[1] = fma(w[0], q10, 0.5 * fma(w[1] + w[2], dE, -((w[3] + w[4]) * dW)));
    D[2] = w[0] * q20;
    D[3] = fma(w[0], q01, 0.5 * fma(w[2] + w[4], dN, -((w[1] + w[3]) * dS)));
    D[4] = fma(w[0], q11, 0.25 * (fma(w[2], bNE, -(w[1] * bSE)) + fma(w[3], bSW, -(w[4] * bNW))));
    D[5] = w[0] * q21;
    D[6] = w[0] * q02;
    D[7] = w[0] * q12;
    D[8] = w[0] * q22;
    return st;
}

}  // namespace mp

#endif
