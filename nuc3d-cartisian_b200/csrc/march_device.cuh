// Device pieces shared by the FP64 kernels that walk lines cell by cell
// (march_kernels.cu, thomas_kernels.cu).
#pragma once

#include "nuc3d_device.cuh"

namespace nuc3d {

// Smoothness indicators (schemes.hpp:33-34) times 3/4 as sums of two squares of
// first differences x = A_k, y = A_{k+1} (y the one nearer the face's cell):
//   3/4 beta = (x - 11/8 y)^2 + 39/64 y^2     outer sub-stencils
//   3/4 beta = (z - 5/8 y)^2 + 39/64 y^2      middle one (differences y, z)
// (13/12 (y - x)^2 + 1/4 (3y - x)^2 and its middle counterpart, completed to
// squares), so the second square is shared by neighbouring indicators and
// carried from cell to cell.  The scaling is common to all weights.
__device__ __forceinline__ double outer_is(double x, double y, double sy) {
    const double t = fma_(-1.375, y, x);
    return fma_(t, t, sy);
}
__device__ __forceinline__ double middle_is(double y, double z, double sy) {
    const double t = fma_(-0.625, y, z);
    return fma_(t, t, sy);
}

// 1/x for normal x: the hardware approximation r0 (relative error e0 below
// 2^-19) corrected by r0 (1 + e + e^2), e = 1 - x r0, whose error e0^3 lies
// below the rounding; three operations against drcp_nr's four.
__device__ __forceinline__ double rcp3(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma_(-x, r, 1.0);
    return fma_(r, fma_(e, e, e), r);
}

// Nonlinear combination: three times the face's offset from f2 is num / den.
// With w_k the
// weights without their linear factors 0.1 (1, 6, 3) and G_k the candidates'
// offsets q_k - f2 times 3, 2 and 6 (schemes.hpp:14-18),
//   3 offset = (w0 G0 + 3 w1 G1 + 3/2 w2 G2) / (w0 + 6 w1 + 3 w2).
// Every constant of the sweep's inner loop (the third is left to the
// derivative's factor) has a zero low word and so is an immediate of its
// instruction; others cost two more issue slots at each use.
template <int SCHEME>
__device__ __forceinline__ void combine(double is0, double is1, double is2, double G0, double G1,
                                        double G2, double &num, double &den) {
    double w0, w1, w2;
    if constexpr (SCHEME == SCHEME_Z) {
        // about (4 3/4 eps)^2, eps = 1e-40, with a zero low word (it only decides
        // between sub-stencils that are constant to 1e-20)
        const double ss2 = __hiloint2double(0x2f8557c2, 0);
        const double tau = sub_(is2, is0);
        const double t2 = mul_(tau, tau);
        const double s0 = fma_(is0, is0, ss2), s1 = fma_(is1, is1, ss2), s2 = fma_(is2, is2, ss2);
        const double p12 = mul_(s1, s2), p02 = mul_(s0, s2), p01 = mul_(s0, s1);
        const double P = mul_(s0, p12);
        w0 = fma_(t2, p12, P);
        w1 = fma_(t2, p02, P);
        w2 = fma_(t2, p01, P);
    } else {
        const double ss = 3.0e-6;  // 4 3/4 eps, eps = 1e-6
        double s0 = add_(ss, is0), s1 = add_(ss, is1), s2 = add_(ss, is2);
        s0 = mul_(s0, s0);
        s1 = mul_(s1, s1);
        s2 = mul_(s2, s2);
        w0 = mul_(s1, s2);
        w1 = mul_(s0, s2);
        w2 = mul_(s0, s1);
    }
    const double v1 = mul_(3.0, w1), v2 = mul_(1.5, w2);
    num = fma_(v2, G2, fma_(v1, G1, mul_(w0, G0)));
    den = fma_(2.0, add_(v1, v2), w0);
}

// Twice the split fluxes of equation e (warp-uniform) of one cell: the LF
// split's halves (physicsModel.cpp:546-565) are left to the derivative's
// factor, an exact scaling.
template <int DIR, bool LF>
__device__ __forceinline__ void split_one(int riemann, int e, double q, double un, double p,
                                          double c, double &fp, double &fm) {
    if (LF) {
        const double lam = add_(fabs(un), c);
        const double f = fma_(un, e == 4 ? add_(q, p) : q, e == 1 + DIR ? p : 0.0);
        fp = fma_(lam, q, f);
        fm = fma_(-lam, q, f);
    } else {
        SplitCell sc;
        split_prepare(riemann, un, p, c, sc);
        split_eq<DIR>(riemann, sc, e, q, fp, fm);
        fp = add_(fp, fp);
        fm = add_(fm, fm);
    }
}

__device__ __forceinline__ void cp_async8(double *smem, const double *gmem) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

}  // namespace nuc3d
