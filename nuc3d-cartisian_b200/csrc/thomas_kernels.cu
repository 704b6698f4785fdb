// FP64 CRWENO5 sweeps along y and z (bounded lines): one thread per line and
// equation, both signs' tridiagonal systems by the reference's own recurrences
// (crweno5.cpp:45-402).
//
// A warp takes 32 lines adjacent in memory and, in turn, the equations of its
// set (0, 3 / 1, 4 / 2).  Forward it walks the cells: split (LF / AUSM / AUSMp),
// upwind windows, the compact row of the newest '+' and '-' face and its
// elimination, c' and d' of both signs to scratch.  Backward it walks the faces:
// x = d' - c' x', F = F+ + F-, and adds the flux difference to the RHS.  Explicit
// WENO5-JS faces (0..3 and n-3..n) are rows with c' = 0.
//
// The line kernel (k_crweno_lines, lanes along one line) spends about four
// instructions on its partitioned solve, shared-memory rows and index work for
// each FP64 one and is bound by instruction issue; here a row costs about 110
// instructions forward, 82 of them FP64, and 25 back.  Bound: HBM, for the 64
// bytes of c' and d' that each face and equation writes and reads back (160^3: 485
// bytes of DRAM traffic per cell at 5.8 TB/s, FP64 pipe 31 %).  192^3:
// y 1.01 -> 0.61 ms, z 1.02 -> 0.59 ms per launch (5.6 TB/s; 16 warps of 128
// registers per SM with 8 faces' loads together on the way back; 20 warps of 96
// with 4 measured 0.62 / 0.61).
//
// Scratch: 12 values per cell, in fields that hold nothing at this point of a
// stage: 8 of the viscous fluxes (computed after these sweeps) and 4 of the
// state slot that is neither u_n nor the stage's input (rows 0..n-1 of a line
// lie at its cells; face n stays in registers).
#include <type_traits>

#include "march_device.cuh"
#include "nuc3d_device.cuh"
#include "rhs_kernels.h"

namespace nuc3d {

namespace {

constexpr int kThreads = 128;

// one compact row times a common positive factor (crweno5.cpp:136-161): with
// w_k the weights without their linear factors 0.1 (2, 5, 3) and the upwind
// differences x = f2 - f1, y = f3 - f2,
//   lo = 4 w0 + 5 w1,  b = 2 w0 + 10 w1 + 6 w2,  hi = 3 w2,
//   d = (lo + b + hi) f2 - w0 x + 5/2 (w1 + 3 w2) y
struct Row {
    double lo, b, hi, d;
};
__device__ __forceinline__ Row compact_row(double is0, double is1, double is2, double f2, double x,
                                           double y) {
    const double ss = 3.0e-6;  // 4 3/4 eps, eps = 1e-6
    double s0 = add_(ss, is0), s1 = add_(ss, is1), s2 = add_(ss, is2);
    s0 = mul_(s0, s0);
    s1 = mul_(s1, s1);
    s2 = mul_(s2, s2);
    const double w0 = mul_(s1, s2), w1 = mul_(s0, s2), w2 = mul_(s0, s1);
    Row r;
    r.lo = fma_(4.0, w0, mul_(5.0, w1));
    r.b = fma_(2.0, w0, fma_(10.0, w1, mul_(6.0, w2)));
    r.hi = mul_(3.0, w2);
    const double c3 = fma_(7.5, w2, mul_(2.5, w1));
    r.d = fma_(add_(add_(r.lo, r.b), r.hi), f2, fma_(c3, y, -mul_(w0, x)));
    return r;
}

// One sign's window and elimination: differences of cells p-4..p (a ring, as in
// march_kernels.cu), the newest three values, c' and d' of the last row.
template <int SIGN>
struct System {
    double A[4], sa, v[4], cp, dp;
    __device__ __forceinline__ void init(const double f[4]) {
#pragma unroll
        for (int j = 0; j < 3; ++j) A[j] = sub_(f[j + 1], f[j]);
        sa = mul_(39.0 / 64.0, mul_(A[1], A[1]));
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = f[j];  // cell of step s's newest at v[s & 3]
        cp = dp = 0.0;
    }
    // cell p arrives (step s = 0..3 in turn); the new face's row is eliminated.
    // fixed: an explicit face.
    template <int s>
    __device__ __forceinline__ void step(double f, bool fixed) {
        const double a0 = A[s & 3], a1 = A[(s + 1) & 3], a2 = A[(s + 2) & 3];
        const double a3 = sub_(f, v[(s + 3) & 3]), s1 = sa;
        A[(s + 3) & 3] = a3;
        v[s & 3] = f;
        sa = mul_(39.0 / 64.0, mul_(a2, a2));
        const double f2 = v[(s + 2) & 3];  // cell p - 2
        const double lo_is = outer_is(a0, a1, s1), mid = middle_is(a1, a2, s1),
                     hi_is = outer_is(a3, a2, sa);
        if (fixed) {  // warp-uniform
            double num, den;
            if (SIGN > 0)
                combine<SCHEME_JS>(lo_is, mid, hi_is, fma_(2.5, a1, -a0), fma_(2.0, a2, a1),
                                   fma_(4.0, a2, -a3), num, den);
            else
                combine<SCHEME_JS>(hi_is, mid, lo_is, fma_(-2.5, a2, a3), fma_(-2.0, a1, -a2),
                                   fma_(-4.0, a1, a0), num, den);
            cp = 0.0;
            dp = fma_(num, mul_(rcp3(den), 1.0 / 3.0), f2);
            return;
        }
        // '+': upwind-side coupling to the face below; '-' mirrored
        // (crweno5.cpp:335-338)
        const Row r = SIGN > 0 ? compact_row(lo_is, mid, hi_is, f2, a1, a2)
                               : compact_row(hi_is, mid, lo_is, f2, -a2, -a1);
        const double a = SIGN > 0 ? r.lo : r.hi, c = SIGN > 0 ? r.hi : r.lo;
        const double inv = rcp3(fma_(-cp, a, r.b));
        cp = mul_(c, inv);
        dp = mul_(fma_(-dp, a, r.d), inv);
    }
};

}  // namespace

// the equations set, set + 3 of one line; scratch: c'+, d'+, c'-, d'- (fields np
// apart).  Pointers and extents are read from the box table where they are
// used, to leave the registers to the two systems.
template <int DIR, bool LF>
__device__ __forceinline__ void thomas_lines(const BoxDev &bd, int set, unsigned base, bool ok,
                                             int in_slot, double *const scratch,
                                             double (&buf)[2][4][4][32]) {
    const int lane = threadIdx.x & 31, n = bd.p.n[DIR], st = (int)bd.p.stride[DIR];
    const int riemann = bd.p.riemann;
#pragma unroll 1
    for (int e = set; e < 5; e += 3) {
        // rows r0 .. r0+3 (row r: cell r - 4, wrapped; rows 0 .. n+6)
        auto issue = [&](int r0, int b) {
            const long long np = bd.np;
            const double *const Q = fieldU(bd, in_slot, e), *const W = fieldW(bd, 0);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int pos = r0 + j - 4;
                if (pos < 0) pos += n;
                if (pos >= n) pos -= n;
                const unsigned o = base + pos * st;
                cp_async8(&buf[b][0][j][lane], Q + o);
                cp_async8(&buf[b][1][j][lane], W + DIR * np + o);
                cp_async8(&buf[b][2][j][lane], W + 3 * np + o);
                cp_async8(&buf[b][3][j][lane], W + 4 * np + o);
            }
            cp_async_commit();
        };
        auto flux = [&](int b, int s, double &fp, double &fm) {
            split_one<DIR, LF>(riemann, e, buf[b][0][s][lane], buf[b][1][s][lane],
                               buf[b][2][s][lane], buf[b][3][s][lane], fp, fm);
        };
        System<1> P;
        System<-1> M;
        // forward.  At cell p the newest '+' face is p - 1, the newest '-' face
        // p - 2; the window starts with cells -4..-1.  Faces 0..3 and n-3..n (and
        // those before 0, unused) are explicit.
        issue(0, 0);
        cp_async_wait_all();
        issue(4, 1);
        {
            double fp[4], fm[4];
#pragma unroll
            for (int s = 0; s < 4; ++s) flux(0, s, fp[s], fm[s]);
            P.init(fp);
            M.init(fm);
        }
        double xp = 0.0, xm = 0.0;  // face n
        for (int r0 = 4; r0 < n + 7; r0 += 4) {
            const int b = (r0 >> 2) & 1;
            cp_async_wait_all();  // (each lane reads its own copies alone)
            if (r0 + 4 < n + 7) issue(r0 + 4, b ^ 1);
            const long long np = bd.np;
            // of '+' face r0 - 5 (faces before 0 are not stored)
            double *sc = scratch + ((long long)base + (long long)(r0 - 5) * st);
            auto row = [&](auto k) {
                constexpr int s = decltype(k)::value;
                const int p = r0 + s - 4, mp = p - 1, mm = p - 2;
                if (p > n + 2) return;
                double fp, fm;
                flux(b, s, fp, fm);
                P.template step<s>(fp, mp <= 3 || mp >= n - 3);
                M.template step<s>(fm, mm <= 3 || mm >= n - 3);
                if (ok && mp >= 0 && mp < n) {
                    sc[0] = P.cp;
                    sc[np] = P.dp;
                }
                if (ok && mm >= 0 && mm < n) {
                    sc[2 * np - st] = M.cp;
                    sc[3 * np - st] = M.dp;
                }
                sc += st;
                if (mp == n) xp = P.dp;
                if (mm == n) xm = M.dp;
            };
            row(std::integral_constant<int, 0>{});
            row(std::integral_constant<int, 1>{});
            row(std::integral_constant<int, 2>{});
            row(std::integral_constant<int, 3>{});
        }
        // backward, D faces at a time with their loads together
        const double inv_d = 0.5 * bd.p.inv_d[DIR];
        const long long np = bd.np;
        double *const R = fieldR<double>(bd, e);
        double T = add_(xp, xm);  // F at face m + 1
        constexpr int D = 8;
#pragma unroll 1
        for (int m0 = n - 1; m0 >= 0; m0 -= D) {
            double c1[D], d1[D], c2[D], d2[D], rr[D];
#pragma unroll
            for (int j = 0; j < D; ++j) {
                const unsigned o = base + max(m0 - j, 0) * st;
                const double *const sc = scratch + o;
                c1[j] = sc[0];
                d1[j] = sc[np];
                c2[j] = sc[2 * np];
                d2[j] = sc[3 * np];
                rr[j] = R[o];
            }
#pragma unroll
            for (int j = 0; j < D; ++j) {
                if (m0 - j < 0) break;
                xp = fma_(-c1[j], xp, d1[j]);
                xm = fma_(-c2[j], xm, d2[j]);
                const double F = add_(xp, xm);
                if (ok) R[base + (m0 - j) * st] = fma_(sub_(T, F), inv_d, rr[j]);
                T = F;
            }
        }
    }
}

// Work item (box, line group); unit u: equation set u / nitems of item
// u % nitems (the one-equation set last, so that it fills the tail).
template <int DIR>
__global__ void __launch_bounds__(kThreads, 4)
    k_thomas(const BoxDev *__restrict__ boxes, const WorkItem *__restrict__ items, int nitems,
             int in_slot, int free_slot) {
    __shared__ double sQ[kThreads / 32][2][4][4][32];  // [warp][buffer][q, u_n, p, c][row][line]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = blockIdx.x * (kThreads / 32) + warp;
    if (u >= 3 * nitems) return;
    const WorkItem it = items[u % nitems];
    const int set = u / nitems;
    const BoxDev &bd = boxes[it.box];
    if (!bd.active) return;
    const int nx = bd.p.n[0];
    const int nlines = nx * (DIR == 1 ? bd.p.n[2] : bd.p.n[1]);
    const int L = it.a * 32 + lane;
    const bool ok = L < nlines;
    unsigned base = ok ? L : nlines - 1;  // the line's first cell
    if (DIR == 1) base += (base / nx) * (unsigned)(bd.p.stride[2] - nx);
    double *const scratch = set < 2 ? fieldV<double>(bd, 4 * set) : fieldU(bd, free_slot, 0);
    if (bd.p.riemann == RIEMANN_LF)
        thomas_lines<DIR, true>(bd, set, base, ok, in_slot, scratch, sQ[warp]);
    else
        thomas_lines<DIR, false>(bd, set, base, ok, in_slot, scratch, sQ[warp]);
}

cudaError_t launch_thomas(int dir, const BoxDev *boxes, const WorkItem *items, int nitems,
                          int in_slot, int free_slot, cudaStream_t st) {
    if (nitems <= 0) return cudaSuccess;
    const unsigned grid = (unsigned)((3LL * nitems * 32 + kThreads - 1) / kThreads);
    if (dir == 1)
        k_thomas<1><<<grid, kThreads, 0, st>>>(boxes, items, nitems, in_slot, free_slot);
    else
        k_thomas<2><<<grid, kThreads, 0, st>>>(boxes, items, nitems, in_slot, free_slot);
    return cudaGetLastError();
}

}  // namespace nuc3d
