// FP64 x sweeps of the explicit schemes weno5js, weno5z and weno7js: split and
// reconstruction along the fastest axis, with the con2prim of the cells
// (k_prim's work; euler3d.cpp:23-56, :143-387, physicsModel.cpp:324-356).
//
// A block of 128 threads owns 16 lines and walks `tiles` tiles of 32 cells
// along them.  Per tile: all threads stage the split fluxes of the tile and its
// halo in shared memory, then each thread forms the four faces to the right of
// its run of four cells, equation by equation, and writes their derivatives;
// the face at the run's left comes from the neighbouring lane, the tile's first
// face from the tile before (shared memory).
//
// Bound: the FP64 pipe and the waits between staging and faces (160^3: FP64 pipe
// busy 54 % of the cycles, DRAM 29 %).  A tile has 33 faces; when every tile forms both end
// faces itself, the last run of each line forms five and, as every warp holds
// such a run, all warps take five faces' time for four.  Here only a block's
// first tile does.  Lines are numbered j + ny k, so only the box's last group
// of 16 has idle lines, whatever its extents.
// 256^3 WENO5-Z with con2prim: 0.83 -> 0.745 ms per launch (8 tiles per block; one
// tile per block 0.80); 192 x 96 x 80 WENO7 0.185 -> 0.181 ms.
#include "march_device.cuh"
#include "nuc3d_device.cuh"
#include "prim_device.cuh"
#include "rhs_kernels.h"

namespace nuc3d {

namespace {

constexpr int kThreads = 128;
constexpr int TL = 16, TC = 32, NR = 8, RUN = 4;  // lines, cells, runs of a tile

// The faces of one run and equation: for WENO5 a face is its upwind values plus
// S / 3, S the sum of both signs' offsets (march_kernels.cu), for WENO7 its
// value itself.
template <int SCHEME>
struct Faces;

template <int SCHEME>
struct Faces5 {
    // windows of both signs' face m: cells m-3 .. m+1 ('+') and m-2 .. m+2 ('-')
    double a0, a1, a2, a3, sa, fp, b0, b1, b2, b3, sb, fm;
    // cells m-3 .. m and m-2 .. m+1
    template <typename FP, typename FM>
    __device__ __forceinline__ void init(const FP &p, const FM &q, int m) {
        double f0 = p(m - 3), f1 = p(m - 2), f2 = p(m - 1);
        fp = p(m);
        a1 = sub_(f1, f0);
        a2 = sub_(f2, f1);
        a3 = sub_(fp, f2);
        sa = mul_(39.0 / 64.0, mul_(a2, a2));
        f0 = q(m - 2), f1 = q(m - 1), f2 = q(m);
        fm = q(m + 1);
        b1 = sub_(f1, f0);
        b2 = sub_(f2, f1);
        b3 = sub_(fm, f2);
        sb = mul_(39.0 / 64.0, mul_(b2, b2));
    }
    // gains cells m+1 and m+2: S of face m
    __device__ __forceinline__ double step(double p, double q, bool quirk) {
        const double s1 = sa, q1 = sb;
        a0 = a1;
        a1 = a2;
        a2 = a3;
        a3 = sub_(p, fp);
        fp = p;
        b0 = b1;
        b1 = b2;
        b2 = b3;
        b3 = sub_(q, fm);
        fm = q;
        const double m2 = mul_(a2, a2);
        sa = mul_(39.0 / 64.0, m2);
        sb = mul_(39.0 / 64.0, mul_(b2, b2));
        double np, dp, nm, dm;
        {
            const double is0 = outer_is(a0, a1, s1), is1 = middle_is(a1, a2, s1);
            double is2;
            if (SCHEME == SCHEME_Z) {
                // as in march_kernels.cu; quirk: weno5z.cpp:80
                const double t = fma_(quirk ? -3.0 : -1.375, a2, a3);
                is2 = fma_(mul_(quirk ? 0.1875 : 1.0, t), t, mul_(quirk ? 0.8125 : 39.0 / 64.0, m2));
            } else {
                is2 = outer_is(a3, a2, sa);
            }
            combine<SCHEME>(is0, is1, is2, fma_(2.5, a1, -a0), fma_(2.0, a2, a1),
                            fma_(4.0, a2, -a3), np, dp);
        }
        {
            const double is2 = outer_is(b0, b1, q1), is1 = middle_is(b1, b2, q1);
            const double is0 = outer_is(b3, b2, sb);
            combine<SCHEME>(is0, is1, is2, fma_(-2.5, b2, b3), fma_(-2.0, b1, -b2),
                            fma_(-4.0, b1, b0), nm, dm);
        }
        return fma_(nm, rcp3(dm), mul_(np, rcp3(dp)));
    }
    // the part of F(m) - F(m-1) that is not S: f+(m-1) - f+(m-2) + f-(m) - f-(m-1)
    __device__ __forceinline__ double lin() const { return add_(a1, b1); }
};
template <>
struct Faces<SCHEME_JS> : Faces5<SCHEME_JS> {};
template <>
struct Faces<SCHEME_Z> : Faces5<SCHEME_Z> {};

template <>
struct Faces<SCHEME_W7> {
    double p[7], q[7];  // cells m-4 .. m+2 and m-3 .. m+3 (upwind-oriented by the call)
    template <typename FP, typename FM>
    __device__ __forceinline__ void init(const FP &fp, const FM &fm, int m) {
#pragma unroll
        for (int j = 1; j < 7; ++j) {
            p[j] = fp(m - 5 + j);
            q[j] = fm(m - 4 + j);
        }
    }
    // gains cells m+2 and m+3: the face's value
    __device__ __forceinline__ double step(double pn, double qn, bool) {
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            p[j] = p[j + 1];
            q[j] = q[j + 1];
        }
        p[6] = pn;
        q[6] = qn;
        return add_(weno7_face(p[0], p[1], p[2], p[3], p[4], p[5], p[6]),
                    weno7_face(q[6], q[5], q[4], q[3], q[2], q[1], q[0]));
    }
    __device__ __forceinline__ double lin() const { return 0.0; }
};

template <int SCHEME>
struct XGeom {
    static constexpr int H = scheme_halo(SCHEME);
    static constexpr int NF = TC + 2 * H;             // staged cells
    static constexpr int S = (NF + RUN - 1) / RUN;    // interleave stride
    static constexpr int SF = TL * RUN * S;           // staged values per flux
    static constexpr size_t SMEM = sizeof(double) * (size_t)(10 * SF + 5 * TL);
    // position pc (cell c0 - H + pc) of line l: interleaved so that the runs of a
    // line (stride 4) read consecutive words
    __device__ static int at(int l, int pc) { return (l * RUN + pc % RUN) * S + pc / RUN; }
};

}  // namespace

// Work item (box, group of 16 lines, first cell of a chunk of `tiles` tiles where
// LISTED, else blockIdx.y is the chunk: a cell read from the item costs the weno7js
// kernel spills, 192 x 96 x 80 177.7 -> 180.2 us).
// The primitives are recovered from the state and W is written for the tile's
// own cells; PM 2: their eigenvalues are folded into the box's maxima as well.
template <int SCHEME, int PM, bool LISTED>
__global__ void __launch_bounds__(kThreads, SCHEME == SCHEME_W7 ? 3 : 4)
    k_xsweep(const BoxDev *__restrict__ boxes, const WorkItem *__restrict__ items, int in_slot,
             int tiles) {
    using G = XGeom<SCHEME>;
    constexpr int H = G::H, NF = G::NF, SF = G::SF;
    constexpr bool W7 = SCHEME == SCHEME_W7;
    extern __shared__ __align__(16) double sF[];  // [10][SF], then [5][TL] first faces
    double *const sC = sF + 10 * SF;
    const WorkItem it = items[blockIdx.x];
    const BoxDev &bd = boxes[it.box];
    const BoxParams &bp = bd.p;
    const int n = bp.n[0];
    const int first = LISTED ? it.b : blockIdx.y * tiles * TC;
    if (!bd.active) return;
    const long long np = bd.np;
    const int nlines = bp.n[1] * bp.n[2], L0 = it.a * TL;
    const double *const qbase = fieldU(bd, in_slot, 0);
    const int riemann = bp.riemann;
    const PrimConst pk(bp);
    double eg[3] = {0.0, 0.0, 0.0};
    const int l = threadIdx.x / NR, r = threadIdx.x % NR, m0 = r * RUN;
    const bool ok = L0 + l < nlines;
    const bool zq = SCHEME == SCHEME_Z && (bp.quirks & QK_WENOZ_BETA2);
    // (the WENO5 fluxes are staged doubled, see split_one)
    const double inv_d = W7 ? bp.inv_d[0] : 0.5 * bp.inv_d[0];
    const double inv_s = W7 ? inv_d : inv_d * (1.0 / 3.0);
    double *const Rl = fieldR<double>(bd, 0) + (unsigned)(n * (ok ? L0 + l : 0));

    const int last = min(first + tiles * TC, n);
    for (int c0 = first; c0 < last; c0 += TC) {
        if (c0 > first) __syncthreads();  // the tile before is consumed
        for (int t = threadIdx.x; t < TL * NF; t += kThreads) {
            const int tl = t / NF, pc = t - tl * NF;
            double *const slot = sF + G::at(tl, pc);
            if (L0 + tl >= nlines) {
#pragma unroll
                for (int v = 0; v < 10; ++v) slot[v * SF] = 0.0;
                continue;
            }
            int pos = c0 - H + pc;
            const bool own = pc >= H && pc < H + TC && pos < n;
            if (pos < 0) pos += n;
            while (pos >= n) pos -= n;
            const unsigned g = n * (L0 + tl) + pos;
            double q[5];
#pragma unroll
            for (int v = 0; v < 5; ++v) q[v] = qbase[v * np + g];
            PrimCell o;
            prim_cell(pk, q, o);
            if (own) {
                prim_store(bd, g, o);
                if (PM == 2) {
                    eg[0] = fmax(add_(fabs(o.u), o.c), eg[0]);
                    eg[1] = fmax(add_(fabs(o.v), o.c), eg[1]);
                    eg[2] = fmax(add_(fabs(o.w), o.c), eg[2]);
                }
            }
            const double un = o.u, pr = o.p, c = o.c;
            if (!W7 && riemann == RIEMANN_LF) {  // block-uniform
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    double fp, fm;
                    split_one<0, true>(riemann, v, q[v], un, pr, c, fp, fm);
                    slot[v * SF] = fp;
                    slot[(5 + v) * SF] = fm;
                }
            } else {
                SplitCell sc;
                split_prepare(riemann, un, pr, c, sc);
#pragma unroll
                for (int v = 0; v < 5; ++v) {
                    double fp, fm;
                    split_eq<0>(riemann, sc, v, q[v], fp, fm);
                    slot[v * SF] = W7 ? fp : add_(fp, fp);
                    slot[(5 + v) * SF] = W7 ? fm : add_(fm, fm);
                }
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int e = 0; e < 5; ++e) {
            auto fp = [&](int c) { return sF[e * SF + G::at(l, c + H)]; };
            auto fm = [&](int c) { return sF[(5 + e) * SF + G::at(l, c + H)]; };
            auto quirk = [&](int m) { return zq && c0 + m >= 3 && c0 + m <= n - 3; };
            constexpr int A = H - 2;  // '+' gains cell m + A, '-' m + A + 1
            double S0 = 0.0;          // of the run's left face
            if (r == 0) {
                if (c0 == first) {
                    Faces<SCHEME> w;
                    w.init(fp, fm, 0);
                    S0 = w.step(fp(A), fm(A + 1), quirk(0));
                } else {
                    S0 = sC[e * TL + l];
                }
            }
            Faces<SCHEME> w;
            w.init(fp, fm, m0 + 1);
            double S[RUN], d[RUN];
#pragma unroll
            for (int k = 0; k < RUN; ++k) {
                const int m = m0 + 1 + k;
                S[k] = w.step(fp(m + A), fm(m + A + 1), quirk(m));
                d[k] = w.lin();
            }
            const double left = __shfl_up_sync(0xffffffffu, S[RUN - 1], 1);
            if (r > 0) S0 = left;
            // a line's lanes share a warp: its r = 0 has read the tile before's face
            // (a shuffle alone orders no memory) before r = NR-1 replaces it
            __syncwarp();
            if (r == NR - 1) sC[e * TL + l] = S[RUN - 1];
#pragma unroll
            for (int k = RUN - 1; k >= 0; --k) {
                const double o = sub_(S[k], k > 0 ? S[k - 1] : S0);
                d[k] = W7 ? mul_(o, inv_s) : fma_(o, inv_s, mul_(d[k], inv_d));
            }
            if (ok) {
                double *const out = Rl + e * np + c0 + m0;
                if (n % 2 == 0) {  // block-uniform: 16-byte aligned pairs
#pragma unroll
                    for (int k = 0; k < RUN; k += 2)
                        if (c0 + m0 + k < n)
                            *reinterpret_cast<double2 *>(out + k) = make_double2(d[k], d[k + 1]);
                } else {
#pragma unroll
                    for (int k = 0; k < RUN; ++k)
                        if (c0 + m0 + k < n) out[k] = d[k];
                }
            }
        }
    }
    if (PM == 2) eig_block_max(bd, eg[0], eg[1], eg[2]);
}

namespace {
using XSweep = void (*)(const BoxDev *, const WorkItem *, int, int);
template <int SCHEME>
XSweep xsweep_pm(int prim_mode, bool listed) {
    if (listed) return prim_mode == 2 ? k_xsweep<SCHEME, 2, true> : k_xsweep<SCHEME, 1, true>;
    return prim_mode == 2 ? k_xsweep<SCHEME, 2, false> : k_xsweep<SCHEME, 1, false>;
}
XSweep xsweep_kernel(int scheme, int prim_mode, bool listed, size_t &smem) {
    smem = scheme == SCHEME_W7  ? XGeom<SCHEME_W7>::SMEM
           : scheme == SCHEME_Z ? XGeom<SCHEME_Z>::SMEM
                                : XGeom<SCHEME_JS>::SMEM;
    return scheme == SCHEME_JS  ? xsweep_pm<SCHEME_JS>(prim_mode, listed)
           : scheme == SCHEME_Z ? xsweep_pm<SCHEME_Z>(prim_mode, listed)
                                : xsweep_pm<SCHEME_W7>(prim_mode, listed);
}
}  // namespace

cudaError_t prepare_xsweep_kernels() {
    for (int s : {SCHEME_JS, SCHEME_Z, SCHEME_W7})
        for (int m = 0; m < 4; ++m) {
            size_t smem;
            const XSweep k = xsweep_kernel(s, 1 + m % 2, m / 2 == 1, smem);
            cudaError_t e =
                cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

cudaError_t launch_xsweep(int scheme, const BoxDev *boxes, const WorkItem *items, int nitems,
                          int chunks, int in_slot, int tiles, int prim_mode, cudaStream_t st) {
    if (nitems <= 0) return cudaSuccess;
    size_t smem;
    const XSweep k = xsweep_kernel(scheme, prim_mode, chunks == 0, smem);
    k<<<dim3(nitems, chunks > 0 ? chunks : 1), kThreads, smem, st>>>(boxes, items, in_slot, tiles);
    return cudaGetLastError();
}

}  // namespace nuc3d
