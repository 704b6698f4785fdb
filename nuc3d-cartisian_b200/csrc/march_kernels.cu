// FP64 WENO5-JS / WENO5-Z sweeps along y and z: marching warps.
//
// One RK stage's inviscid derivative along one direction (LF / AUSM / AUSMp
// split + reconstruction + flux difference, euler3d.cpp:23-56, :143-387) for
// the explicit five-point schemes in FP64.  A team is 5 warps x 32 lines: warp
// e owns equation e, lane l owns line l of the team's group, and every thread
// walks its line cell by cell over a chunk of `len` cells, carrying both
// upwind windows ('+' and '-') in registers.  One persistent block of four
// teams per SM takes (line group, chunk) items in turn; teams meet only at
// their own named barriers.
//
// Bound: the FP64 pipe and the latency of its chains (about 86 FP64 instructions
// per cell and equation, 158 instructions in all; 160^3: FP64 pipe busy 60 % of
// the cycles, issue slots 55 %, DRAM 39 %, with the 20 warps that the registers
// admit).  A march forms each difference, square and split once
// per cell: a tile of 32 cells whose threads each hold a run of 2 or 4 faces
// (k_inviscid, which these sweeps replaced) rebuilds its
// windows for every run and stages 38 cells for 32.  256^3 WENO5-Z, per launch:
// y 0.68 -> 0.59 ms, z 0.70 -> 0.57 ms.
// Measured beside it: one warp per sign (30 warps of 64 registers) 0.89 / 0.88,
// three teams of 128 registers 0.63 / 0.62, separate blocks of one team with
// the loads a cell ahead in registers 0.70 / 0.70, with the double buffer 0.67.
// Along x the lanes' lines run along the fastest axis and the same march
// behind a transposing staging pass took 0.91-1.05 ms against the tiles' 0.83,
// so x walks tiles (xsweep_kernels.cu).
//
// Window: when cell p arrives both signs hold the cells p-4..p.  With f2 the
// value of cell p-2 that is the '+' stencil of face p-1 and, mirrored, the
// '-' stencil of face p-2 (face m lies between cells m-1 and m), so one window
// position serves both.  Only first differences A_j = f(p-3+j) - f(p-4+j),
// j = 0..3, are carried: a face is f2 plus an offset that depends on the
// differences alone, and the cell derivative is
//   F(i+1) - F(i) = [f+(i) - f+(i-1)] + [f-(i+1) - f-(i)]
//                   + the change of the two signs' offsets,
// which never subtracts two nearly equal fluxes.
#include <type_traits>

#include "march_device.cuh"
#include "nuc3d_device.cuh"
#include "rhs_kernels.h"

namespace nuc3d {

namespace {

constexpr int kTeam = 5 * 32;         // threads of a team
constexpr int kTeams = 4;             // per block
constexpr int kThreads = kTeams * kTeam;
constexpr int kSMs = 148;             // one block each

// barrier of team t alone (barrier 0 is __syncthreads)
__device__ __forceinline__ void team_sync(int t) {
    asm volatile("bar.sync %0, %1;\n" ::"r"(1 + t), "n"(kTeam) : "memory");
}

// Both signs' windows of one line and equation.  The differences sit in rings of
// four registers: step<s> (s = 0..3 in turn) finds the oldest in slot s and
// puts the new one in slot (s + 3) % 4, so a loop unrolled by four moves no
// registers.  The split fluxes arrive doubled (split_one); every eps above
// carries the factor.
template <int SCHEME>
struct Window {
    double A[4], sa, fp;  // '+': differences, 39/64 a2^2, newest value
    double B[4], sb, fm;  // '-'
    double op;            // '+' offset of the newest '+' face
    double S;             // offset sum of the last complete face (op, S: times 3)

    // the chunk's first four cells
    __device__ __forceinline__ void init(const double p[4], const double m[4]) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            A[j] = sub_(p[j + 1], p[j]);
            B[j] = sub_(m[j + 1], m[j]);
        }
        sa = mul_(39.0 / 64.0, mul_(A[1], A[1]));
        sb = mul_(39.0 / 64.0, mul_(B[1], B[1]));
        fp = p[3];
        fm = m[3];
        op = S = 0.0;
    }
    // Cell p arrives with split fluxes p_, m_; quirk: face p-1 takes
    // weno5z.cpp:80's beta2 (its first term reads f2 - 2 f3 + f3 = -a2).  From
    // the third call on F(p-2) - F(p-3), the flux difference of cell p-3, is
    // lin + off / 3.
    template <int s>
    __device__ __forceinline__ void step(double p_, double m_, bool quirk, double &lin,
                                         double &off) {
        const double a0 = A[s & 3], a1 = A[(s + 1) & 3], a2 = A[(s + 2) & 3];
        const double b0 = B[s & 3], b1 = B[(s + 1) & 3], b2 = B[(s + 2) & 3];
        const double a3 = sub_(p_, fp), s1 = sa, m2 = mul_(a2, a2);
        const double b3 = sub_(m_, fm), q1 = sb;
        A[(s + 3) & 3] = a3;
        B[(s + 3) & 3] = b3;
        fp = p_;
        fm = m_;
        sa = mul_(39.0 / 64.0, m2);
        sb = mul_(39.0 / 64.0, mul_(b2, b2));
        double np, dp, nm, dm;
        {
            const double is0 = outer_is(a0, a1, s1), is1 = middle_is(a1, a2, s1);
            double is2;
            if (SCHEME == SCHEME_Z) {
                // t (a3 + x a2)^2 + y a2^2: the outer form above, or
                // 3/4 (13/12 a2^2 + 1/4 (a3 - 3 a2)^2); coefficients, as a
                // branch would split the phase's basic block
                const double t = fma_(quirk ? -3.0 : -1.375, a2, a3);
                is2 = fma_(mul_(quirk ? 0.1875 : 1.0, t), t, mul_(quirk ? 0.8125 : 39.0 / 64.0, m2));
            } else {
                is2 = outer_is(a3, a2, sa);
            }
            combine<SCHEME>(is0, is1, is2, fma_(2.5, a1, -a0), fma_(2.0, a2, a1),
                            fma_(4.0, a2, -a3), np, dp);
        }
        {
            // mirrored: upwind-oriented differences are -b3, -b2, -b1, -b0
            const double is2 = outer_is(b0, b1, q1), is1 = middle_is(b1, b2, q1);
            const double is0 = outer_is(b3, b2, sb);
            combine<SCHEME>(is0, is1, is2, fma_(-2.5, b2, b3), fma_(-2.0, b1, -b2),
                            fma_(-4.0, b1, b0), nm, dm);
        }
        const double Sn = fma_(nm, rcp3(dm), op);  // face p-2: '-' now, '+' from before
        op = mul_(np, rcp3(dp));
        lin = add_(a0, b1);
        off = sub_(Sn, S);
        S = Sn;
    }
};

// y (DIR 1) and z (DIR 2) sweeps.  Work item (box, line group, first cell); the
// launch's unit u is chunk u / nitems of item u % nitems.  Lines are numbered
// i + nx k (y) or i + nx j (z), so a group's lanes read consecutive addresses (y:
// up to a row end) whatever the box's extents, and only the box's last group has
// idle lanes.  Cells arrive in phases of four through a double buffer in shared
// memory filled with cp.async a phase ahead: each warp copies its equation's
// state and RHS, the first four warps the u_n, p and c of a row each.  A warp
// carries both signs of its equation and stores its own rows, so the warps share
// u_n, p and c alone; the team's barrier at the head of a phase says that these
// have arrived and that the other buffer has been read.
struct MarchSmem {
    double Q[2][5][2][4][32];  // [buffer][equation][state, RHS][row][line]
    double W[2][12][32];       // [buffer][row x (u_n, p, c)][line]
};

template <int SCHEME, int DIR, bool LF>
__device__ __forceinline__ void march_item(const BoxDev &bd, int group, int c0, int in_slot,
                                           int len, int team, MarchSmem &sm) {
    const BoxParams &bp = bd.p;
    const int n = bp.n[DIR];
    const int nrow = min(len, n - c0) + 6;  // cells c0-3 .. c1+2
    const int e = (threadIdx.x >> 5) - 5 * team, lane = threadIdx.x & 31;
    const int nx = bp.n[0];
    const int nlines = nx * (DIR == 1 ? bp.n[2] : bp.n[1]);
    const int L = group * 32 + lane;
    const bool ok = L < nlines;
    unsigned base = ok ? L : nlines - 1;  // the line's first cell
    if (DIR == 1) base += (base / nx) * (unsigned)(bp.stride[2] - nx);
    const int riemann = bp.riemann;
    const bool zq = SCHEME == SCHEME_Z && (bp.quirks & QK_WENOZ_BETA2);
    const double inv_d = 0.5 * bp.inv_d[DIR], inv_3d = inv_d * (1.0 / 3.0);

    // rows r0 .. r0+3 of the chunk (row r: cell c0 - 3 + r, wrapped) and the RHS
    // of cells c0 + r - 6 into buffer buf.  (Pointers and extents are read from
    // the box table here, once a phase, to leave the registers to the window.)
    auto issue = [&](int r0, int buf) {
        const int st = (int)bd.p.stride[DIR], nn = bd.p.n[DIR];
        const long long np = bd.np;
        int pos = c0 - 3 + r0;
        if (pos < 0) pos += nn;
        if (pos >= nn) pos -= nn;
        unsigned o = base + pos * st, oi = base + st * (c0 + r0 - 6);
        const double *const q = fieldU(bd, in_slot, e), *const w = fieldW(bd, 0);
        const double *const r = fieldR<double>(bd, e);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (r0 + j < nrow) {
                cp_async8(&sm.Q[buf][e][0][j][lane], q + o);
                if (r0 + j >= 6) cp_async8(&sm.Q[buf][e][1][j][lane], r + oi);
                if (e == j) {  // the first four warps a row each
                    cp_async8(&sm.W[buf][3 * j][lane], w + DIR * np + o);
                    cp_async8(&sm.W[buf][3 * j + 1][lane], w + 3 * np + o);
                    cp_async8(&sm.W[buf][3 * j + 2][lane], w + 4 * np + o);
                }
            }
            o += st;
            oi += st;
            if (++pos == nn) {
                pos = 0;
                o = base;
            }
        }
        cp_async_commit();
    };
    auto flux = [&](int buf, int s, double &fp, double &fm) {
        split_one<DIR, LF>(riemann, e, sm.Q[buf][e][0][s][lane], sm.W[buf][3 * s][lane],
                           sm.W[buf][3 * s + 1][lane], sm.W[buf][3 * s + 2][lane], fp, fm);
    };
    Window<SCHEME> w;
    team_sync(team);  // the previous item's buffers are read
    issue(0, 0);
    cp_async_wait_all();
    team_sync(team);
    issue(4, 1);
    {
        double fp[4], fm[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) flux(0, s, fp[s], fm[s]);
        w.init(fp, fm);
    }
    for (int r0 = 4; r0 < nrow; r0 += 4) {
        const int buf = (r0 >> 2) & 1;
        cp_async_wait_all();
        team_sync(team);
        if (r0 + 4 < nrow) issue(r0 + 4, buf ^ 1);
        double *const out = fieldR<double>(bd, e);
        const int st = (int)bd.p.stride[DIR];
        unsigned o = base + st * (c0 + r0 - 6);
        // rows past the chunk's last (in its last phase) compute from stale
        // shared memory and are not stored
        auto row = [&](auto sc) {
            constexpr int s = decltype(sc)::value;
            const int r = r0 + s, p = c0 - 3 + r;
            double fp, fm, lin, off;
            flux(buf, s, fp, fm);
            w.template step<s>(fp, fm, zq && p >= 4 && p <= n - 2, lin, off);
            const double rn = fma_(off, inv_3d, fma_(lin, inv_d, sm.Q[buf][e][1][s][lane]));
            if (ok && r >= 6 && r < nrow) out[o] = rn;
            o += st;
        };
        row(std::integral_constant<int, 0>{});
        row(std::integral_constant<int, 1>{});
        row(std::integral_constant<int, 2>{});
        row(std::integral_constant<int, 3>{});
    }
}

template <int SCHEME, int DIR>
__global__ void __launch_bounds__(kThreads, 1)
    k_march(const BoxDev *__restrict__ boxes, const WorkItem *__restrict__ items, int nitems,
            int chunks, int in_slot, int len) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int team = threadIdx.x / kTeam;
    MarchSmem &sm = reinterpret_cast<MarchSmem *>(smem_raw)[team];
    for (int u = team * gridDim.x + blockIdx.x; u < nitems * chunks;
         u += kTeams * gridDim.x) {
        const WorkItem it = items[u % nitems];
        const int c0 = it.b + (u / nitems) * len;
        const BoxDev &bd = boxes[it.box];
        if (!bd.active) continue;
        if (bd.p.riemann == RIEMANN_LF)
            march_item<SCHEME, DIR, true>(bd, it.a, c0, in_slot, len, team, sm);
        else
            march_item<SCHEME, DIR, false>(bd, it.a, c0, in_slot, len, team, sm);
    }
}

using March = void (*)(const BoxDev *, const WorkItem *, int, int, int, int);
template <int SCHEME>
March march_kernel(int dir) {
    return dir == 1 ? k_march<SCHEME, 1> : k_march<SCHEME, 2>;
}
constexpr size_t kSmem = kTeams * sizeof(MarchSmem);

}  // namespace

cudaError_t prepare_march_kernels() {
    for (int d = 1; d < 3; ++d)
        for (March k : {march_kernel<SCHEME_JS>(d), march_kernel<SCHEME_Z>(d)}) {
            cudaError_t e =
                cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

cudaError_t launch_march(int scheme, int dir, const BoxDev *boxes, const WorkItem *items,
                         int nitems, int chunks, int in_slot, int len, cudaStream_t st) {
    if (nitems <= 0) return cudaSuccess;
    const March k = scheme == SCHEME_JS ? march_kernel<SCHEME_JS>(dir) : march_kernel<SCHEME_Z>(dir);
    if (chunks == 0) chunks = 1;  // items are chunks
    const int units = nitems * chunks;
    k<<<units < kSMs ? units : kSMs, kThreads, kSmem, st>>>(boxes, items, nitems, chunks, in_slot,
                                                           len);
    return cudaGetLastError();
}

}  // namespace nuc3d
