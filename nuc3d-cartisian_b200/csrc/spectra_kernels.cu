// Shell-binned spectra of a box's current state: postproc::solveFFT
// (postproc.cpp:931-1184) with fft::solveFFT_forward (fft.cpp:182-283) and the
// two fft::solveShell binnings (fft.cpp:384-572), FP64.
//
//   k_spec_fields  u, v, w, the helicity field w.u, the enstrophy field
//                  |w|^2/2 (solveQ's fields, postproc.cpp:812-853, vorticity
//                  from the differential scheme's gradients), density and
//                  pressure, rows padded to 2 (nx/2 + 1) reals;
//   cuFFT          forward 3-D D2Z transforms of the seven fields in
//                  place (FFTW_FORWARD sign; the 1/N of fft.cpp:277-278 is
//                  applied when binning).  The fields are real, so the modes
//                  with kx < 0 are the conjugates of their mirrors and carry
//                  the same energies: half the transform, scratch and binning
//                  of complex fields with a zero imaginary part.  (A mode on
//                  a Nyquist plane, whose mirror the fold takes to the same
//                  sign, has |k| >= kmax and is in no shell.);
//   k_spec_bin     per mode: the folded wavenumber, the compressive /
//                  solenoidal / helical split of the velocity transform
//                  (postproc.cpp:1013-1101) and the shell of each binning.
//                  The kinetic spectra use the folded |k| with |k| = 1
//                  substituted at k = 0 (fft.cpp:424-435, the mean flow lands
//                  in shell 1); the scalar spectra use the unfolded
//                  i^2 + j^2 + k^2 of fft.cpp:517-531 (only the non-negative
//                  octant is counted).  A warp takes 32 modes of a (j, k) row
//                  at a time; along a row the shells do not decrease, so a
//                  segmented warp scan sums each shell's run and the runs'
//                  last lanes add to the warp's own shell sums in shared
//                  memory, each shell once: a fixed order without atomics
//                  (128^3: 502 us with one thread per spectrum adding a
//                  block's modes one by one);
//   k_spec_reduce  adds the blocks' shell sums in a fixed order, a warp per sum.
// The grid is fixed, so a box gives the same bits alone or in any batch.
#include <cufft.h>

#include "nuc3d_device.cuh"
#include "spectra_kernels.h"

namespace nuc3d {

namespace {

constexpr int kThreads = 256;

template <int R>
__global__ void __launch_bounds__(kThreads) k_spec_fields(BoxDev b, double *F) {
    const BoxParams &p = b.p;
    const double *rho = fieldU(b, 0, 0);
    const double *u = fieldW(b, 0), *v = fieldW(b, 1), *w = fieldW(b, 2), *pr = fieldW(b, 3);
    const unsigned nx = p.n[0];
    const unsigned pad = 2 * (nx / 2 + 1) - nx;
    const long long NF = p.N + (long long)pad * (p.N / nx);
    for (long long cc = blockIdx.x * (long long)blockDim.x + threadIdx.x; cc < p.N;
         cc += (long long)gridDim.x * blockDim.x) {
        const unsigned c = (unsigned)cc;
        const DiffAt<R> at(p, c);
        const double u0 = u[c], u1 = v[c], u2 = w[c];
        const double w0 = at(w, p, 1) - at(v, p, 2), w1 = at(u, p, 2) - at(w, p, 0),
                     w2 = at(v, p, 0) - at(u, p, 1);
        double *const o = F + cc + (long long)pad * (c / nx);
        o[0] = u0;
        o[NF] = u1;
        o[2 * NF] = u2;
        o[3 * NF] = w0 * u0 + w1 * u1 + w2 * u2;
        o[4 * NF] = (w0 * w0 + w1 * w1 + w2 * w2) * 0.5;
        o[5 * NF] = rho[c];
        o[6 * NF] = pr[c];
    }
}

// shell of |k| (fft.cpp:432-433): floor(|k|), or floor + 1 past the half
__device__ __forceinline__ int shell_of(double kmag) {
    const double fl = floor(kmag);
    return ((kmag - fl) - 0.5 <= 0) ? (int)fl : (int)fl + 1;
}

__device__ __forceinline__ double folded(int i, int n) {
    return (2 * i >= n) ? (double)i - n : (double)i;  // fft.cpp:424-426
}

__device__ __forceinline__ double sq(double x) { return x * x; }

// adds the lanes' values to h[q * ks + shell] (shell < 0: nowhere); equal
// shells sit in adjacent lanes
template <int NQ>
__device__ __forceinline__ void add_runs(double (&v)[NQ], int shell, double *h, int ks) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const bool same = __shfl_up_sync(0xffffffffu, shell, o) == shell && lane >= o;
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const double t = __shfl_up_sync(0xffffffffu, v[q], o);
            if (same) v[q] += t;
        }
    }
    const int next = __shfl_down_sync(0xffffffffu, shell, 1);
    if (shell >= 0 && (lane == 31 || next != shell)) {
#pragma unroll
        for (int q = 0; q < NQ; ++q) h[q * ks + shell] += v[q];
    }
    __syncwarp();
}

__global__ void __launch_bounds__(kThreads) k_spec_bin(const double2 *F, int nx, int ny, int nz,
                                                        int kmax, double *partials) {
    extern __shared__ __align__(16) double sm[];  // [warp][kSpectra][kmax + 1]
    const int NW = blockDim.x >> 5, ks = kmax + 1, nh = nx / 2 + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = threadIdx.x; t < NW * kSpectra * ks; t += blockDim.x) sm[t] = 0.0;
    __syncthreads();
    double *const hist = sm + warp * kSpectra * ks;
    const long long rows = (long long)ny * nz, NH = rows * nh;
    const double inv_n = 1.0 / ((double)nx * ny * nz), kc = (double)kmax;
    for (long long row = blockIdx.x * NW + warp; row < rows; row += (long long)gridDim.x * NW) {
        const int k = (int)(row / ny), j = (int)(row - (long long)k * ny);
        const double ky = folded(j, ny), kz = folded(k, nz);
        const double k2 = ky * ky + kz * kz;
        const long long r2 = (long long)j * j + (long long)k * k;
        const bool scal = r2 < (long long)kmax * kmax;  // (implies k2 < kmax^2)
        if (k2 >= kc * kc) continue;
        for (int i0 = 0; i0 < nh && i0 < kmax; i0 += 32) {
            const int i = i0 + lane;
            const long long m = row * nh + i;
            double kmag = sqrt((double)i * i + k2);
            if (kmag < 1e-6) kmag = 1.0;
            const bool in = i < nh && kmag < kc;
            double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
            if (in) {
                const double ik = 1.0 / kmag;
                // unit wavevector (the zero vector at k = 0)
                const double e[3] = {folded(i, nx) * ik, ky * ik, kz * ik};
                double ur[3], ui[3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    const double2 f = F[d * NH + m];
                    ur[d] = f.x * inv_n;  // fft.cpp:277-278
                    ui[d] = f.y * inv_n;
                }
                const double ku_r = e[0] * ur[0] + e[1] * ur[1] + e[2] * ur[2];
                const double ku_i = e[0] * ui[0] + e[1] * ui[1] + e[2] * ui[2];
                double sr[3], si[3];
                double a = 0.0, c = 0.0, s = 0.0, l = 0.0, r = 0.0;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    sr[d] = ur[d] - ku_r * e[d];
                    si[d] = ui[d] - ku_i * e[d];
                    a += sq(ur[d]) + sq(ui[d]);
                    c += sq(ur[d] - sr[d]) + sq(ui[d] - si[d]);
                    s += sq(sr[d]) + sq(si[d]);
                }
                // i k x s / |k| (postproc.cpp:1052-1059)
                const double xr[3] = {-(e[1] * si[2] - e[2] * si[1]), e[0] * si[2] - e[2] * si[0],
                                      -(e[0] * si[1] - e[1] * si[0])};
                const double xi[3] = {e[1] * sr[2] - e[2] * sr[1], -(e[0] * sr[2] - e[2] * sr[0]),
                                      e[0] * sr[1] - e[1] * sr[0]};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    l += sq(sr[d] - xr[d]) + sq(si[d] - xi[d]);
                    r += sq(sr[d] + xr[d]) + sq(si[d] + xi[d]);
                }
                // 1/2, twice where the mirror mode is left out
                const double w = i == 0 ? 0.5 : 1.0;
                v[0] = w * a;
                v[1] = w * c;
                v[2] = w * s;
                v[3] = 0.25 * w * l;
                v[4] = 0.25 * w * r;
            }
            add_runs<5>(v, in ? shell_of(kmag) : -1, hist, ks);
            if (!scal) continue;
            const long long k0 = (long long)i * i + r2;
            const bool on = i < nh && k0 < (long long)kmax * kmax;
            double q[4] = {0.0, 0.0, 0.0, 0.0};
            if (on) {
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    const double2 f = F[(3 + d) * NH + m];
                    q[d] = sq(f.x * inv_n) + sq(f.y * inv_n);
                }
            }
            add_runs<4>(q, on ? shell_of(sqrt((double)k0)) : -1, hist + 5 * ks, ks);
        }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kSpectra * kmax; t += blockDim.x) {
        const int h = (t / kmax) * ks + t % kmax;
        double s = 0.0;
        for (int w = 0; w < NW; ++w) s += sm[w * kSpectra * ks + h];
        partials[(size_t)blockIdx.x * kSpectra * kmax + t] = s;
    }
}

// one warp per sum
__global__ void k_spec_reduce(const double *partials, int nblocks, int n, double *out) {
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= n) return;
    double s = 0.0;
    for (int b = lane; b < nblocks; b += 32) s += partials[(size_t)b * n + t];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) out[t] = s;
}

size_t align256(size_t n) { return (n + 255) / 256 * 256; }
size_t fields_bytes(const BoxParams &p) {
    return align256(sizeof(double2) * kSpectraFields * (size_t)(p.n[0] / 2 + 1) * p.n[1] * p.n[2]);
}
size_t partials_bytes(const BoxParams &p) {
    return align256(sizeof(double) * (size_t)kSpecBlocks * kSpectra * spectra_kmax(p));
}
size_t out_bytes(const BoxParams &p) {
    return align256(sizeof(double) * (size_t)kSpectra * spectra_kmax(p));
}

}  // namespace

int SpectraPlan::prepare(const BoxParams &p, cudaStream_t st) {
    cufftResult r = CUFFT_SUCCESS;
    if (!made || n[0] != p.n[0] || n[1] != p.n[1] || n[2] != p.n[2]) {
        release();
        cufftHandle h;
        r = cufftCreate(&h);
        if (r != CUFFT_SUCCESS) return (int)r;
        made = true;
        handle = (int)h;
        for (int d = 0; d < 3; ++d) n[d] = p.n[d];
        // forward 3-D transforms (x fastest: dims nz, ny, nx), the seven fields
        // together where they are small and launches count, else one by one
        // with a work area of one field
        batch = p.N <= 64 * 64 * 64 ? kSpectraFields : 1;
        const long long nh = p.n[0] / 2 + 1, rows = (long long)p.n[1] * p.n[2];
        long long dims[3] = {p.n[2], p.n[1], p.n[0]}, real[3] = {p.n[2], p.n[1], 2 * nh},
                  half[3] = {p.n[2], p.n[1], nh};
        r = cufftSetAutoAllocation(h, 0);
        if (r == CUFFT_SUCCESS)
            r = cufftMakePlanMany64(h, 3, dims, real, 1, 2 * nh * rows, half, 1, nh * rows,
                                    CUFFT_D2Z, batch, &work);
    }
    if (r == CUFFT_SUCCESS) r = cufftSetStream((cufftHandle)handle, st);
    return (int)r;
}

void SpectraPlan::release() {
    if (made) cufftDestroy((cufftHandle)handle);
    *this = SpectraPlan();
}

size_t spectra_scratch_bytes(const BoxParams &p, size_t work) {
    return fields_bytes(p) + partials_bytes(p) + out_bytes(p) + work;
}

cudaError_t launch_spectra(const BoxDev &b, const SpectraPlan &plan, void *scratch,
                           double **d_out, int *fft_status, cudaStream_t st) {
    const BoxParams &p = b.p;
    const int kmax = spectra_kmax(p);
    char *c = static_cast<char *>(scratch);
    double *F = reinterpret_cast<double *>(c);
    double *partials = reinterpret_cast<double *>(c += fields_bytes(p));
    double *out = reinterpret_cast<double *>(c += partials_bytes(p));
    *d_out = out;
    if (diff_reach(p) == 3)
        k_spec_fields<3><<<4 * 148, kThreads, 0, st>>>(b, F);
    else
        k_spec_fields<4><<<4 * 148, kThreads, 0, st>>>(b, F);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cufftResult r = cufftSetWorkArea((cufftHandle)plan.handle, c + out_bytes(p));
    const size_t field = 2 * (size_t)(p.n[0] / 2 + 1) * p.n[1] * p.n[2];
    for (int f = 0; f < kSpectraFields && r == CUFFT_SUCCESS; f += plan.batch)
        r = cufftExecD2Z((cufftHandle)plan.handle, F + f * field,
                         reinterpret_cast<cufftDoubleComplex *>(F + f * field));
    *fft_status = (int)r;
    if (r != CUFFT_SUCCESS) return cudaSuccess;
    // warps per block: as many shell tables as fit 200 KB, at most 8 (a box
    // of 2^31 cells has kmax <= 645)
    constexpr int kMaxSmem = 200 * 1024;
    const size_t table = sizeof(double) * kSpectra * (size_t)(kmax + 1);
    const int warps = (int)(kMaxSmem / table < 8 ? kMaxSmem / table : 8);
    const size_t smem = table * warps;
    // (the same limit from every call: it is shared with the other host threads)
    e = cudaFuncSetAttribute(k_spec_bin, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
    if (e != cudaSuccess) return e;
    k_spec_bin<<<kSpecBlocks, 32 * warps, smem, st>>>(reinterpret_cast<const double2 *>(F), p.n[0],
                                                    p.n[1], p.n[2], kmax, partials);
    const int n = kSpectra * kmax;
    k_spec_reduce<<<(n + 3) / 4, 128, 0, st>>>(partials, kSpecBlocks, n, out);
    return cudaGetLastError();
}

}  // namespace nuc3d
