// Spectral shell forcing on the device, FP64: physicsModel::AddForcing_Const
// (physicsModel.cpp:1368-1641), called once per RHS evaluation after the RHS
// is assembled (NaiverStokes3d.cpp:58, euler3d.cpp:273).
//
// The reference transforms u, v, w with full 3-D FFTs (forward normalised by
// 1/N, backward unnormalised; fft.cpp:182-279), but only the modes of the
// shell |k - k_f| < 0.5 take part, so here the transforms are direct sums
// over the wavevectors with |k_d| <= K = floor(k_f + 1/2), done as three
// separable passes each way against precomputed twiddle tables:
//   forward  x (one warp per line) -> y (one warp per row) -> z + mode algebra
//            (one block, one warp per column)
//   backward z -> y -> x, the x pass fused with the RHS update.
// The fields are real, so only kx = 0..K is formed: the modes with kx < 0 are
// the conjugates of their mirrors (weight 2 in the sums).  The mean power is
// taken in mode space, <f.u> = sum over modes of Re(f^ . conj(u^)) (Parseval:
// the forced modes are exactly those of u^), so the fields are read twice in
// all, once each way.  160^3, K = 2: 0.50 -> 0.15 ms per RHS evaluation against
// block-wide reductions per line, a serial z pass and a third pass for <f.u>.
// Per mode (physicsModel.cpp:1480-1531): the solenoidal part s = u^ - (k.u^)k
// / |k|^2 and the compressive part c = u^ - s; s gains the helical term
// sigma (i k x s) / |k|; the shell energies E_s, E_c (modes with
// |kmag' - k_f| < 0.5, kmag' = 1 at k = 0) give theta = sqrt(|A - E_c| / E_s)
// and the forcing spectrum s (theta - 1) on the modes with |kmag - k_f| < 0.5
// (kmag unmodified, so k = 0 counts in E_s but is not forced).  In physical
// space (rho taken as 1, physicsModel.cpp:1617-1640):
//   R[1..3] -= f,   R[4] -= f.u - <f.u>.
//
// The band forcing at a fixed injection rate (NUC3D_FORCING_BAND, not in the
// reference) shares every pass: on the modes with 0 < |k| <= k_f it forces
// the solenoidal part s (no helical term) as f = s P / (2 E_b), E_b the band's
// solenoidal energy sum |s|^2 / 2.  Since s is orthogonal to the compressive
// part, sum Re(f . conj(u^)) = P: the mean power <f.u> is P.
#include "forcing_kernels.h"

namespace nuc3d {

namespace {

constexpr int kThreads = 128;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b) {  // a * conj(b)
    return make_double2(a.x * b.x + a.y * b.y, a.y * b.x - a.x * b.y);
}

// T[m * n + j] = exp(+i 2 pi k_m j / n), k_m = -K + m
__global__ void k_force_twiddle(double2 *T, int K, int n) {
    const int M = 2 * K + 1;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < M * n; t += gridDim.x * blockDim.x) {
        const int m = t / n, j = t % n;
        long long r = ((long long)(m - K) * j) % n;
        if (r < 0) r += n;
        double s, c;
        sincospi(2.0 * (double)r / (double)n, &s, &c);
        T[t] = make_double2(c, s);
    }
}

// sums v[0..NV) over the warp's lanes, NV a power of two: returns in each lane
// the total of the value with index lane >> (5 - log2 NV) (a butterfly that
// halves the values with every exchange)
template <int NV>
__device__ __forceinline__ double warp_sums(double (&v)[NV]) {
    const int lane = threadIdx.x & 31;
    int o = 16;
#pragma unroll
    for (int h = NV / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = lane & o;
#pragma unroll
        for (int j = 0; j < h; ++j) {
            const double keep = up ? v[j + h] : v[j], send = up ? v[j] : v[j + h];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    return v[0];
}
constexpr int pow2_above(int n) { return n <= 1 ? 1 : 2 * pow2_above((n + 1) / 2); }

// forward x: A[c][m][line] = sum_i u_c(i, line) exp(-i 2 pi m i / nx), m = 0..K
template <int K>
__global__ void __launch_bounds__(kThreads) k_force_fx(BoxDev b, const double2 *Tx, double2 *A) {
    constexpr int X = K + 1, NV = pow2_above(6 * X);
    const BoxParams &p = b.p;
    const int nx = p.n[0], lane = threadIdx.x & 31;
    const long long lines = (long long)p.n[1] * p.n[2];
    const long long line = blockIdx.x * (long long)(kThreads / 32) + (threadIdx.x >> 5);
    if (line >= lines) return;
    double acc[NV];  // [c][m][re, im]
#pragma unroll
    for (int s = 0; s < NV; ++s) acc[s] = 0.0;
    const double *const u = fieldW(b, 0) + line * nx;
    for (int i = lane; i < nx; i += 32) {
        const double f[3] = {u[i], u[b.np + i], u[2 * b.np + i]};
#pragma unroll
        for (int m = 0; m < X; ++m) {
            const double2 t = Tx[(K + m) * nx + i];
#pragma unroll
            for (int c = 0; c < 3; ++c) {  // u * conj(t)
                acc[(c * X + m) * 2] += f[c] * t.x;
                acc[(c * X + m) * 2 + 1] -= f[c] * t.y;
            }
        }
    }
    const double s = warp_sums<NV>(acc);
    constexpr int R = 32 / NV;  // lanes per value
    const int q = lane / R;
    if (lane % R == 0 && q < 6 * X)
        reinterpret_cast<double *>(A + (long long)(q / 2) * lines + line)[q % 2] = s;
}

// sum_j v_j conj(T[m * n + j]) for m = 0..M-1 of one row, by one warp; out
// receives the M sums
template <int K>
__device__ __forceinline__ void row_modes(const double2 *v, const double2 *T, int n, double2 *out,
                                          long long stride) {
    constexpr int M = 2 * K + 1, NV = pow2_above(2 * M);
    const int lane = threadIdx.x & 31;
    double acc[NV];
#pragma unroll
    for (int s = 0; s < NV; ++s) acc[s] = 0.0;
    for (int j = lane; j < n; j += 32) {
        const double2 a = v[j];
#pragma unroll
        for (int m = 0; m < M; ++m) {
            const double2 c = cmulc(a, T[m * n + j]);
            acc[2 * m] += c.x;
            acc[2 * m + 1] += c.y;
        }
    }
    const double s = warp_sums<NV>(acc);
    constexpr int R = 32 / NV;
    const int q = lane / R;
    if (lane % R == 0 && q < 2 * M)
        reinterpret_cast<double *>(out + (q / 2) * stride)[q % 2] = s;
}

// forward y: B[c][mx][my][k] = sum_j A[c][mx][j + ny k] conj(Ty[my][j])
template <int K>
__global__ void __launch_bounds__(kThreads)
    k_force_fy(const double2 *A, const double2 *Ty, double2 *B, int ny, int nz) {
    constexpr int M = 2 * K + 1;
    const int w = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (w >= 3 * (K + 1) * nz) return;
    const int k = w % nz, cmx = w / nz;
    row_modes<K>(A + ((long long)cmx * nz + k) * ny, Ty, ny, B + (long long)cmx * M * nz + k, nz);
}

__device__ __forceinline__ double kmag0_of(double kx, double ky, double kz) {
    return sqrt(kx * kx + ky * ky + kz * kz);
}

// forward z + mode algebra + shell energies + forcing spectrum + mean power
// (one block).  scal: [0] E_s, [1] E_c, [2] theta, [3] <f.u>
constexpr int kModeThreads = 512;
template <int K>
__global__ void __launch_bounds__(kModeThreads)
    k_force_modes(const double2 *B, const double2 *Tz, double2 *Fh, double *scal, ForceParams fp,
                  int nx, int ny, int nz) {
    constexpr int X = K + 1, M = 2 * K + 1, NM = X * M * M;
    const double inv_n = 1.0 / ((double)nx * ny * nz);
    __shared__ double2 sU[3][NM], sS[3][NM];  // u^ and s (after the helical term)
    __shared__ double red[3][kModeThreads / 32], tot[3];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int col = warp; col < 3 * X * M; col += kModeThreads / 32)  // (c, mx, my)
        row_modes<K>(B + (long long)col * nz, Tz, nz, &sU[col / (X * M)][col % (X * M)], X * M);
    __syncthreads();
    auto sum = [&](int q, double v) {  // v over the block into tot[q], in a fixed order
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) red[q][warp] = v;
        __syncthreads();
        if (threadIdx.x == 0) {
            double s = 0.0;
            for (int w = 0; w < kModeThreads / 32; ++w) s += red[q][w];
            tot[q] = s;
        }
        __syncthreads();
    };
    // mode index: (mx M + my) + X M mz
    double e2[2] = {0.0, 0.0};
    for (int mode = threadIdx.x; mode < NM; mode += kModeThreads) {
        const int mx = (mode / M) % X, my = mode % M, mz = mode / (X * M);
        const double kk[3] = {(double)mx, (double)(my - K), (double)(mz - K)};
        const double wt = mx == 0 ? 0.5 : 1.0;  // 1/2, twice with the mirror mode
        double2 uh[3];
        for (int c = 0; c < 3; ++c) {  // fft.cpp:277-278
            uh[c] = make_double2(sU[c][mode].x * inv_n, sU[c][mode].y * inv_n);
            sU[c][mode] = uh[c];
        }
        const double kmag0 = kmag0_of(kk[0], kk[1], kk[2]);
        const double kmag = kmag0 < 1e-6 ? 1.0 : kmag0;
        const double ku_re = (kk[0] * uh[0].x + kk[1] * uh[1].x + kk[2] * uh[2].x) / kmag;
        const double ku_im = (kk[0] * uh[0].y + kk[1] * uh[1].y + kk[2] * uh[2].y) / kmag;
        double2 s[3], cc[3];
        for (int c = 0; c < 3; ++c) {
            s[c] = make_double2(uh[c].x - ku_re * kk[c] / kmag, uh[c].y - ku_im * kk[c] / kmag);
            cc[c] = make_double2(uh[c].x - s[c].x, uh[c].y - s[c].y);
        }
        auto energy = [&](const double2 (&v)[3]) {
            return wt * (v[0].x * v[0].x + v[1].x * v[1].x + v[2].x * v[2].x + v[0].y * v[0].y +
                         v[1].y * v[1].y + v[2].y * v[2].y);
        };
        if (fp.band) {
            // band forcing: the solenoidal part alone, energy over 0 < |k| <= k_f
            if (kmag0 > 0.0 && kmag0 <= fp.k + 1e-12) e2[0] += energy(s);
        } else {
            // helical term (physicsModel.cpp:1512-1526)
            const double2 t[3] = {s[0], s[1], s[2]};
            s[0].x += fp.hel * (-(kk[1] * t[2].y - kk[2] * t[1].y) / kmag);
            s[1].x += fp.hel * ((kk[0] * t[2].y - kk[2] * t[0].y) / kmag);
            s[2].x += fp.hel * (-(kk[0] * t[1].y - kk[1] * t[0].y) / kmag);
            s[0].y += fp.hel * ((kk[1] * t[2].x - kk[2] * t[1].x) / kmag);
            s[1].y += fp.hel * (-(kk[0] * t[2].x - kk[2] * t[0].x) / kmag);
            s[2].y += fp.hel * ((kk[0] * t[1].x - kk[1] * t[0].x) / kmag);
            if (fabs(kmag - fp.k) < 0.5) {
                e2[0] += energy(s);
                e2[1] += energy(cc);
            }
        }
        for (int c = 0; c < 3; ++c) sS[c][mode] = s[c];
    }
    sum(0, e2[0]);
    sum(1, e2[1]);
    // shell: theta - 1 multiplies the shell's modes; band: the gain P / (2 E_b)
    // (zero for a band of exactly zero energy; one that holds only rounding noise,
    // E_b ~ 1e-33, is driven by its noise at the full rate)
    const double theta = fp.band ? 0.0 : sqrt(fabs(fp.amp - tot[1]) / tot[0]);
    const double gain = fp.band ? (tot[0] > 0.0 ? fp.amp / (2.0 * tot[0]) : 0.0) : theta - 1.0;
    double power = 0.0;
    for (int mode = threadIdx.x; mode < NM; mode += kModeThreads) {
        const int mx = (mode / M) % X, my = mode % M, mz = mode / (X * M);
        const double kmag = kmag0_of(mx, my - K, mz - K);  // unmodified at k = 0
        const bool on = fp.band ? (kmag > 0.0 && kmag <= fp.k + 1e-12) : fabs(kmag - fp.k) < 0.5;
        for (int c = 0; c < 3; ++c) {
            const double2 s = sS[c][mode];
            const double2 f =
                on ? make_double2(s.x * gain, s.y * gain) : make_double2(0.0, 0.0);
            Fh[c * NM + mode] = f;
            power += (mx == 0 ? 1.0 : 2.0) * (f.x * sU[c][mode].x + f.y * sU[c][mode].y);
        }
    }
    sum(2, power);
    if (threadIdx.x == 0) {
        scal[0] = tot[0];
        scal[1] = tot[1];
        scal[2] = fp.band ? gain : theta;
        scal[3] = tot[2];
    }
}

// backward z: S[c][mx][my][k] = sum_mz Fh[c][mx,my,mz] Tz[mz][k]
template <int K>
__global__ void k_force_bz(const double2 *Fh, const double2 *Tz, double2 *S, int nz) {
    constexpr int X = K + 1, M = 2 * K + 1;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * X * M * nz) return;
    const int k = t % nz, col = t / nz, c = col / (X * M), xy = col % (X * M);
    double2 s = make_double2(0.0, 0.0);
#pragma unroll
    for (int mz = 0; mz < M; ++mz) {
        const double2 v = cmul(Fh[c * X * M * M + xy + X * M * mz], Tz[mz * nz + k]);
        s.x += v.x;
        s.y += v.y;
    }
    S[t] = s;
}

// backward y: Y[c][mx][j + ny k] = sum_my S[c][mx][my][k] Ty[my][j]
template <int K>
__global__ void k_force_by(const double2 *S, const double2 *Ty, double2 *Y, int ny, int nz) {
    constexpr int X = K + 1, M = 2 * K + 1;
    const long long lines = (long long)ny * nz;
    const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (t >= 3 * X * lines) return;
    const int cmx = (int)(t / lines), line = (int)(t - cmx * lines);
    const int k = line / ny, j = line - k * ny;
    double2 s = make_double2(0.0, 0.0);
#pragma unroll
    for (int my = 0; my < M; ++my) {
        const double2 v = cmul(S[((long long)cmx * M + my) * nz + k], Ty[my * ny + j]);
        s.x += v.x;
        s.y += v.y;
    }
    Y[t] = s;
}

// backward x and the RHS update, one warp per line:
// f_c(i) = Re Y[c][0] + 2 Re sum_{m > 0} Y[c][m][line] Tx[m][i]
template <int K, typename Bk>
__global__ void __launch_bounds__(kThreads)
    k_force_bx(BoxDev b, const double2 *Tx, const double2 *Y, const double *scal) {
    constexpr int X = K + 1;
    const BoxParams &p = b.p;
    const int nx = p.n[0], lane = threadIdx.x & 31;
    const long long lines = (long long)p.n[1] * p.n[2], np = b.np;
    const long long line = blockIdx.x * (long long)(kThreads / 32) + (threadIdx.x >> 5);
    if (line >= lines) return;
    double2 y[3][X];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < X; ++m) {
            y[c][m] = Y[(long long)(c * X + m) * lines + line];
            if (m > 0) {
                y[c][m].x *= 2.0;
                y[c][m].y *= 2.0;
            }
        }
    const double aver = scal[3];
    const double *const u = fieldW(b, 0) + line * nx;
    Bk *const r = fieldR<Bk>(b, 0) + line * nx;
    for (int i = lane; i < nx; i += 32) {
        double f[3] = {y[0][0].x, y[1][0].x, y[2][0].x};
#pragma unroll
        for (int m = 1; m < X; ++m) {
            const double2 t = Tx[(K + m) * nx + i];
#pragma unroll
            for (int c = 0; c < 3; ++c) f[c] += y[c][m].x * t.x - y[c][m].y * t.y;
        }
        const double fu = f[0] * u[i] + f[1] * u[np + i] + f[2] * u[2 * np + i];  // rho0 = 1
#pragma unroll
        for (int c = 0; c < 3; ++c) r[(1 + c) * np + i] = Bk(double(r[(1 + c) * np + i]) - f[c]);
        r[4 * np + i] = Bk(double(r[4 * np + i]) - (fu - aver));
    }
}

int grid_for(long long n) {
    long long g = (n + 255) / 256;
    return (int)(g < 1 ? 1 : (g > 4096 ? 4096 : g));
}

template <int K, typename Bk>
cudaError_t launch_k(const BoxDev &b, const ForceScratch &s, ForceParams fp, cudaStream_t st) {
    const BoxParams &p = b.p;
    const int nx = p.n[0], ny = p.n[1], nz = p.n[2];
    const long long lines = (long long)ny * nz;
    constexpr int X = K + 1, M = 2 * K + 1, W = kThreads / 32;
    auto blocks = [](long long n, int per) { return (unsigned)((n + per - 1) / per); };
    k_force_fx<K><<<blocks(lines, W), kThreads, 0, st>>>(b, s.tx, s.a);
    k_force_fy<K><<<blocks(3LL * X * nz, W), kThreads, 0, st>>>(s.a, s.ty, s.b, ny, nz);
    k_force_modes<K><<<1, kModeThreads, 0, st>>>(s.b, s.tz, s.fh, s.scal, fp, nx, ny, nz);
    k_force_bz<K><<<blocks(3LL * X * M * nz, 256), 256, 0, st>>>(s.fh, s.tz, s.b, nz);
    k_force_by<K><<<blocks(3LL * X * lines, 256), 256, 0, st>>>(s.b, s.ty, s.a, ny, nz);
    k_force_bx<K, Bk><<<blocks(lines, W), kThreads, 0, st>>>(b, s.tx, s.a, s.scal);
    return cudaGetLastError();
}

}  // namespace

int forcing_K(double k_f) { return (int)std::floor(k_f + 0.5); }

size_t forcing_scratch_bytes(const BoxParams &p, double k_f) {
    const int K = forcing_K(k_f), X = K + 1, M = 2 * K + 1;
    const long long lines = (long long)p.n[1] * p.n[2];
    size_t b = 0;
    b += sizeof(double2) * (size_t)M * (p.n[0] + p.n[1] + p.n[2]);  // twiddles
    b += sizeof(double2) * 3 * (size_t)X * lines;                   // a
    b += sizeof(double2) * 3 * (size_t)X * M * p.n[2];              // b
    b += sizeof(double2) * 3 * (size_t)X * M * M;                   // fh
    b += 8 * sizeof(double);                                        // scal
    return b + 8 * 256;
}

ForceScratch forcing_layout(const BoxParams &p, double k_f, void *base) {
    const int K = forcing_K(k_f), X = K + 1, M = 2 * K + 1;
    const long long lines = (long long)p.n[1] * p.n[2];
    char *c = static_cast<char *>(base);
    auto take = [&](size_t bytes) {
        char *r = c;
        c += (bytes + 255) / 256 * 256;
        return r;
    };
    ForceScratch s{};
    s.tx = reinterpret_cast<double2 *>(take(sizeof(double2) * M * p.n[0]));
    s.ty = reinterpret_cast<double2 *>(take(sizeof(double2) * M * p.n[1]));
    s.tz = reinterpret_cast<double2 *>(take(sizeof(double2) * M * p.n[2]));
    s.a = reinterpret_cast<double2 *>(take(sizeof(double2) * 3 * (size_t)X * lines));
    s.b = reinterpret_cast<double2 *>(take(sizeof(double2) * 3 * (size_t)X * M * p.n[2]));
    s.fh = reinterpret_cast<double2 *>(take(sizeof(double2) * 3 * (size_t)X * M * M));
    s.scal = reinterpret_cast<double *>(take(8 * sizeof(double)));
    return s;
}

cudaError_t forcing_prepare(const BoxParams &p, double k_f, const ForceScratch &s, cudaStream_t st) {
    const int K = forcing_K(k_f), M = 2 * K + 1;
    k_force_twiddle<<<grid_for((long long)M * p.n[0]), 256, 0, st>>>(s.tx, K, p.n[0]);
    k_force_twiddle<<<grid_for((long long)M * p.n[1]), 256, 0, st>>>(s.ty, K, p.n[1]);
    k_force_twiddle<<<grid_for((long long)M * p.n[2]), 256, 0, st>>>(s.tz, K, p.n[2]);
    return cudaGetLastError();
}

template <typename Bk>
cudaError_t launch_forcing(const BoxDev &b, const ForceScratch &s, ForceParams fp, cudaStream_t st) {
    switch (fp.K) {
        case 0: return launch_k<0, Bk>(b, s, fp, st);
        case 1: return launch_k<1, Bk>(b, s, fp, st);
        case 2: return launch_k<2, Bk>(b, s, fp, st);
        case 3: return launch_k<3, Bk>(b, s, fp, st);
        default: return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_forcing<double>(const BoxDev &, const ForceScratch &, ForceParams,
                                            cudaStream_t);
template cudaError_t launch_forcing<float>(const BoxDev &, const ForceScratch &, ForceParams,
                                           cudaStream_t);

}  // namespace nuc3d
