// Shell-binned spectra of one box (spectra_kernels.cu).  Internal.
#pragma once

#include <cuda_runtime.h>

#include "rhs_kernels.h"

namespace nuc3d {

constexpr int kSpectra = 9;         // kin, kinc, kins, kinl, kinr, hel, ens, den, pre
constexpr int kSpectraFields = 7;   // transformed fields: u, v, w, hel, ens, rho, p
constexpr int kSpecBlocks = 296;    // fixed binning grid (2 x 148): results do not depend on the batch

inline int spectra_kmax(const BoxParams &p) {
    int m = p.n[0] < p.n[1] ? p.n[0] : p.n[1];
    return (m < p.n[2] ? m : p.n[2]) / 2;
}
// The transforms' cuFFT plan of one box size, made on first use and again when
// the size changes (making one takes about 2 ms of host time).  It owns no work
// area: a call hands it part of its scratch.
struct SpectraPlan {
    int n[3] = {0, 0, 0};
    int handle = 0;
    int batch = 1;    // fields per transform call
    size_t work = 0;  // bytes of the work area
    bool made = false;
    int prepare(const BoxParams &p, cudaStream_t st);  // cuFFT status
    void release();
};
// device scratch of a spectra evaluation: the seven transformed fields, the
// per-block shell partials, the result and the plan's work area
size_t spectra_scratch_bytes(const BoxParams &p, size_t work);
// Spectra of box b (W must hold the primitives of U[0]) by a prepared plan;
// *d_out receives the device address (in scratch) of the kSpectra * kmax
// results.  Returns a CUDA error; *fft_status is set when cuFFT fails.
cudaError_t launch_spectra(const BoxDev &b, const SpectraPlan &plan, void *scratch,
                           double **d_out, int *fft_status, cudaStream_t st);

}  // namespace nuc3d
