// band_reduce.cuh -- dense symmetric matrix -> band of half-bandwidth 32 (the first stage of the
// two-stage tridiagonal reduction; band_eig.cuh chases the band).
#pragma once

#include <cuda_runtime.h>

#include "band_eig.cuh"

namespace dvr3d {

struct BandReduce {
    double *A;         // n x n, lower triangle used, lda a multiple of 8; overwritten. With `keep`
    long long lda;     // panel q's block reflector vectors V stay in A[32 (q + 1) :, 32 q : 32 q + 32]
    int n;
    bool keep;         // keep V and T for launch_band_reduce_back
    double *C;         // out: the band's lower triangle, element (i, j) at C[j (kBandLd - 1) + i]
                       // (band_storage_doubles(n))
    double *T;         // [band_reduce_panels(n)][32 x 32] triangular factors
    double *work;      // band_reduce_work_doubles(n)
    cudaStream_t side; // the updates run here, beside the panels; joined before the call's last work on st
    cudaEvent_t ready, done;  // of the caller's, timing disabled
    int *err;          // cleared by the caller; set to kDevBarrierTimeout when a wait runs out
    unsigned long long wait_limit;  // polls of a wait, 0: the default
};

// Whether the current device takes the panel kernel's cluster.
bool band_reduce_available();
constexpr int kBandLd = kBandMaxBw + 1;
inline size_t band_storage_doubles(int n) { return (size_t)n * kBandLd; }
inline int band_reduce_panels(int n) { return (n + kBandMaxBw - 1) / kBandMaxBw; }
size_t band_reduce_work_doubles(int n);
cudaError_t launch_band_reduce(const BandReduce &b, cudaStream_t st);
// Z (n x nev, ldz even) <- Q Z with A = Q (band) Q^T; work: band_reduce_back_doubles(nev).
size_t band_reduce_back_doubles(int nev);
cudaError_t launch_band_reduce_back(const BandReduce &b, double *Z, long long ldz, int nev, double *work, cudaStream_t st);

}  // namespace dvr3d
