// fft.cuh -- cuFFT real<->half-complex plans over the cubic meshes of Mesh.
#pragma once

#include "common.cuh"

namespace conan {

// R2C / C2R pair for `batch` meshes of n^R cells stored back to back
// (real stride n^R, spectrum stride nh*n^(R-1)). Axis 0 is the fastest axis
// of both the real mesh and the half-complex spectrum. The work area is
// supplied by the owner so several plans can share one buffer.
struct FFTPair {
    cufftHandle r2c = 0, c2r = 0;
    size_t work_bytes = 0;
    bool dbl = false;

    int create(const Mesh &m, bool is_double, int batch) {
        return make(m.R, m.n, 1LL << m.cshift, (long long)m.mspec, is_double, batch);
    }
    // The same half-spectrum layout with the slowest axis left in real space: 2D
    // transforms of every z plane of 3D meshes, 1D ones of every row of 2D ones.
    int create_planes(const Mesh &m, bool is_double, int batch) {
        const long long rows = m.R == 3 ? m.n : 1;  // per plane
        return make(m.R - 1, m.n, rows * m.n, rows * m.nh, is_double, batch * m.n);
    }
    // `batch` pairs of rank-dimensional transforms of n cells per side, real_dist
    // and cplx_dist values apart. A pair that cannot be made whole has no
    // handles, so that they always stand for plans.
    int make(int rank, int side, long long real_dist, long long cplx_dist, bool is_double, int batch) {
        dbl = is_double;
        cufftResult r = plan(rank, side, real_dist, cplx_dist, batch);
        if (r == CUFFT_ALLOC_FAILED) {  // see alloc_retry
            destroy();
            cudaGetLastError();
            release_caches();
            r = plan(rank, side, real_dist, cplx_dist, batch);
        }
        if (r == CUFFT_SUCCESS) return CONAN_OK;
        destroy();
        return set_error(CONAN_ERR_CUDA, "%d FFT plans of dimension %d and %d cells failed: cufft error %d", batch, rank,
                         side, (int)r);
    }
    cufftResult plan(int rank, int side, long long real_dist, long long cplx_dist, int batch) {
        int n[3] = {side, side, side};
        size_t w1 = 0, w2 = 0;
        cufftResult r = cufftCreate(&r2c);
        if (r == CUFFT_SUCCESS) r = cufftCreate(&c2r);
        if (r == CUFFT_SUCCESS) r = cufftSetAutoAllocation(r2c, 0);
        if (r == CUFFT_SUCCESS) r = cufftSetAutoAllocation(c2r, 0);
        if (r == CUFFT_SUCCESS)
            r = cufftMakePlanMany(r2c, rank, n, nullptr, 1, (int)real_dist, nullptr, 1, (int)cplx_dist,
                                  dbl ? CUFFT_D2Z : CUFFT_R2C, batch, &w1);
        if (r == CUFFT_SUCCESS)
            r = cufftMakePlanMany(c2r, rank, n, nullptr, 1, (int)cplx_dist, nullptr, 1, (int)real_dist,
                                  dbl ? CUFFT_Z2D : CUFFT_C2R, batch, &w2);
        work_bytes = w1 > w2 ? w1 : w2;
        return r;
    }
    int bind(void *work, cudaStream_t s) {
        CONAN_CUFFT(cufftSetWorkArea(r2c, work));
        CONAN_CUFFT(cufftSetWorkArea(c2r, work));
        CONAN_CUFFT(cufftSetStream(r2c, s));
        CONAN_CUFFT(cufftSetStream(c2r, s));
        return CONAN_OK;
    }
    void destroy() {
        if (r2c) cufftDestroy(r2c);
        if (c2r) cufftDestroy(c2r);
        r2c = c2r = 0;
    }
    int forward(float *in, cufftComplex *out) {
        CONAN_CUFFT(cufftExecR2C(r2c, in, out));
        return CONAN_OK;
    }
    int forward(double *in, cufftDoubleComplex *out) {
        CONAN_CUFFT(cufftExecD2Z(r2c, in, out));
        return CONAN_OK;
    }
    // Unnormalised inverse; overwrites `in`.
    int inverse(cufftComplex *in, float *out) {
        CONAN_CUFFT(cufftExecC2R(c2r, in, out));
        return CONAN_OK;
    }
    int inverse(cufftDoubleComplex *in, double *out) {
        CONAN_CUFFT(cufftExecZ2D(c2r, in, out));
        return CONAN_OK;
    }
};

}  // namespace conan
