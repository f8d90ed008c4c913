// ic.cuh -- device-side building blocks of the initial conditions, shared by
// the ic entry points, the differentiable model and the ensemble.
#pragma once

#include "common.cuh"
#include "fft.cuh"

namespace conan {

enum { IC_SCALE_FREE = 0, IC_CDM = 1 };

struct ICFilter {
    int mode;
    double ns;      // spectral slope
    double t;       // Fourier::scale parameter, scale * N / L (cells)
    double L;       // box size
    double Omega0;  // CDM branch
    double h;       // H0 / 100 (CDM branch)
};

// FP64 scratch of the field functions below (`part`): the partial sums of
// IC_BLOCKS blocks, a few scalars behind them, and from IC_PART on the filter
// tables of the meshes that use them: 3D, IC_TABLE_N cells per side and more
// (an eighth of the modes' values; below that a launch costs more than the
// values, and in 2D a quarter of few modes).
constexpr int IC_BLOCKS = 512, IC_PART = 1024, IC_TABLE_N = 32;
enum { IC_VAR = 0, IC_AMP, IC_SCALE, IC_DOT };  // scalars at part + IC_BLOCKS
inline size_t ic_table_values(const Mesh &m) {
    const size_t h = m.n / 2 + 1;
    return m.R == 3 && m.n >= IC_TABLE_N ? h * h * h : 0;
}
inline size_t ic_scratch(const Mesh &m) {
    const size_t np = ic_table_values(m);
    return IC_PART + (np ? np + m.n / 2 + 1 : 0);
}

int check_ic_params(const conan_ic_params *p);

// Philox white noise into a device mesh.
template <typename T> int noise_device(const Mesh &m, unsigned long long seed, T *mesh, cudaStream_t st);
// Noise mesh (kept) -> density mesh (may be the same; uses spec as scratch).
template <typename T>
int grf_device(const conan_ic_params &p, const Mesh &m, T *noise, T *mesh, typename Cplx<T>::type *spec, FFTPair &fft,
               double *part, cudaStream_t st);
// Adjoint of grf_device: dL/dw from dL/d(density) (dbar is overwritten).
template <typename T>
int grf_adjoint_device(const conan_ic_params &p, const Mesh &m, const T *w, T *dbar, T *wbar,
                       typename Cplx<T>::type *spec, typename Cplx<T>::type *spec2, T *tmp, FFTPair &fft,
                       double *part, cudaStream_t st);
// Density mesh -> potential mesh, in place (a symmetric operator: it is its
// own adjoint).
template <typename T>
int potential_device(const Mesh &m, double L, T *mesh, typename Cplx<T>::type *spec, FFTPair &fft,
                     cudaStream_t st);

}  // namespace conan
