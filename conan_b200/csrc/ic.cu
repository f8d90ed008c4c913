// ic.cu -- initial conditions on the GPU: white noise, the Gaussian random
// field of the `ic` tool (src/ic/ic.cc:37-98), its potential
// (src/ic/ic.cc:100-117) and the Zel'dovich displacement record
// (src/ic/ic.cc:119-146). Meshes are real with axis 0 fastest; all
// filtering happens on the R2C half spectrum.
#include <cmath>
#include <vector>

#include "hostio.cuh"
#include "ic.cuh"
#include "pm.cuh"

namespace conan {

__global__ void k_noise_philox_f64(double *__restrict__ out, size_t n, unsigned long long seed) {
    size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * j >= n) return;
    double z0, z1;
    philox_normal_pair(seed, j, &z0, &z1);
    out[2 * j] = z0;
    if (2 * j + 1 < n) out[2 * j + 1] = z1;
}

template <typename T>
__global__ void k_noise_philox(T *__restrict__ out, size_t n, unsigned long long seed) {
    size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (2 * j >= n) return;
    double z0, z1;
    philox_normal_pair(seed, j, &z0, &z1);
    out[2 * j] = (T)z0;
    if (2 * j + 1 < n) out[2 * j + 1] = (T)z1;
}

// CDM<R>, src/ic/ic.cc:14-35, at physical k (kspace(N, L)).
__device__ inline double ic_cdm(const ICFilter &F, double kk) {
    const double e1 = 2.718281828459045, Theta = 2.7255 / 2.7, A = 1122670;
    double q = kk * Theta * Theta / (F.Omega0 * F.h), L0 = log(2 * e1 + 1.8 * q),
           C0 = 14.2 + 731.0 / (1 + 62.5 * q), T0 = L0 / (L0 + C0 * q * q);
    return sqrt(A * pow(kk, F.ns) * T0 * T0);
}

// Spectral factor of the mode with integer wave vector kv, |kv|^2 = k2 (see ICFilter).
__device__ inline double ic_power(const ICFilter &F, const Mesh &m, const int *kv, long long k2) {
    if (F.mode == IC_CDM) return ic_cdm(F, sqrt((double)k2) * (2 * M_PI / F.L));
    // Scale-free: k in radians per cell (kspace(N, N), src/ic/ic.cc:61-64),
    // sqrt(P(|k|)) with P = k^ns; times Fourier::scale(t) (fourier.hh:79-100)
    // where the caller smooths.
    double s2 = 0;
    for (int a = 0; a < m.R; ++a) {
        const double k = kv[a] * (2 * M_PI / m.n);
        s2 += k * k;
    }
    return sqrt(pow(sqrt(s2), F.ns));
}
__device__ inline double ic_smooth(const ICFilter &F, int n, int kv) {
    return exp(F.t * (cos(kv * (2 * M_PI / n)) - 1));
}

// Filter values in tables (3D meshes of IC_TABLE_N cells per side and more):
// p[|kz|][|ky|][|kx|] the spectral factors of one octant (a factor only sees
// the squares of its wave numbers), e[|k|] the smoothing of one axis. Both
// hold what the formulas give for those modes, so a filter's bits do not
// depend on the table. Null: every mode evaluates the formulas.
struct ICTable {
    const double *p, *e;
};

// An eighth of the modes' pow and sqrt, and n/2 + 1 exp and cos instead of
// three per mode: bound by FP64 instructions (0.24 ms at 512^3, where the modes'
// own evaluation took 2.29 ms of the variance and 0.95 of the filter).
__global__ void __launch_bounds__(256) k_ic_table(ICFilter F, Mesh m, double *__restrict__ p, double *__restrict__ e) {
    const int h = m.n / 2 + 1, kx = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (kx >= h) return;
    const int kv[3] = {kx, (int)blockIdx.y, (int)blockIdx.z};
    if (kv[1] == 0 && kv[2] == 0) e[kx] = ic_smooth(F, m.n, kx);
    p[((size_t)kv[2] * h + kv[1]) * h + kx] =
        ic_power(F, m, kv, (long long)kv[0] * kv[0] + (long long)kv[1] * kv[1] + (long long)kv[2] * kv[2]);
}

// Half-spectrum element with its row (the indices along y and z) and its kx;
// walking by steps smaller than a mesh needs no division.
struct ICMode {
    size_t row;
    int kx;
    __device__ ICMode(size_t e, const Mesh &m) {
        int kv[3];
        spec_k2(e, m, kv);
        kx = kv[0];
        row = (e - (size_t)kx) / (unsigned)m.nh;
    }
    __device__ void step(size_t rows, int k, const Mesh &m) {  // by rows * nh + k, k < nh
        row += rows;
        kx += k;
        if (kx >= m.nh) {
            kx -= m.nh;
            ++row;
        }
    }
    __device__ long long wave(const Mesh &m, int *kv) const {
        kv[0] = kx;
        long long s = (long long)kx * kx;
        for (int a = 1; a < m.R; ++a) {
            const int w = wave_index((int)((row >> ((a - 1) * m.shift)) & (size_t)(m.n - 1)), m.n);
            kv[a] = w;
            s += (long long)w * w;
        }
        return s;
    }
};

// Filter value of a mode.
__device__ inline double ic_filter_at(const ICFilter &F, const ICTable &tab, const Mesh &m, const ICMode &mode,
                                      bool with_s) {
    int kv[3];
    const long long k2 = mode.wave(m, kv);
    if (tab.p) {
        const int h = m.n / 2 + 1;
        const double p = __ldg(tab.p + ((size_t)abs(kv[2]) * h + abs(kv[1])) * h + kv[0]);
        if (!with_s) return p;
        return p * (__ldg(tab.e + kv[0]) * __ldg(tab.e + abs(kv[1])) * __ldg(tab.e + abs(kv[2])));
    }
    const double p = ic_power(F, m, kv, k2);
    if (!with_s) return p;
    double s = 1.0;
    for (int a = 0; a < m.R; ++a) s *= ic_smooth(F, m.n, kv[a]);
    return p * s;
}

// Per-block sums of w |x_hat|^2 PS(k)^2 over the half spectrum (DC excluded):
// the variance of the smoothed field by Parseval. Each thread sums its modes
// in order (the sum's bits follow from that and the grid), with four loads in
// flight and no index division (512^3: 2.29 -> 0.71 ms).
template <typename T>
__global__ void __launch_bounds__(256) k_ic_var(const typename Cplx<T>::type *__restrict__ spec, Mesh m, ICFilter F,
                                                ICTable tab, double *__restrict__ part) {
    double s = 0;
    const size_t stride = (size_t)gridDim.x * blockDim.x, srows = stride / (unsigned)m.nh;
    const int sk = (int)(stride - srows * (unsigned)m.nh);
    size_t e0 = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    ICMode mode(e0, m);
    for (; e0 < m.spec; e0 += 4 * stride) {
        typename Cplx<T>::type z[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (e0 + j * stride < m.spec) z[j] = spec[e0 + j * stride];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const size_t e = e0 + j * stride;
            if (e != 0 && e < m.spec) {
                const double f = ic_filter_at(F, tab, m, mode, true);
                s += spec_weight(mode.kx, m.n) * ((double)z[j].x * z[j].x + (double)z[j].y * z[j].y) * f * f;
            }
            mode.step(srows, sk, m);
        }
    }
    s = block_sum<double>(s);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// Four modes at e0 (a multiple of 4), those beyond the end left out.
__device__ inline void load4(const cufftComplex *p, size_t e0, size_t n, cufftComplex *z) {
    if (e0 + 4 <= n) {
        const float4 *v = reinterpret_cast<const float4 *>(p + e0);
        const float4 a = v[0], b = v[1];
        z[0] = make_float2(a.x, a.y);
        z[1] = make_float2(a.z, a.w);
        z[2] = make_float2(b.x, b.y);
        z[3] = make_float2(b.z, b.w);
    } else {
        for (int j = 0; j < 4; ++j)
            if (e0 + j < n) z[j] = p[e0 + j];
    }
}
__device__ inline void store4(cufftComplex *p, size_t e0, size_t n, const cufftComplex *z) {
    if (e0 + 4 <= n) {
        float4 *v = reinterpret_cast<float4 *>(p + e0);
        v[0] = make_float4(z[0].x, z[0].y, z[1].x, z[1].y);
        v[1] = make_float4(z[2].x, z[2].y, z[3].x, z[3].y);
    } else {
        for (int j = 0; j < 4; ++j)
            if (e0 + j < n) p[e0 + j] = z[j];
    }
}
__device__ inline void load4(const cufftDoubleComplex *p, size_t e0, size_t n, cufftDoubleComplex *z) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (e0 + j < n) z[j] = p[e0 + j];
}
__device__ inline void store4(cufftDoubleComplex *p, size_t e0, size_t n, const cufftDoubleComplex *z) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
        if (e0 + j < n) p[e0 + j] = z[j];
}

// Scalars that stay on the device, so that no filter waits for the host: sums
// the IC_BLOCKS partials in part, in order, into scal.
// what 0: the variance of the smoothed field and what follows from it; 1: the
// y . dbar of the field's adjoint, giving the factor of its second term.
__global__ void __launch_bounds__(IC_BLOCKS) k_ic_scalars(const double *__restrict__ part, int what, double sigma,
                                                          double nc, double *__restrict__ scal) {
    __shared__ double v[IC_BLOCKS];
    v[threadIdx.x] = part[threadIdx.x];
    __syncthreads();
    if (threadIdx.x != 0) return;
    double s = 0;
#pragma unroll 16
    for (int i = 0; i < IC_BLOCKS; ++i) s += v[i];
    if (what == 0) {
        const double var = s / (nc * nc);  // mean of the smoothed field squared
        scal[IC_VAR] = var;
        scal[IC_AMP] = sigma / sqrt(var);
        scal[IC_SCALE] = sigma / (nc * sqrt(var));
    } else {
        scal[IC_DOT] = -(scal[IC_AMP] / scal[IC_VAR]) * s / nc;
    }
}

// out = in * f(k)^power * scale * *amp (amp null: 1), DC = 0 (f the scale-free
// or CDM filter; out may be in). Four modes per thread: one index division
// and 16-byte accesses for them (512^3: 0.95 ms with a pow per mode and a
// division each, 0.35 with both gone).
template <typename T>
__global__ void __launch_bounds__(256)
    k_ic_filter(const typename Cplx<T>::type *in, typename Cplx<T>::type *out, Mesh m, ICFilter F, ICTable tab,
                bool with_s, int power, double scale, const double *__restrict__ amp) {
    const size_t e0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e0 >= m.spec) return;
    typename Cplx<T>::type z[4];
    load4(in, e0, m.spec, z);
    ICMode mode(e0, m);
    const double sc = amp ? scale * *amp : scale;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        if (e0 + j < m.spec) {
            double f = 0.0;
            if (e0 + j != 0) {
                const double v = ic_filter_at(F, tab, m, mode, with_s);
                f = (power == 2 ? v * v : v) * sc;
            }
            z[j].x = (T)((double)z[j].x * f);
            z[j].y = (T)((double)z[j].y * f);
        }
        mode.step(0, 1, m);
    }
    store4(out, e0, m.spec, z);
}

// spec *= gsp / |n|^2 (physical -1/k^2 with the 1/size normalisation folded
// into gsp), DC = 0. Four modes per thread: 0.32 -> 0.24 ms at 512^3.
template <typename T>
__global__ void __launch_bounds__(256) k_ic_potential(typename Cplx<T>::type *spec, Mesh m, double gsp) {
    const size_t e0 = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * 4;
    if (e0 >= m.spec) return;
    typename Cplx<T>::type z[4];
    load4(spec, e0, m.spec, z);
    ICMode mode(e0, m);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int kv[3];
        const long long k2 = mode.wave(m, kv);
        const double g = k2 > 0 ? gsp / (double)k2 : 0.0;
        z[j].x = (T)((double)z[j].x * g);
        z[j].y = (T)((double)z[j].y * g);
        mode.step(0, 1, m);
    }
    store4(spec, e0, m.spec, z);
}

// out = in * i sin(2 pi n_axis / N) * scale (Fourier::derivative,
// src/base/fourier.hh:111-118, on kspace(N, N)).
template <typename T>
__global__ void k_ic_deriv(const typename Cplx<T>::type *__restrict__ in,
                           typename Cplx<T>::type *__restrict__ out, Mesh m, int axis, double scale) {
    size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= m.spec) return;
    int kv[3];
    spec_k2(e, m, kv);
    double s = sin(kv[axis] * (2 * M_PI / m.n)) * scale;
    auto z = in[e];
    typename Cplx<T>::type r;
    r.x = (T)(-(double)z.y * s);
    r.y = (T)((double)z.x * s);
    out[e] = r;
}

// AoS scatter of one component: out[i * R + c] = in[i].
template <typename T>
__global__ void k_interleave(const T *__restrict__ in, double *__restrict__ out, size_t n, int R, int c) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i * R + c] = (double)in[i];
}

int check_ic_params(const conan_ic_params *p) {
    if (!p) return set_error(CONAN_ERR_ARG, "null parameters");
    if (p->dim < 1 || p->dim > 3)
        return set_error(CONAN_ERR_UNSUPPORTED, "only 1, 2 and 3 dimensions supported (dim = %d)", p->dim);
    if (p->mbits < 1 || p->mbits > 12) return set_error(CONAN_ERR_ARG, "mbits = %d out of range", p->mbits);
    long long cells = 1;
    for (int i = 0; i < p->dim; ++i) cells *= 1LL << p->mbits;
    if (cells >= (1LL << 32)) return set_error(CONAN_ERR_ARG, "mesh of %lld cells too large", cells);
    if (!(p->size > 0)) return set_error(CONAN_ERR_ARG, "box size must be positive");
    if (p->precision != CONAN_FP32 && p->precision != CONAN_FP64)
        return set_error(CONAN_ERR_ARG, "precision must be CONAN_FP32 or CONAN_FP64");
    return CONAN_OK;
}

// Scoped device buffers and plan for one ic call.
template <typename T> struct ICWork {
    typedef typename Cplx<T>::type CT;
    Mesh m{};
    T *mesh = nullptr;
    CT *spec = nullptr, *spec2 = nullptr;
    double *xfer = nullptr, *part = nullptr;
    void *work = nullptr;
    FFTPair fft;
    cudaStream_t st = nullptr;
    ~ICWork() {
        if (!st) return;
        for (void *p : {(void *)mesh, (void *)spec, (void *)spec2, (void *)xfer, (void *)part, work}) pool_free(p, st);
        cudaStreamSynchronize(st);
        plan_return(m, sizeof(T) == 8, &fft);
        cudaStreamDestroy(st);
    }
    template <typename U> int alloc(U **p, size_t n) {
        void *q = nullptr;
        CONAN_CUDA(pool_alloc(&q, n * sizeof(U), st));
        *p = (U *)q;
        return CONAN_OK;
    }
    int setup(const conan_ic_params &p, bool need_spec2) {
        m = make_mesh(p.dim, 1 << p.mbits);
        CONAN_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        CONAN_TRY(alloc(&mesh, m.cells));
        CONAN_TRY(alloc(&spec, m.spec));
        if (need_spec2) CONAN_TRY(alloc(&spec2, m.spec));
        CONAN_TRY(alloc(&xfer, m.cells * (need_spec2 ? p.dim : 1)));
        CONAN_TRY(alloc(&part, ic_scratch(m)));
        CONAN_TRY(plan_take(m, sizeof(T) == 8, &fft));
        CONAN_TRY(alloc((char **)&work, fft.work_bytes ? fft.work_bytes : 16));
        CONAN_TRY(fft.bind(work, st));
        return CONAN_OK;
    }
    unsigned gc() const { return (unsigned)((m.cells + 255) / 256); }
    unsigned gs() const { return (unsigned)((m.spec + 255) / 256); }
    int upload(const double *h) {
        CONAN_TRY(copy_to_device(xfer, h, m.cells * sizeof(double), st));
        k_convert<double, T><<<gc(), 256, 0, st>>>(xfer, mesh, m.cells, 1.0, 0.0);
        CONAN_LAUNCHED();
        return CONAN_OK;
    }
    int download(double *h) {
        k_convert<T, double><<<gc(), 256, 0, st>>>(mesh, xfer, m.cells, 1.0, 0.0);
        CONAN_LAUNCHED();
        CONAN_TRY(copy_to_host(h, xfer, m.cells * sizeof(double), st));
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }
};

static ICFilter filter_of(const conan_ic_params &p, const Mesh &m) {
    ICFilter F{};
    F.mode = p.scale_free ? IC_SCALE_FREE : IC_CDM;
    F.ns = p.ns;
    F.L = p.size;
    F.Omega0 = p.Omega0;
    F.h = p.H0 / 100.0;
    F.t = p.scale * m.n / p.size;  // Fourier::scale<R>(sigma * N/L), ic.cc:63
    return F;
}

// The filter's tables in the scratch area (see ic_scratch), where the mesh uses them.
static int filter_tables(const ICFilter &F, const Mesh &m, double *part, cudaStream_t st, ICTable *tab) {
    *tab = ICTable{nullptr, nullptr};
    const size_t np = ic_table_values(m);
    if (!np) return CONAN_OK;
    double *p = part + IC_PART, *e = p + np;
    const unsigned h = (unsigned)m.n / 2 + 1, bs = h >= 256 ? 256 : h >= 128 ? 128 : h >= 64 ? 64 : 32;
    k_ic_table<<<dim3((h + bs - 1) / bs, h, h), bs, 0, st>>>(F, m, p, e);
    CONAN_LAUNCHED();
    *tab = ICTable{p, e};
    return CONAN_OK;
}

// Variance of the smoothed field of spectrum spec into the scratch scalars.
template <typename T>
static int field_variance(const conan_ic_params &p, const Mesh &m, const typename Cplx<T>::type *spec,
                          const ICFilter &F, const ICTable &tab, double *part, cudaStream_t st) {
    k_ic_var<T><<<IC_BLOCKS, 256, 0, st>>>(spec, m, F, tab, part);
    CONAN_LAUNCHED();
    k_ic_scalars<<<1, IC_BLOCKS, 0, st>>>(part, 0, p.sigma, (double)m.cells, part + IC_BLOCKS);
    CONAN_LAUNCHED();
    return CONAN_OK;
}

// Device pipeline of _generate_random_field<R>, src/ic/ic.cc:37-98, from the
// real mesh `noise` (an out-of-place R2C leaves its input alone) to the
// density in `mesh`. Nothing waits for the host.
template <typename T>
int grf_device(const conan_ic_params &p, const Mesh &m, T *noise, T *mesh, typename Cplx<T>::type *spec,
               FFTPair &fft, double *part, cudaStream_t st) {
    CONAN_TRY(fft.forward(noise, spec));
    const ICFilter F = filter_of(p, m);
    ICTable tab;
    CONAN_TRY(filter_tables(F, m, part, st, &tab));
    const unsigned gs = (unsigned)((m.spec + 1023) / 1024);  // four modes per thread
    const double nc = (double)m.cells;
    if (p.scale_free) {
        CONAN_TRY(field_variance<T>(p, m, spec, F, tab, part, st));
        k_ic_filter<T><<<gs, 256, 0, st>>>(spec, spec, m, F, tab, p.smooth != 0, 1, 1.0,
                                           part + IC_BLOCKS + IC_SCALE);
    } else {
        const double res = p.size / m.n;
        k_ic_filter<T><<<gs, 256, 0, st>>>(spec, spec, m, F, tab, false, 1, 1.0 / (nc * std::pow(res, 0.5 * m.R)),
                                           nullptr);
    }
    CONAN_LAUNCHED();
    CONAN_TRY(fft.inverse(spec, mesh));
    return CONAN_OK;
}
template int grf_device<float>(const conan_ic_params &, const Mesh &, float *, float *, cufftComplex *, FFTPair &,
                               double *, cudaStream_t);
template int grf_device<double>(const conan_ic_params &, const Mesh &, double *, double *, cufftDoubleComplex *,
                                FFTPair &, double *, cudaStream_t);

// _compute_potential<R>, src/ic/ic.cc:100-117, in place on a device mesh.
template <typename T>
int potential_device(const Mesh &m, double L, T *mesh, typename Cplx<T>::type *spec, FFTPair &fft,
                     cudaStream_t st) {
    CONAN_TRY(fft.forward(mesh, spec));
    double gsp = -std::pow(L / (2 * M_PI), 2) / (double)m.cells;
    k_ic_potential<T><<<(unsigned)((m.spec + 1023) / 1024), 256, 0, st>>>(spec, m, gsp);
    CONAN_LAUNCHED();
    CONAN_TRY(fft.inverse(spec, mesh));
    return CONAN_OK;
}
template int potential_device<float>(const Mesh &, double, float *, cufftComplex *, FFTPair &, cudaStream_t);
template int potential_device<double>(const Mesh &, double, double *, cufftDoubleComplex *, FFTPair &,
                                      cudaStream_t);

// Per-block sums of a . b (FP64, fixed order).
template <typename T>
__global__ void k_dot_partial(const T *__restrict__ a, const T *__restrict__ b, size_t n, double *__restrict__ part) {
    double s = 0;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        s += (double)a[i] * (double)b[i];
    s = block_sum<double>(s);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

// y += *alpha x
template <typename T>
__global__ void k_axpy(T *__restrict__ y, const T *__restrict__ x, size_t n, const double *__restrict__ alpha) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = (T)((double)y[i] + *alpha * (double)x[i]);
}

// Adjoint of the Gaussian random field of grf_device: given the noise w and
// dL/d(density) in dbar (overwritten), writes dL/dw into wbar. Scale-free:
// density = s y with y = L_F w, s = sigma / sqrt(var), var = |L_PS w|^2 / N,
// L_X = C2R diag(X) R2C / N (DC = 0), all symmetric, so
//   wbar = s L_F dbar - (s / var) (y . dbar) / N  L_PS L_PS w.
// CDM: density = A w with A symmetric, wbar = A dbar.
// Scratch: spec, spec2 (half spectra), tmp (mesh), part (ic_scratch doubles).
template <typename T>
int grf_adjoint_device(const conan_ic_params &p, const Mesh &m, const T *w, T *dbar, T *wbar,
                       typename Cplx<T>::type *spec, typename Cplx<T>::type *spec2, T *tmp, FFTPair &fft,
                       double *part, cudaStream_t st) {
    const ICFilter F = filter_of(p, m);
    ICTable tab;
    CONAN_TRY(filter_tables(F, m, part, st, &tab));
    const unsigned gs = (unsigned)((m.spec + 1023) / 1024), gc = (unsigned)((m.cells + 255) / 256);
    const double nc = (double)m.cells;
    if (!p.scale_free) {
        double scale = 1.0 / (nc * std::pow(p.size / m.n, 0.5 * m.R));
        CONAN_TRY(fft.forward(dbar, spec));
        k_ic_filter<T><<<gs, 256, 0, st>>>(spec, spec, m, F, tab, false, 1, scale, nullptr);
        CONAN_LAUNCHED();
        CONAN_TRY(fft.inverse(spec, wbar));
        return CONAN_OK;
    }
    const double *scal = part + IC_BLOCKS;
    CONAN_TRY(fft.forward(const_cast<T *>(w), spec));  // an out-of-place R2C leaves its input alone
    CONAN_TRY(field_variance<T>(p, m, spec, F, tab, part, st));
    // y = L_F w
    k_ic_filter<T><<<gs, 256, 0, st>>>(spec, spec2, m, F, tab, p.smooth != 0, 1, 1.0 / nc, nullptr);
    CONAN_LAUNCHED();
    CONAN_TRY(fft.inverse(spec2, tmp));
    k_dot_partial<T><<<IC_BLOCKS, 256, 0, st>>>(tmp, dbar, m.cells, part);
    CONAN_LAUNCHED();
    k_ic_scalars<<<1, IC_BLOCKS, 0, st>>>(part, 1, p.sigma, nc, part + IC_BLOCKS);
    CONAN_LAUNCHED();
    // q = L_PS L_PS w into tmp
    k_ic_filter<T><<<gs, 256, 0, st>>>(spec, spec2, m, F, tab, true, 2, 1.0 / nc, nullptr);
    CONAN_LAUNCHED();
    CONAN_TRY(fft.inverse(spec2, tmp));
    // wbar = s L_F dbar
    CONAN_TRY(fft.forward(dbar, spec));
    k_ic_filter<T><<<gs, 256, 0, st>>>(spec, spec, m, F, tab, p.smooth != 0, 1, 1.0 / nc, scal + IC_AMP);
    CONAN_LAUNCHED();
    CONAN_TRY(fft.inverse(spec, wbar));
    k_axpy<T><<<gc, 256, 0, st>>>(wbar, tmp, m.cells, scal + IC_DOT);
    CONAN_LAUNCHED();
    return CONAN_OK;
}
template int grf_adjoint_device<float>(const conan_ic_params &, const Mesh &, const float *, float *, float *,
                                       cufftComplex *, cufftComplex *, float *, FFTPair &, double *, cudaStream_t);
template int grf_adjoint_device<double>(const conan_ic_params &, const Mesh &, const double *, double *,
                                        double *, cufftDoubleComplex *, cufftDoubleComplex *, double *, FFTPair &,
                                        double *, cudaStream_t);

template <typename T> int noise_device(const Mesh &m, unsigned long long seed, T *mesh, cudaStream_t st) {
    size_t pairs = (m.cells + 1) / 2;
    k_noise_philox<T><<<(unsigned)((pairs + 255) / 256), 256, 0, st>>>(mesh, m.cells, seed);
    CONAN_LAUNCHED();
    return CONAN_OK;
}
template int noise_device<float>(const Mesh &, unsigned long long, float *, cudaStream_t);
template int noise_device<double>(const Mesh &, unsigned long long, double *, cudaStream_t);

template <typename T> int ic_generate(const conan_ic_params &p, const double *noise, double *out) {
    ICWork<T> w;
    CONAN_TRY(w.setup(p, false));
    if (noise)
        CONAN_TRY(w.upload(noise));
    else
        CONAN_TRY(noise_device<T>(w.m, p.seed, w.mesh, w.st));
    CONAN_TRY(grf_device<T>(p, w.m, w.mesh, w.mesh, w.spec, w.fft, w.part, w.st));
    return w.download(out);
}

template <typename T> int ic_potential(const conan_ic_params &p, double *inout) {
    ICWork<T> w;
    CONAN_TRY(w.setup(p, false));
    CONAN_TRY(w.upload(inout));
    CONAN_TRY(potential_device<T>(w.m, p.size, w.mesh, w.spec, w.fft, w.st));
    return w.download(inout);
}

template <typename T> int ic_displacement(const conan_ic_params &p, const double *pot, double *psi) {
    ICWork<T> w;
    CONAN_TRY(w.setup(p, true));
    CONAN_TRY(w.upload(pot));
    CONAN_TRY(w.fft.forward(w.mesh, w.spec));
    double scale = 1.0 / ((double)w.m.cells / p.size * w.m.n);  // real_part(size / L * N)
    for (int a = 0; a < p.dim; ++a) {
        k_ic_deriv<T><<<w.gs(), 256, 0, w.st>>>(w.spec, w.spec2, w.m, a, scale);
        CONAN_LAUNCHED();
        CONAN_TRY(w.fft.inverse(w.spec2, w.mesh));
        k_interleave<T><<<w.gc(), 256, 0, w.st>>>(w.mesh, w.xfer, w.m.cells, p.dim, a);
        CONAN_LAUNCHED();
    }
    CONAN_TRY(copy_to_host(psi, w.xfer, w.m.cells * p.dim * sizeof(double), w.st));
    CONAN_CUDA(cudaStreamSynchronize(w.st));
    return CONAN_OK;
}

}  // namespace conan

using namespace conan;

extern "C" {

int conan_ic_noise(const conan_ic_params *p, double *noise_out) {
    CONAN_TRY(check_ic_params(p));
    if (!noise_out) return set_error(CONAN_ERR_ARG, "null output");
    CONAN_TRY(device_guard(p->device));
    ICWork<double> w;
    CONAN_TRY(w.setup(*p, false));
    size_t pairs = (w.m.cells + 1) / 2;
    k_noise_philox_f64<<<(unsigned)((pairs + 255) / 256), 256, 0, w.st>>>(w.xfer, w.m.cells, p->seed);
    CONAN_LAUNCHED();
    CONAN_TRY(copy_to_host(noise_out, w.xfer, w.m.cells * sizeof(double), w.st));
    CONAN_CUDA(cudaStreamSynchronize(w.st));
    return CONAN_OK;
}

int conan_ic_generate(const conan_ic_params *p, const double *noise_or_null, double *density_out) {
    CONAN_TRY(check_ic_params(p));
    if (!density_out) return set_error(CONAN_ERR_ARG, "null output");
    CONAN_TRY(device_guard(p->device));
    return p->precision == CONAN_FP64 ? ic_generate<double>(*p, noise_or_null, density_out)
                                      : ic_generate<float>(*p, noise_or_null, density_out);
}

int conan_ic_potential(const conan_ic_params *p, double *inout) {
    CONAN_TRY(check_ic_params(p));
    if (!inout) return set_error(CONAN_ERR_ARG, "null buffer");
    CONAN_TRY(device_guard(p->device));
    return p->precision == CONAN_FP64 ? ic_potential<double>(*p, inout) : ic_potential<float>(*p, inout);
}

int conan_ic_displacement(const conan_ic_params *p, const double *potential, double *psi_out) {
    CONAN_TRY(check_ic_params(p));
    if (!potential || !psi_out) return set_error(CONAN_ERR_ARG, "null buffer");
    CONAN_TRY(device_guard(p->device));
    return p->precision == CONAN_FP64 ? ic_displacement<double>(*p, potential, psi_out)
                                      : ic_displacement<float>(*p, potential, psi_out);
}

}  // extern "C"
