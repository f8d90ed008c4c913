// pm.cu -- the particle-mesh solver handle (conan_pm_*), the B200
// replacement of the reference's Gravity<R> solver (src/run/nbody.hh:53-219)
// driven by LeapFrog::run (src/run/leapfrog.hh:33-46).
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "fft.cuh"
#include "fft_plane.cuh"
// The forward plane pass zeroes the accumulator behind its reads (1) or a
// memset does it afterwards (0); a compile-time tunable.
#ifndef PLANE_CLEAR
#define PLANE_CLEAR 1
#endif
#include "fft_line64.cuh"
#include "fft_z.cuh"
#include "hostio.cuh"
#include "ic.cuh"
#include "pm.cuh"

#include <type_traits>

namespace conan {

std::string &last_error() {
    static thread_local std::string s;
    return s;
}

int set_error(int code, const char *fmt, ...) {
    char buf[1024];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    last_error() = buf;
    return code;
}

int err_word_status(int h) {
    if (!h) return CONAN_OK;
    if (h & 8)
        return set_error(CONAN_ERR_TIMEOUT,
                         "a bounded wait for a bulk tensor copy into shared memory ran out (code %d)", h);
    return set_error(CONAN_ERR_STATE, "kernel self-check failed (code %d): corrupt cell offsets or payload", h);
}

double adot(double H0, double Om, double OL, double a) {
    // Cosmology::operator(), src/run/cosmology.hh:16-23.
    double Ok = 1 - Om - OL;
    return H0 * a * std::sqrt(OL + Om * std::pow(a, -3) + Ok * std::pow(a, -2));
}

int check_pm_params(const conan_pm_params *p) {
    if (!p) return set_error(CONAN_ERR_ARG, "null parameters");
    if (p->dim < 1 || p->dim > 3)
        return set_error(CONAN_ERR_UNSUPPORTED, "dim = %d: the GPU path supports 1, 2 and 3 dimensions",
                         p->dim);
    if (!is_pow2(p->n_mass) || p->n_mass < 2)
        return set_error(CONAN_ERR_ARG, "n_mass = %d must be a power of two >= 2", p->n_mass);
    if (!is_pow2(p->f)) return set_error(CONAN_ERR_ARG, "f = %d must be a power of two >= 1", p->f);
    long long nf = (long long)p->n_mass * p->f;
    long long cells = 1;
    for (int i = 0; i < p->dim; ++i) cells *= nf;
    if (cells >= (1LL << 32))
        return set_error(CONAN_ERR_ARG, "force mesh of %lld cells exceeds 2^32 - 1", cells);
    if (!(p->size > 0)) return set_error(CONAN_ERR_ARG, "box size must be positive");
    if (p->precision != CONAN_FP32 && p->precision != CONAN_FP64)
        return set_error(CONAN_ERR_ARG, "precision must be CONAN_FP32 or CONAN_FP64");
    if (p->gradient != CONAN_GRAD_FD4 && p->gradient != CONAN_GRAD_SPECTRAL)
        return set_error(CONAN_ERR_ARG, "gradient must be CONAN_GRAD_FD4 or CONAN_GRAD_SPECTRAL");
    if (!(p->H0 > 0)) return set_error(CONAN_ERR_ARG, "H0 must be positive");
    return CONAN_OK;
}

int device_guard(int dev) {
    int n = 0;
    cudaError_t e = cudaGetDeviceCount(&n);
    if (e != cudaSuccess || n == 0)
        return set_error(CONAN_ERR_CUDA, "no CUDA device available (%s)", cudaGetErrorString(e));
    if (dev < 0 || dev >= n) return set_error(CONAN_ERR_ARG, "device %d out of range (%d devices)", dev, n);
    CONAN_CUDA(cudaSetDevice(dev));
    return CONAN_OK;
}

// ------------------------------------------------------------------ PM --

// cudaGraphInstantiate, with the failure that conan_selftest_fail_graph asks for.
static thread_local int g_fail_graph = -1;
static cudaError_t graph_instantiate(cudaGraphExec_t *x, cudaGraph_t g) {
    if (g_fail_graph >= 0 && g_fail_graph-- == 0) return cudaErrorMemoryAllocation;
    return alloc_retry([&] { return cudaGraphInstantiate(x, g, 0); });
}

// exp(-2 pi i k / n), k < n (a multiple of 8), as pairs (re, im), each value the
// double nearest to the exact one: the angle is reduced to the first octant in
// integers and evaluated in long double. (cos and sin of the rounded double angle
// are off by up to 6.5e-16. The force's rms error against long double over that
// of the same 2D solve by library transforms, 64^2 to 512^2 cells: 0.96 to 0.97
// with this table, 1.03 to 1.08 with that one.)
void unit_roots(int n, double *w) {
    const int quarter = n / 4;
    for (int k = 0; k < n; ++k) {
        const int q = k / quarter, r = k % quarter;
        const bool upper = r > n / 8;
        const long double a = 2 * 3.14159265358979323846264338327950288L * (upper ? quarter - r : r) / n;
        const double ca = (double)std::cos(a), sa = (double)std::sin(a);
        const double c = upper ? sa : ca, s = upper ? ca : sa;
        // (c - i s) (-i)^q
        w[2 * k] = q == 0 ? c : q == 1 ? -s : q == 2 ? -c : s;
        w[2 * k + 1] = q == 0 ? -s : q == 1 ? -c : q == 2 ? s : c;
    }
}

template <typename T, int R> struct PM : PMBase {
    typedef typename Cplx<T>::type CT;
    typedef typename Pay<T>::elem PE;

    conan_pm_params prm{};
    Mesh mf{}, mm{};
    size_t np = 0;
    double res_f = 0, res_m = 0, mass = 1, G = 0;
    Parts<T> P{};
    T *mesh = nullptr;
    T *gm[3] = {nullptr, nullptr, nullptr};
    G4<T> *grad = nullptr;  // packed FD4 gradient mesh
    CT *spec = nullptr, *spec2 = nullptr;
    uint32_t *count = nullptr, *off = nullptr, *rank = nullptr, *bsum = nullptr;
    int *err = nullptr;  // device error word set by kernel self-checks
    PE *pay = nullptr;
    // Host transfers pass through two staging chunks of stage_n doubles each,
    // allocated at creation: no transfer allocates device memory, and the
    // chunks alternate on the handle's stream.
    double *stage[2] = {nullptr, nullptr};
    size_t stage_n = 0;
    static constexpr size_t STAGE_MAX = (size_t)1 << 24;  // doubles per chunk (128 MiB)
    void *work = nullptr;
    FFTPair fft;
    // FD4 meshes whose Poisson solve is the transforms of all axes but the last
    // (fft2) around a shared-memory pass along that one: FP32 3D of 64..1024 cells
    // per side (fft_z.cuh), FP64 2D of 64..1024 and 3D of 64..512 (fft_line64.cuh)
    FFTPair fft2;
    CT *ztw = nullptr;  // exp(-2 pi i k / n), k < n
    bool zpass = false;
    cudaStream_t st = nullptr;
    Profiler prof;
    std::vector<void *> allocs;
    double a_pos = 0, a_mom = 0;
    bool ranks_pending = false;
    int mesh_holds = 0;  // 0 nothing, 1 delta, 2 phi
    unsigned cb_every = 1;
    size_t bytes = 0;

    ~PM() override {
        if (st) cudaStreamSynchronize(st);
        for (auto &g : pieces) cudaGraphExecDestroy(g.exec);
        fft.destroy();
        fft2.destroy();
        for (void *p : allocs) cudaFree(p);
        if (st) cudaStreamDestroy(st);
    }

    template <typename U> int alloc(U **p, size_t n) {
        void *q = nullptr;
        size_t b = n * sizeof(U);
        if (b == 0) b = 16;
        const cudaError_t e = device_alloc(&q, b);
        if (e != cudaSuccess) {
            cudaGetLastError();
            return set_error(CONAN_ERR_ALLOC, "cudaMalloc of %zu bytes failed: %s", b, cudaGetErrorString(e));
        }
        allocs.push_back(q);
        bytes += b;
        *p = (U *)q;
        return CONAN_OK;
    }

    // `batch` equal boxes stored back to back (ensembles); 1 for conan_pm.
    int create(const conan_pm_params &p, int batch = 1) {
        prm = p;
        int nf = p.n_mass * p.f;
        mf = make_mesh(R, nf, batch);
        mm = make_mesh(R, p.n_mass, batch);
        np = mm.cells;
        res_f = p.size / nf;
        res_m = p.size / p.n_mass;
        mass = std::pow(double(nf) / p.n_mass, R);  // src/run/nbody.hh:85
        G = 3. / 2 * p.Omega_m * p.H0 * p.H0;       // src/run/cosmology.hh:13
        CONAN_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        P.np = np;
        P.mshift = mm.shift;
        P.f = p.f;
        P.bshift = R * mm.shift;
        for (int k = 0; k < R; ++k) {
            CONAN_TRY(alloc(&P.d[k], np));
            CONAN_TRY(alloc(&P.p[k], np));
        }
        CONAN_TRY(alloc(&mesh, mf.cells));
        CONAN_TRY(alloc(&spec, mf.spec));
        if (p.gradient == CONAN_GRAD_SPECTRAL) {
            CONAN_TRY(alloc(&spec2, mf.spec));
            for (int k = 0; k < R; ++k) CONAN_TRY(alloc(&gm[k], mf.cells));
        } else {
            CONAN_TRY(alloc(&grad, mf.cells));
        }
        CONAN_TRY(alloc(&count, mf.cells));
        CONAN_TRY(alloc(&off, mf.cells + 1));
        CONAN_TRY(alloc(&rank, np));
        size_t nb = (mf.cells + SCAN_CHUNK - 1) / SCAN_CHUNK;
        CONAN_TRY(alloc(&bsum, nb));
        CONAN_TRY(alloc(&pay, np * Pay<T>::words));
        stage_n = std::min(STAGE_MAX, std::max(np * (size_t)R, std::max(mf.cells, mm.cells)));
        CONAN_TRY(alloc(&stage[0], stage_n));
        CONAN_TRY(alloc(&stage[1], stage_n));
        CONAN_TRY(alloc(&err, 1));
        CONAN_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
        CONAN_CUDA(cudaMemsetAsync(count, 0, mf.cells * sizeof(uint32_t), st));
        dep_variant = dep_default();
        bool lag = sizeof(T) == 4 &&
                   ((lag_small<R>(np) && lag_set(LAG_SMALL, false)) || lag_try<0>() || lag_try<1>() || lag_try<2>());
        // On fine meshes (f >= 2) a window that fits shared memory only fits
        // a small tile and holds many cells per particle, each of which gets
        // about one corner: clearing and flushing it costs more than the
        // atomics it saves. Deposit directly from the largest tile then.
        if (sizeof(T) == 4 && (!lag || (double)lwin.cells > LAG_WINDOW_CELLS_PER_PARTICLE * lag_particles()))
            lag = lag_try<0>(true) || lag_try<1>(true) || lag_try<2>(true);
        if (lag) {
            CONAN_TRY(alloc(&lacc, mf.cells));
            CONAN_CUDA(cudaMemsetAsync(lacc, 0, mf.cells * sizeof(unsigned long long), st));
            dep_variant = DEP_LAG;
            CONAN_TRY(tma_setup());
            pers = LAG_PERSIST != 0;
            CONAN_TRY(pers_setup());
        }
        if (sizeof(T) == 8 && np <= DIRECT_MAX && mf.cells <= DIRECT_MAX) {
            CONAN_TRY(alloc(&dacc, mf.cells));
            CONAN_CUDA(cudaMemsetAsync(dacc, 0, mf.cells * sizeof(ulonglong2), st));
            dep_variant = DEP_DIRECT;
        }
        const bool split = sizeof(T) == 4 ? R == 3 && mf.n <= 1024 : (R == 3 && mf.n <= 512) || (R == 2 && mf.n <= 1024);
        zpass = split && p.gradient == CONAN_GRAD_FD4 && mf.n >= 64;
        if (!zpass || sizeof(T) == 4) CONAN_TRY(fft.create(mf, sizeof(T) == 8, batch));
        size_t wbytes = fft.work_bytes;
        if (zpass) {
            CONAN_TRY(fft2.create_planes(mf, sizeof(T) == 8, batch));
            CONAN_TRY(zpass_setup());
            wbytes = std::max(wbytes, fft2.work_bytes);
            if (lacc) CONAN_TRY(plane_setup());
        }
        // CONAN_GRAD_KERNEL: cell or zm picks the gradient-mesh kernel at
        // creation (before any autotuning)
        grad_zm = mf.cells > ((size_t)1 << 21);
        if (const char *gk = getenv("CONAN_GRAD_KERNEL")) grad_zm = !strcmp(gk, "zm");
        CONAN_TRY(alloc((char **)&work, wbytes));
        if (fft.r2c) CONAN_TRY(fft.bind(work, st));
        if (zpass) CONAN_TRY(fft2.bind(work, st));
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }

    // Half spectrum of the density in mesh by the full transforms, for the power
    // spectrum. FP64 handles that solve around the line pass make those
    // transforms' plans at the first one (creation with both pairs: 64^2 cells 1.6
    // ms against 1.0, 256^2 3.4 against 2.7, 64^3 6.8 against 6.0); their work
    // area is the gradient mesh (32 bytes per cell), which only lives from a solve
    // to its kick.
    int full_spectrum() {
        if (!fft.r2c) {
            CONAN_TRY(fft.create(mf, sizeof(T) == 8, mf.batch));
            void *w = grad;
            if (fft.work_bytes > mf.cells * sizeof(G4<T>)) CONAN_TRY(alloc((char **)&w, fft.work_bytes));
            CONAN_TRY(fft.bind(w, st));
        }
        CONAN_TIMED(prof, "fft_r2c", st, CONAN_TRY(fft.forward(mesh, spec)));
        mesh_holds = 1;
        return CONAN_OK;
    }

    // Particles per staging chunk (whole particles of R doubles).
    size_t stage_particles() const { return stage_n / (size_t)R; }

    // Absolute FP64 state of the n particles of view v into host X, Pm
    // (either may be null), chunk by chunk through the staging buffers;
    // returns after the last copy.
    int export_state(const Parts<T> &v, size_t n, double *X, double *Pm) {
        const size_t cp = stage_particles();
        for (size_t i0 = 0; i0 < n; i0 += cp) {
            const size_t cnt = std::min(cp, n - i0);
            CONAN_TIMED(prof, "export", st,
                        (k_export<T, R><<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(
                            v, res_f, i0, cnt, X ? stage[0] : nullptr, Pm ? stage[1] : nullptr)));
            if (X) CONAN_TRY(copy_to_host(X + i0 * R, stage[0], cnt * R * sizeof(double), st));
            if (Pm) CONAN_TRY(copy_to_host(Pm + i0 * R, stage[1], cnt * R * sizeof(double), st));
        }
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }

    // Converts n host doubles into the device array out (type T), chunk by
    // chunk through the staging buffers.
    int upload_mesh(const double *in, T *out, size_t n) {
        for (size_t c0 = 0, b = 0; c0 < n; c0 += stage_n, b ^= 1) {
            const size_t cnt = std::min(stage_n, n - c0);
            CONAN_TRY(copy_to_device(stage[b], in + c0, cnt * sizeof(double), st));
            CONAN_TIMED(prof, "convert", st,
                        (k_convert<double, T><<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(stage[b], out + c0, cnt,
                                                                                          1.0, 0.0)));
        }
        return CONAN_OK;
    }

    // Largest lattice and mesh whose FP64 deposit goes straight to the
    // accumulator by default: up to there the counting sort's five launches
    // cost more than the atomics (per FP64 step, 2D 256^2 31 -> 21 us, 1024^2
    // 108 -> 104, 3D 64^3 64 -> 52; 128^3 286 against 280 us, 307 against 316
    // where clustered, and 256^3 1.94 against 2.19 ms).
    static constexpr size_t DIRECT_MAX = (size_t)1 << 20;

    dim3 grid_p() const { return dim3((unsigned)((np + 255) / 256)); }

    // --- deposit ---------------------------------------------------------
    // 0 .. DEP_VARIANTS-1: sorted deposit with tile shape DepTile<R, V>;
    // DEP_LAG: Lagrangian-window deposit (FP32). Chosen by the autotuner.
    // DEP_DIRECT: corners straight into a two-word accumulator (FP64, small
    // lattices; reported as the sorted deposit, whose bits it has, and left for
    // good when the caller asks for that one by name).
    static constexpr int DEP_LAG = DEP_VARIANTS, DEP_DIRECT = DEP_LAG + 1;
    int dep_variant = 0;
    unsigned config = 0;  // changes of the kernels' choice: what was captured before is stale

    // Lagrangian deposit: accumulator mesh, lattice-tile variant and window.
    unsigned long long *lacc = nullptr;
    int lag_v = -1;  // LagTile<R, V> variant that fits this mesh, -1: none
    LagWin lwin{};
    size_t lag_smem = 0;

    ulonglong2 *dacc = nullptr;  // direct FP64 deposit
    bool direct_on() const { return sizeof(T) == 8 && dep_variant == DEP_DIRECT && dacc; }

    bool lag_on() const { return sizeof(T) == 4 && dep_variant == DEP_LAG && lag_v >= 0 && lacc; }

    // f(V) with lattice-tile variant v as a compile-time constant.
    template <typename F> static int lag_call(int v, F f) {
        if (v == 0) return f(std::integral_constant<int, 0>{});
        if (v == 1) return f(std::integral_constant<int, 1>{});
        if (v == 2) return f(std::integral_constant<int, 2>{});
        if constexpr (R > 1)
            if (v == LAG_SMALL) return f(std::integral_constant<int, LAG_SMALL>{});
        return set_error(CONAN_ERR_STATE, "no lattice tile %d", v);
    }

    template <int V> static constexpr double lag_tile_particles() {
        return (double)LagTile<R, V>::LX * LagTile<R, V>::LY * LagTile<R, V>::LZ;
    }
    double lag_particles() const {
        double n = 0;
        lag_call(lag_v, [&](auto v) {
            n = lag_tile_particles<decltype(v)::value>();
            return CONAN_OK;
        });
        return n;
    }

    // direct: a window of two cells per axis, so that (nearly) every corner
    // goes straight to the accumulator mesh with one integer atomic.
    template <int V> bool lag_try(bool direct = false) {
        typedef LagTile<R, V> L;
        const int n = mm.n;
        if (n < L::LX || (R >= 2 && n < L::LY) || (R == 3 && n < L::LZ)) return false;
        LagWin w{};
        w.w[0] = direct ? 2 : L::LX * prm.f + L::M;
        w.w[1] = R >= 2 ? (direct ? 2 : L::LY * prm.f + L::M) : 1;
        w.w[2] = R == 3 ? (direct ? 2 : L::LZ * prm.f + L::M) : 1;
        w.cells = (w.w[0] * w.w[1] * w.w[2] + 3) & ~3;
        size_t sh = (size_t)w.cells * LAG_PLANES * sizeof(uint32_t);
        if (sh > 112 * 1024) return false;
        if constexpr (sizeof(T) == 4) {  // set once here, outside any stream capture
            auto kern = k_deposit_lag<R, L::LX, L::LY, L::LZ, L::THREADS>;
            auto fused = k_gkd_lag<R, L::LX, L::LY, L::LZ, L::THREADS>;
            if (!raise_dyn_smem(kern, sh) || !raise_dyn_smem(fused, sh)) return false;
        }
        lwin = w;
        lag_smem = sh;
        lag_v = V;
        return true;
    }

    template <int V> int launch_lag() {
        if constexpr (sizeof(T) == 4) {
            typedef LagTile<R, V> L;
            size_t tiles = (size_t)(mm.n / L::LX) * (R >= 2 ? mm.n / L::LY : 1) * (R == 3 ? mm.n / L::LZ : 1) *
                           (size_t)mm.batch;
            auto kern = k_deposit_lag<R, L::LX, L::LY, L::LZ, L::THREADS>;
            CONAN_TIMED(prof, "deposit", st, (kern<<<(unsigned)tiles, L::THREADS, lag_smem, st>>>(P, mf, lwin, lacc)));
            return CONAN_OK;
        } else {
            return set_error(CONAN_ERR_UNSUPPORTED, "the Lagrangian deposit is FP32 only");
        }
    }

    // The fused gather/kick/drift + deposit of variant V (FP32, FD4).
    // TMA staging of the 3D tile's particle arrays (FP32, 32x8x8 tiles):
    // tensor maps over d[k], p[k] built once at creation.
    TileMaps tmaps{};
    bool tma_ok = false;
    size_t tma_smem = 0;

    int tma_setup() {
        tma_ok = false;
        if constexpr (sizeof(T) == 4 && R == 3) {
            const char *off = getenv("CONAN_NO_TMA");
            if (off && *off && *off != '0') return CONAN_OK;
            if (lag_v >= 0) return lag_call(lag_v, [&](auto v) { return tma_setup_v<decltype(v)::value>(); });
        }
        return CONAN_OK;
    }

    // Tensor maps over d[k], p[k] with the box of one particle group of
    // lattice tile V (LX x LY x THREADS / (LX LY)), and the staged kernel's
    // shared memory; tma_ok stays false when anything is missing (the
    // kernels then read global memory directly).
    template <int V> int tma_setup_v() {
        typedef LagTile<3, V> L;
        typedef CUresult (*Encode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn) {
            cudaGetLastError();
            return CONAN_OK;
        }
        const cuuint64_t n = (cuuint64_t)mm.n;
        const cuuint64_t dims[3] = {n, n, n * (cuuint64_t)mm.batch};
        const cuuint64_t strides[2] = {n * 4, n * n * 4};
        // one z-plane of the tile per copy
        const cuuint32_t box[3] = {L::LX, L::LY, 1}, estr[3] = {1, 1, 1};
        float *arr[6] = {P.d[0], P.d[1], P.d[2], P.p[0], P.p[1], P.p[2]};
        for (int a = 0; a < 6; ++a)
            if (((Encode)fn)(&tmaps.a[a], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, arr[a], dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                             CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return CONAN_OK;
        const size_t stage_bytes = (size_t)(6 * L::LX * L::LY * L::LZ * 4 + 128);
        // the window after the staged arrays, or over them
        tma_smem = LAG_STAGE_KEEP ? stage_bytes + lag_smem : std::max(lag_smem, stage_bytes);
        auto kern = k_gkd_lag_tma<3, L::LX, L::LY, L::LZ, L::THREADS>;
        if (!raise_dyn_smem(kern, tma_smem)) return CONAN_OK;
        tma_ok = true;
        return CONAN_OK;
    }

    // Persistent staged launch (3D, lattice tiles 32x8x8 and 16x8x8 with twice
    // the threads, two staging buffers): on when `pers` and its set-up
    // succeeded for the current tile variant.
    bool pers = false, pers_ok = false;
    unsigned pers_grid = 0;
    size_t pers_smem = 0;
    template <int V> struct PersT {
        typedef LagTile<3, V> L;
        static constexpr int THREADS = 2 * L::THREADS;
    };
    int pers_setup() {
        pers_ok = false;
        if constexpr (sizeof(T) == 4 && R == 3) {
            if (!pers || !tma_ok || lag_v > 1) return CONAN_OK;
            return lag_v == 0 ? pers_setup_v<0>() : pers_setup_v<1>();
        }
        return CONAN_OK;
    }
    template <int V> int pers_setup_v() {
        typedef LagTile<3, V> L;
        constexpr int TH = PersT<V>::THREADS;
        auto kern = k_gkd_lag_pers<3, L::LX, L::LY, L::LZ, TH>;
        pers_smem = 128 + 2 * 6 * (size_t)(L::LX * L::LY * L::LZ) * 4 + lag_smem;
        if (!raise_dyn_smem(kern, pers_smem)) return CONAN_OK;
        int nb = 0, sms = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kern, TH, pers_smem) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, prm.device) != cudaSuccess || nb < 1) {
            cudaGetLastError();
            return CONAN_OK;
        }
        pers_grid = (unsigned)(nb * sms);
        pers_ok = true;
        return CONAN_OK;
    }

    int launch_gkd_lag(const GKD &c, const char *name) {
        return lag_call(lag_v, [&](auto v) { return launch_gkd_lag_v<decltype(v)::value>(c, name); });
    }
    template <int V> int launch_gkd_lag_v(const GKD &c, const char *name) {
        if constexpr (sizeof(T) == 4) {
            typedef LagTile<R, V> L;
            size_t tiles = (size_t)(mm.n / L::LX) * (R >= 2 ? mm.n / L::LY : 1) * (R == 3 ? mm.n / L::LZ : 1) *
                           (size_t)mm.batch;
            if constexpr (R == 3 && V <= 1) {
                if (pers_ok && tma_ok && (LAG_TMA_GATHER || !c.kick)) {
                    constexpr int TH = PersT<V>::THREADS;
                    auto pk = k_gkd_lag_pers<3, L::LX, L::LY, L::LZ, TH>;
                    const unsigned grid = (unsigned)std::min<size_t>(pers_grid, tiles);
                    CONAN_TIMED(prof, name, st,
                                (pk<<<grid, TH, pers_smem, st>>>(P, mf, grad, c, lwin, lacc, tmaps, err,
                                                                  (unsigned)tiles)));
                    return CONAN_OK;
                }
            }
            if constexpr (R == 3) {
                // staged (512^3, 32x8x8 tiles): drift+deposit 1.87 against 2.33
                // ms; with the gather, keeping the drifted displacements in the
                // staged memory and a one-plane window 3.55 against 3.76 ms
                if (tma_ok && (LAG_TMA_GATHER || !c.kick)) {
                    auto tk = k_gkd_lag_tma<3, L::LX, L::LY, L::LZ, L::THREADS>;
                    const int rec = prof.begin(name, st);
                    tk<<<(unsigned)tiles, L::THREADS, tma_smem, st>>>(P, mf, grad, c, lwin, lacc, tmaps, err);
                    cudaError_t e = cudaGetLastError();
                    if (e != cudaSuccess)
                        return set_error(CONAN_ERR_CUDA,
                                         "staged launch failed: %s (tile %dx%dx%d, %d threads, %zu tiles, %zu bytes "
                                         "shared, window %d cells)",
                                         cudaGetErrorString(e), L::LX, L::LY, L::LZ, L::THREADS, tiles, tma_smem,
                                         lwin.cells);
                    prof.end(rec, st);
                    return CONAN_OK;
                }
            }
            auto kern = k_gkd_lag<R, L::LX, L::LY, L::LZ, L::THREADS>;
            CONAN_TIMED(prof, name, st,
                        (kern<<<(unsigned)tiles, L::THREADS, lag_smem, st>>>(P, mf, grad, c, lwin, lacc)));
            return CONAN_OK;
        } else {
            return set_error(CONAN_ERR_UNSUPPORTED, "the Lagrangian deposit is FP32 only");
        }
    }

    // lag_ready: the accumulator holds the deposit of the current positions,
    // made by the fused kernel and not yet turned into the density mesh.
    bool lag_ready = false;
    int drop_lag_deposit() {
        if (lag_ready) {
            if (direct_on()) CONAN_CUDA(cudaMemsetAsync(dacc, 0, mf.cells * sizeof(ulonglong2), st));
            else CONAN_CUDA(cudaMemsetAsync(lacc, 0, mf.cells * sizeof(unsigned long long), st));
        }
        lag_ready = false;
        return CONAN_OK;
    }

    // A call failed between its launches: the host does not know which of them
    // ran, so the ranks and accumulators may hold anything.
    bool stale = false;

    // Particle positions were replaced: ranks and a fused deposit are stale.
    int positions_reset() {
        if (stale) {
            CONAN_CUDA(cudaMemsetAsync(count, 0, mf.cells * sizeof(uint32_t), st));
            if (lacc) CONAN_CUDA(cudaMemsetAsync(lacc, 0, mf.cells * sizeof(unsigned long long), st));
            if (dacc) CONAN_CUDA(cudaMemsetAsync(dacc, 0, mf.cells * sizeof(ulonglong2), st));
            ranks_pending = lag_ready = stale = false;
            mesh_holds = 0;
            return CONAN_OK;
        }
        if (ranks_pending) CONAN_CUDA(cudaMemsetAsync(count, 0, mf.cells * sizeof(uint32_t), st));
        ranks_pending = false;
        return drop_lag_deposit();
    }

    // After such a call: what it may have left is cleared before it returns (its
    // message kept), since a graph that is replayed later asks no host flag.
    // Within a caller's capture the next call on the host does that.
    int failed(int rc) {
        const std::string msg = last_error();
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        stale = true;
        if (cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs == cudaStreamCaptureStatusNone &&
            positions_reset() == CONAN_OK)
            cudaStreamSynchronize(st);
        last_error() = msg;
        return rc;
    }

    // The Lagrangian deposit of the current positions into the accumulator
    // mesh (unless the fused gather kernel did it already).
    int lag_accumulate() {
        if (!lag_ready) {
            // The staged tiles (neither kick nor drift) where they have a full
            // window: 256^3 512 -> 411 us, 128^3 70 -> 63 for displacements of
            // three cells. The small tiles hide little behind one or two
            // particles per thread (64^3 staged 20.4 us, old tiles 16.5), and
            // with the two-cell window the momenta's loads are not worth the
            // wait (256^3 f = 2 1050 against 955 us, 64^3 f = 4 50 against 48).
            if (tma_ok && !pers_ok && lag_v != LAG_SMALL && lwin.w[0] > 2) {
                const GKD c{0, 0, 0, 0, 0, 0};
                CONAN_TRY(launch_gkd_lag(c, "deposit"));
            } else {
                CONAN_TRY(lag_call(lag_v, [&](auto v) { return launch_lag<decltype(v)::value>(); }));
            }
        }
        lag_ready = false;
        return CONAN_OK;
    }

    // The accumulator's density contrast into out.
    int acc_mesh(T *out) {
        size_t nt = (mf.cells + 3) / 4;  // four cells per thread
        CONAN_TIMED(prof, "deposit_mesh", st,
                    (k_acc_mesh<T><<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(lacc, out, mf.cells, mass)));
        return CONAN_OK;
    }

    int deposit_lag() {
        CONAN_TRY(lag_accumulate());
        CONAN_TRY(acc_mesh(mesh));
        CONAN_TIMED(prof, "deposit_clear", st,
                    CONAN_CUDA(cudaMemsetAsync(lacc, 0, mf.cells * sizeof(unsigned long long), st)));
        mesh_holds = 1;
        return CONAN_OK;
    }

    // CONAN_DEPOSIT_SORTED or CONAN_DEPOSIT_LAGRANGIAN.
    int set_deposit(int mode) override {
        CONAN_TRY(drop_lag_deposit());  // a pending fused deposit belongs to the old mode
        ++config;
        if (mode == CONAN_DEPOSIT_SORTED) {
            dep_variant = dep_default();
            return CONAN_OK;
        }
        if (mode == CONAN_DEPOSIT_LAGRANGIAN) {
            if (sizeof(T) != 4 || lag_v < 0 || !lacc)
                return set_error(CONAN_ERR_UNSUPPORTED,
                                 "the Lagrangian deposit needs FP32 and a lattice of at least one tile per axis");
            dep_variant = DEP_LAG;
            return CONAN_OK;
        }
        return set_error(CONAN_ERR_ARG, "unknown deposit mode %d", mode);
    }
    int get_deposit(int *mode) override {
        if (!mode) return set_error(CONAN_ERR_ARG, "null mode");
        *mode = lag_on() ? CONAN_DEPOSIT_LAGRANGIAN : CONAN_DEPOSIT_SORTED;
        return CONAN_OK;
    }

    // The sorted deposit's tile shape before any autotuning: the largest that
    // gives every SM a tile, else the small one.
    int dep_default() const {
        typedef DepTile<R, 0> D;
        const size_t tiles = mf.cells / ((size_t)D::TX * D::TY * D::TZ);
        return tiles < 148 && dep_fits<DEP_SMALL>() ? DEP_SMALL : 0;
    }

    // Tiled deposit with tile variant V; returns 1 when V does not fit the
    // mesh (the caller falls back), CONAN_OK or an error code.
    template <int V> int deposit_tiles(double scale) {
        typedef DepTile<R, V> D;
        if (mf.n < D::TX || mf.n < D::TY || mf.n < D::TZ) return 1;
        size_t tiles = (size_t)(mf.n / D::TX) * (R >= 2 ? mf.n / D::TY : 1) * (R == 3 ? mf.n / D::TZ : 1) *
                       (size_t)mf.batch;
        constexpr size_t sh = deposit_smem<T, R, V>();
        auto kern = k_deposit<T, R, D::TX, D::TY, D::TZ, D::THREADS>;
        if (sh > 48 * 1024)
            CONAN_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
        CONAN_TIMED(prof, "deposit", st,
                    (kern<<<(unsigned)tiles, D::THREADS, sh, st>>>(off, pay, mesh, mf, scale, (uint32_t)np, err)));
        return CONAN_OK;
    }

    int rank_pass() {
        if (ranks_pending) CONAN_CUDA(cudaMemsetAsync(count, 0, mf.cells * sizeof(uint32_t), st));
        CONAN_TIMED(prof, "rank", st, (k_rank<T, R><<<grid_p(), 256, 0, st>>>(P, mf, count, rank)));
        ranks_pending = true;
        return CONAN_OK;
    }

    int deposit() {
        if (lag_on()) return deposit_lag();
        if constexpr (sizeof(T) == 8) {
            if (direct_on()) {
                if (!lag_ready)
                    CONAN_TIMED(prof, "deposit", st, (k_deposit_direct<R><<<grid_p(), 256, 0, st>>>(P, mf, dacc)));
                lag_ready = false;
                CONAN_TIMED(prof, "deposit_mesh", st,
                            (k_direct_mesh<<<(unsigned)((mf.cells + 255) / 256), 256, 0, st>>>(dacc, mesh, mf.cells,
                                                                                                mass)));
                mesh_holds = 1;
                return CONAN_OK;
            }
        }
        if (!ranks_pending) CONAN_TRY(rank_pass());
        CONAN_TIMED(prof, "scan", st, scan_exclusive(count, mf.cells, bsum, off, st));
        ranks_pending = false;
        CONAN_TIMED(prof, "scatter", st,
                    (k_scatter<T, R><<<grid_p(), 256, 0, st>>>(P, mf, off, rank, pay, nullptr)));
        double scale = mass;
        int rc = 1;  // 1: the variant does not fit this mesh
        if (dep_variant == 1) rc = deposit_tiles<1>(scale);
        if (dep_variant == 2) rc = deposit_tiles<2>(scale);
        if (dep_variant == DEP_SMALL) rc = deposit_tiles<DEP_SMALL>(scale);
        if (rc == 1) rc = deposit_tiles<0>(scale);
        if (rc > 1) return rc;
        if (rc == 1) {
            CONAN_TIMED(prof, "deposit", st,
                        (k_deposit_pull<T, R><<<(unsigned)((mf.cells + 255) / 256), 256, 0, st>>>(
                            off, pay, mesh, mf, scale)));
        }
        mesh_holds = 1;
        return CONAN_OK;
    }

    // --- Poisson: mesh (delta) -> mesh (phi) [and gradient meshes] ------
    // Green's function multiply of the half spectrum s (one CTA per row).
    int green(CT *s, double gs) {
        const unsigned rows = (unsigned)(mf.spec / (size_t)mf.nh);
        const int threads = mf.nh >= 256 ? 256 : ((mf.nh + 31) / 32) * 32;
        CONAN_TIMED(prof, "green", st, (k_green<T><<<rows, threads, 0, st>>>(s, mf, (T)gs)));
        return CONAN_OK;
    }

    int zpass_setup() {
        std::vector<CT> w((size_t)mf.n);
        if constexpr (sizeof(T) == 8) {
            unit_roots(mf.n, reinterpret_cast<double *>(w.data()));
        } else {
            for (int k = 0; k < mf.n; ++k) {
                const double a = -2.0 * M_PI * (double)k / (double)mf.n;
                w[k].x = (T)std::cos(a);
                w[k].y = (T)std::sin(a);
            }
        }
        CONAN_TRY(alloc(&ztw, (size_t)mf.n));
        CONAN_CUDA(cudaMemcpy(ztw, w.data(), w.size() * sizeof(CT), cudaMemcpyHostToDevice));
        if constexpr (sizeof(T) == 4) {
            switch (mf.n) {
                case 64: return zpass_attr<64>();
                case 128: return zpass_attr<128>();
                case 256: return zpass_attr<256>();
                case 512: return zpass_attr<512>();
                default: return zpass_attr<1024>();
            }
        } else {
            return line_green(0.0, true);
        }
    }
    // The FP64 line pass of this mesh; attr: only set its shared-memory limit.
    int line_green(double gs, bool attr = false) {
        switch (mf.n) {
            case 64: return line_green_n<64>(gs, attr);
            case 128: return line_green_n<128>(gs, attr);
            case 256: return line_green_n<256>(gs, attr);
            case 512: return line_green_n<512>(gs, attr);
            default: return line_green_n<1024>(gs, attr);
        }
    }
    template <int N> int line_green_n(double gs, bool attr) {
        if constexpr (sizeof(T) == 8 && (R == 2 || (R == 3 && N <= 512))) {
            typedef LineT<N, R> L;
            auto k = k_line_green64<N, R>;
            if (attr) {
                if (!raise_dyn_smem(k, L::SMEM))
                    return set_error(CONAN_ERR_CUDA, "line pass: %zu bytes of shared memory refused", L::SMEM);
                return CONAN_OK;
            }
            const dim3 grid((unsigned)((mf.nh + L::TX - 1) / L::TX), R == 3 ? (unsigned)mf.n : 1u, (unsigned)mf.batch);
            CONAN_TIMED(prof, "green", st,
                        (k<<<grid, L::THREADS, L::SMEM, st>>>(reinterpret_cast<double2 *>(spec), mf, gs,
                                                              reinterpret_cast<const double2 *>(ztw))));
            return CONAN_OK;
        } else {
            return set_error(CONAN_ERR_UNSUPPORTED, "no line pass for this mesh");
        }
    }
    // z-pass lines per CTA: 0 the default width, else TX (the autotuner's knob)
    int ztx = 0;
    template <int N, int TX> int zpass_attr1() {
        if constexpr (ZTile<N, TX>::OK)
            if (!raise_dyn_smem(k_zpass_green<N, TX>, ZTile<N, TX>::SMEM))
                return set_error(CONAN_ERR_CUDA, "z pass: %zu bytes of shared memory refused", ZTile<N, TX>::SMEM);
        return CONAN_OK;
    }
    template <int N> int zpass_attr() {
        constexpr int T0 = ZTile<N>::TX;
        CONAN_TRY((zpass_attr1<N, 0>()));
        CONAN_TRY((zpass_attr1<N, T0 / 2>()));
        return zpass_attr1<N, 2 * T0>();
    }
    // widths of the z pass at this mesh size (default first)
    std::vector<int> zpass_widths() const {
        std::vector<int> w{0};
        auto add = [&](auto tag) {
            constexpr int N = decltype(tag)::value;
            constexpr int T0 = ZTile<N>::TX;
            if (ZTile<N, T0 / 2>::OK) w.push_back(T0 / 2);
            if (ZTile<N, 2 * T0>::OK) w.push_back(2 * T0);
        };
        switch (mf.n) {
            case 64: add(std::integral_constant<int, 64>()); break;
            case 128: add(std::integral_constant<int, 128>()); break;
            case 256: add(std::integral_constant<int, 256>()); break;
            case 512: add(std::integral_constant<int, 512>()); break;
            default: add(std::integral_constant<int, 1024>()); break;
        }
        return w;
    }
    template <int N, int TX> void zpass_launch1(float gs) {
        if constexpr (ZTile<N, TX>::OK) {
            typedef ZTile<N, TX> Z;
            const dim3 grid((unsigned)((mf.nh + Z::TX - 1) / Z::TX), (unsigned)mf.n, (unsigned)mf.batch);
            k_zpass_green<N, TX><<<grid, Z::THREADS, Z::SMEM, st>>>(reinterpret_cast<float2 *>(spec), mf, gs,
                                                                         reinterpret_cast<const float2 *>(ztw));
        }
    }
    template <int N> void zpass_launch(float gs) {
        constexpr int T0 = ZTile<N>::TX;
        if (ztx == T0 / 2 && ZTile<N, T0 / 2>::OK) zpass_launch1<N, T0 / 2>(gs);
        else if (ztx == 2 * T0 && ZTile<N, 2 * T0>::OK) zpass_launch1<N, 2 * T0>(gs);
        else zpass_launch1<N, 0>(gs);
    }
    // z FFT, Green multiply and inverse z FFT of the plane spectra (FP32)
    int green_z(double gs) {
        if constexpr (sizeof(T) == 4) {
            switch (mf.n) {
                case 64: CONAN_TIMED(prof, "green", st, zpass_launch<64>((float)gs)); break;
                case 128: CONAN_TIMED(prof, "green", st, zpass_launch<128>((float)gs)); break;
                case 256: CONAN_TIMED(prof, "green", st, zpass_launch<256>((float)gs)); break;
                case 512: CONAN_TIMED(prof, "green", st, zpass_launch<512>((float)gs)); break;
                default: CONAN_TIMED(prof, "green", st, zpass_launch<1024>((float)gs)); break;
            }
            return CONAN_OK;
        } else {
            return line_green(gs);
        }
    }

    // Plane transforms by thread-block clusters (fft_plane.cuh; FP32 3D,
    // n = 256 or 512, Lagrangian deposit): the forward pass reads the
    // accumulator mesh directly, so the step's density is never written.
    // plane_use: the autotuner's choice between them and cuFFT's planes.
    bool plane = false, plane_use = false;
    bool plane_inv = true;  // the inverse too (else cuFFT's 2D C2R after the z pass)
    bool plane_clear = PLANE_CLEAR;  // the forward pass clears the accumulator (else a memset)
    bool plane_on() const { return plane && plane_use && zpass && lag_on(); }
    int plane_kc = 16;       // kx columns per CTA of the plane pass
    unsigned plane_kcs = 0;  // the column counts that launch here (bit 0: 16, bit 1: 32)
    int plane_setup() {
        if constexpr (sizeof(T) == 4 && R == 3) {
            // CONAN_PLANE_PASS: 0 never, 1 both passes from the start, 2 the
            // forward pass from the start (else the default below, until the
            // autotuner decides)
            const char *pp = getenv("CONAN_PLANE_PASS");
            if (pp && *pp == '0') return CONAN_OK;
            // both column counts (clusters of 8 and of 16 CTAs at n = 512)
            // where they launch; the autotuner times both
            if (mf.n == 512) {
                CONAN_TRY((plane_setup_n<512, 32>()));
                CONAN_TRY((plane_setup_n<512, 16>()));
            }
            if (mf.n == 256) {
                CONAN_TRY((plane_setup_n<256, 32>()));
                CONAN_TRY((plane_setup_n<256, 16>()));
            }
            if (!plane) return CONAN_OK;
            // 32 columns per CTA: at 512^3 0.67 ms per forward pass against 0.69
            // with 16 (and 0.70 against 0.81 per inverse pass)
            if (plane_kcs & 2u) plane_kc = 32;
            const char *kc = getenv("CONAN_PLANE_COLUMNS");
            if (kc && atoi(kc) == 16 && (plane_kcs & 1u)) plane_kc = 16;
            if (kc && atoi(kc) == 32 && (plane_kcs & 2u)) plane_kc = 32;
            if (pp && (*pp == '1' || *pp == '2')) {
                plane_use = true;
                plane_inv = *pp == '1';  // 2: the forward pass only
            } else {
                // measured at 512^3: the forward pass here, cuFFT's inverse
                // (5.82 against 5.99 ms per step); elsewhere the autotuner decides
                plane_use = mf.n == 512;
                plane_inv = false;
            }
        }
        return CONAN_OK;
    }
    // On when both kernels launch in clusters of PlaneT::C CTAs on this GPU.
    template <int N, int KC> int plane_setup_n() {
        typedef PlaneT<N, KC> PT;
        if constexpr (PT::OK) {
            auto fk = k_plane_fwd<N, KC>;
            auto ik = k_plane_inv<N, KC>;
            if (!raise_dyn_smem(fk, PT::SMEM) || !raise_dyn_smem(ik, PT::SMEM)) return CONAN_OK;
            if (PT::C > 8 && (cudaFuncSetAttribute(fk, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
                              cudaFuncSetAttribute(ik, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)) {
                cudaGetLastError();
                return CONAN_OK;
            }
            cudaLaunchConfig_t cfg = plane_cfg<N, KC>();
            cudaLaunchAttribute at;
            plane_cluster(cfg, at);
            int nc = 0;
            if (cudaOccupancyMaxActiveClusters(&nc, fk, &cfg) != cudaSuccess || nc < 1 ||
                cudaOccupancyMaxActiveClusters(&nc, ik, &cfg) != cudaSuccess || nc < 1) {
                cudaGetLastError();
                return CONAN_OK;
            }
            plane = true;
            plane_kc = KC;
            plane_kcs |= KC == 16 ? 1u : 2u;
        }
        return CONAN_OK;
    }
    template <int N, int KC> cudaLaunchConfig_t plane_cfg() const {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3((unsigned)PlaneT<N, KC>::C, (unsigned)mf.n, (unsigned)mf.batch);
        cfg.blockDim = dim3((unsigned)PlaneT<N, KC>::THREADS);
        cfg.dynamicSmemBytes = PlaneT<N, KC>::SMEM;
        cfg.stream = st;
        return cfg;
    }
    static void plane_cluster(cudaLaunchConfig_t &cfg, cudaLaunchAttribute &at) {
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = cfg.gridDim.x;
        at.val.clusterDim.y = 1;
        at.val.clusterDim.z = 1;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
    }
    // 23 - log2(mass) when the particle mass is a power of two 2^e with
    // 0 <= e <= 23 (the mesh factor f is a power of two), else -1
    int plane_unit() const {
        int e = 0;
        const double fm = std::frexp(mass, &e);  // mass = fm 2^e, fm in [0.5, 1)
        if (fm != 0.5 || e - 1 < 0 || e - 1 > 23) return -1;
        return 23 - (e - 1);
    }
    template <int N, int KC> int plane_run(double gs) {
        if constexpr (sizeof(T) == 4 && PlaneT<N, KC>::OK) {
            cudaLaunchConfig_t cfg = plane_cfg<N, KC>();
            cudaLaunchAttribute at;
            plane_cluster(cfg, at);
            float2 *sp = reinterpret_cast<float2 *>(spec);
            CONAN_TIMED(prof, "plane_r2c", st,
                        CONAN_CUDA(cudaLaunchKernelEx(&cfg, k_plane_fwd<N, KC>, lacc, sp, mf, 0x1p-23 * mass,
                                                      (const float2 *)ztw, plane_clear ? 1 : 0, plane_unit())));
            if (!plane_clear)
                CONAN_TIMED(prof, "deposit_clear", st,
                            CONAN_CUDA(cudaMemsetAsync(lacc, 0, mf.cells * sizeof(unsigned long long), st)));
            CONAN_TRY(green_z(gs));
            if (plane_inv)
                CONAN_TIMED(prof, "plane_c2r", st,
                            CONAN_CUDA(cudaLaunchKernelEx(&cfg, k_plane_inv<N, KC>, (const float2 *)sp, (float *)mesh,
                                                          mf, (const float2 *)ztw)));
            else
                CONAN_TIMED(prof, "fft_c2r", st, CONAN_TRY(fft2.inverse(spec, mesh)));
            return CONAN_OK;
        } else {
            return set_error(CONAN_ERR_UNSUPPORTED, "no plane pass for this mesh");
        }
    }

    // The deposit of the current positions and the Poisson solve of the
    // kick that follows it: through the cluster plane pass when it is on
    // (which reads the accumulator itself), else deposit() (density mesh) and
    // poisson().
    int deposit_for_solve() { return plane_on() ? lag_accumulate() : deposit(); }
    int solve_deposited(double a) {
        if (!plane_on()) return poisson(a);
        const double gs = poisson_scale(a);
        if (mf.n == 512) CONAN_TRY((plane_kc == 16 ? plane_run<512, 16>(gs) : plane_run<512, 32>(gs)));
        else CONAN_TRY((plane_kc == 16 ? plane_run<256, 16>(gs) : plane_run<256, 32>(gs)));
        CONAN_TRY(fd_gradient(mesh, grad));
        mesh_holds = 2;
        return CONAN_OK;
    }
    // Between the two: the density contrast into out (device).
    int deposited_density(T *out) {
        if (plane_on()) return acc_mesh(out);
        CONAN_CUDA(cudaMemcpyAsync(out, mesh, mf.cells * sizeof(T), cudaMemcpyDeviceToDevice, st));
        return CONAN_OK;
    }
    int deposit_poisson(double a) {
        CONAN_TRY(deposit_for_solve());
        return solve_deposited(a);
    }

    // Green's function factor of a kick at a, with the per-member
    // normalisation 1 / (cells of one box).
    double poisson_scale(double a) const {
        return -G / (a * (double)((size_t)1 << mf.cshift)) * std::pow(prm.size / (2 * M_PI), 2);
    }

    int poisson(double a) {
        const double gs = poisson_scale(a);
        if (zpass) {
            // the planes' (rows') R2C, the last axis with the Green multiply,
            // the planes' C2R
            CONAN_TIMED(prof, "fft_r2c", st, CONAN_TRY(fft2.forward(mesh, spec)));
            CONAN_TRY(green_z(gs));
            CONAN_TIMED(prof, "fft_c2r", st, CONAN_TRY(fft2.inverse(spec, mesh)));
            CONAN_TRY(fd_gradient(mesh, grad));
            mesh_holds = 2;
            return CONAN_OK;
        }
        unsigned gb = (unsigned)((mf.spec + 255) / 256);
        CONAN_TIMED(prof, "fft_r2c", st, CONAN_TRY(fft.forward(mesh, spec)));
        CONAN_TRY(green(spec, gs));
        if (prm.gradient == CONAN_GRAD_SPECTRAL) {
            for (int k = 0; k < R; ++k) {
                CONAN_TIMED(prof, "spec_deriv", st, (k_spec_deriv<T><<<gb, 256, 0, st>>>(spec, spec2, mf, k)));
                CONAN_TIMED(prof, "fft_c2r", st, CONAN_TRY(fft.inverse(spec2, gm[k])));
            }
        }
        CONAN_TIMED(prof, "fft_c2r", st, CONAN_TRY(fft.inverse(spec, mesh)));
        if (prm.gradient == CONAN_GRAD_FD4) CONAN_TRY(fd_gradient(mesh, grad));
        mesh_holds = 2;
        return CONAN_OK;
    }

    // Packed FD4 gradient mesh of phi. Gradient-mesh kernel: columns marching
    // along z (3D, 32 cells per side and more) or one thread per cell in blocks
    // of grad_block threads. The default marches on meshes beyond 2^21 cells,
    // whose potential and gradient leave the L2 (256^3 86 -> 70 us; 128^3 10 us
    // either way, 64^3 2.6 against 3.4 us with a quarter of the threads); the
    // autotuner times both.
    bool grad_zm = false;
    int grad_block = 256;
    bool grad_zm_fits() const { return R == 3 && mf.n >= 32; }

    int fd_gradient(const T *phi, G4<T> *g) {
        if constexpr (R == 3) {
            if (grad_zm && grad_zm_fits()) {
                const unsigned blocks = (unsigned)(mf.cells / (256 * FDZ_PLANES));
                CONAN_TIMED(prof, "fd_grad", st, (k_fd_grad_zm<T><<<blocks, 256, 0, st>>>(phi, g, mf)));
                return CONAN_OK;
            }
        }
        const unsigned bs = (unsigned)grad_block;
        CONAN_TIMED(prof, "fd_grad", st,
                    (k_fd_grad<T, R><<<(unsigned)((mf.cells + bs - 1) / bs), bs, 0, st>>>(phi, g, mf)));
        return CONAN_OK;
    }

    // --- autotuner -----------------------------------------------------------
    // On the current particle state (a clustered one: tile costs grow as the
    // particles cluster) it chooses (1) the deposit: the sorted tile variants,
    // the Lagrangian window tiles V0..V2 and the direct two-cell window
    // (FP32); (2) the gradient-mesh kernel: one thread per cell in blocks of
    // 128, 256 or 512, or z-marching columns. Knobs are tuned one after the
    // other; each candidate runs one untimed and TUNE_STEPS timed leapfrog
    // steps (CUDA events) from a copy of the state, which is restored at the
    // end.
    struct TuneRec {
        std::string knob, value;
        double ms;  // per timed step
        bool chosen;
    };
    std::vector<TuneRec> tuned;
    static constexpr int TUNE_STEPS = 2;
    struct DepCand {
        int mode;  // 0 sorted (v = DEP_DIRECT: direct FP64), 1 Lagrangian window, 2 Lagrangian direct, 3 Lagrangian window, persistent
        int v;
        std::string name;
    };

    template <int V> bool dep_fits() const {
        typedef DepTile<R, V> D;
        return mf.n >= D::TX && mf.n >= D::TY && mf.n >= D::TZ;
    }
    bool lag_set(int v, bool direct) {
        bool ok = false;
        lag_call(v, [&](auto w) {
            ok = lag_try<decltype(w)::value>(direct);
            return CONAN_OK;
        });
        return ok;
    }
    int dep_apply(const DepCand &c) {
        CONAN_TRY(drop_lag_deposit());
        pers = c.mode == 3;
        if (c.mode == 0) {
            dep_variant = c.v;
            return CONAN_OK;
        }
        if (!lag_set(c.v, c.mode == 2)) return set_error(CONAN_ERR_STATE, "deposit candidate %s no longer fits", c.name.c_str());
        dep_variant = DEP_LAG;
        CONAN_TRY(tma_setup());
        return pers_setup();
    }

    // Time of one timed leapfrog step from the saved state.
    int tune_time(T *const *save, double a, double da, double *ms) {
        for (int k = 0; k < R; ++k) {
            CONAN_CUDA(cudaMemcpyAsync(P.d[k], save[k], np * sizeof(T), cudaMemcpyDeviceToDevice, st));
            CONAN_CUDA(cudaMemcpyAsync(P.p[k], save[R + k], np * sizeof(T), cudaMemcpyDeviceToDevice, st));
        }
        CONAN_TRY(positions_reset());
        double aa = a;
        CONAN_TRY(steps(aa, da, 0, 1));
        cudaEvent_t e0 = nullptr, e1 = nullptr;
        CONAN_CUDA(cudaEventCreate(&e0));
        CONAN_CUDA(cudaEventCreate(&e1));
        cudaEventRecord(e0, st);
        int rc = steps(aa, da, 1, 1 + TUNE_STEPS);
        cudaEventRecord(e1, st);
        cudaError_t se = cudaEventSynchronize(e1);
        float t = 0;
        if (se == cudaSuccess) se = cudaEventElapsedTime(&t, e0, e1);
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        if (rc != CONAN_OK) return rc;
        if (se != cudaSuccess) return set_error(CONAN_ERR_CUDA, "autotuner timing: %s", cudaGetErrorString(se));
        *ms = t / TUNE_STEPS;
        return check_err();
    }

    int tune(double a, double da) {
        tuned.clear();
        const double apos = a_pos, amom = a_mom;
        std::vector<T *> save(2 * R, nullptr);
        for (auto &b : save) {
            const cudaError_t e = device_alloc(&b, np * sizeof(T));
            if (e == cudaSuccess) continue;
            cudaGetLastError();
            for (auto c : save) cudaFree(c);
            return set_error(CONAN_ERR_ALLOC, "no memory for the autotuner's copy of the state: %s",
                             cudaGetErrorString(e));
        }
        for (int k = 0; k < R; ++k) {
            CONAN_CUDA(cudaMemcpyAsync(save[k], P.d[k], np * sizeof(T), cudaMemcpyDeviceToDevice, st));
            CONAN_CUDA(cudaMemcpyAsync(save[R + k], P.p[k], np * sizeof(T), cudaMemcpyDeviceToDevice, st));
        }
        const bool prof_was = prof.on;
        prof.on = false;
        int rc = tune_knobs(save.data(), a, da);
        ++config;
        prof.on = prof_was;
        for (int k = 0; k < R && rc == CONAN_OK; ++k) {
            cudaMemcpyAsync(P.d[k], save[k], np * sizeof(T), cudaMemcpyDeviceToDevice, st);
            cudaMemcpyAsync(P.p[k], save[R + k], np * sizeof(T), cudaMemcpyDeviceToDevice, st);
        }
        cudaStreamSynchronize(st);
        for (auto b : save) cudaFree(b);
        if (rc != CONAN_OK) return rc;
        CONAN_TRY(positions_reset());
        mesh_holds = 0;
        a_pos = apos;
        a_mom = amom;
        return CONAN_OK;
    }

    int tune_knobs(T *const *save, double a, double da) {
        // (1) the deposit
        std::vector<DepCand> cands;
        if (dep_fits<0>()) cands.push_back({0, 0, "sorted 32x8x8 / 256 threads"});
        if (dep_fits<1>()) cands.push_back({0, 1, "sorted 32x4x8 / 128 threads"});
        if (dep_fits<2>()) cands.push_back({0, 2, "sorted 32x16x8 / 512 threads"});
        // (where the large tiles fill the chip the small ones only cost tuning
        // time: 128^3 FP32 13.4 against 12.4 ms)
        if (dep_default() == DEP_SMALL) cands.push_back({0, DEP_SMALL, "sorted, tiles of 256 cells / 256 threads"});
        if (dacc) cands.push_back({0, DEP_DIRECT, "direct, two words per cell"});
        if (sizeof(T) == 4 && lacc) {
            const char *tile[4] = {"", "", "", ""};
            if (R == 3) tile[0] = "32x8x8", tile[1] = "16x8x8", tile[2] = "8x8x8", tile[3] = "16x8x4";
            if (R == 2) tile[0] = "64x32", tile[1] = "32x16", tile[2] = "16x16", tile[3] = "16x16 / 256 threads";
            if (R == 1) tile[0] = "2048", tile[1] = "512", tile[2] = "128";
            for (int v = 0; v < (lag_small<R>(np) ? LAG_SMALL + 1 : LAG_SMALL); ++v)
                if (lag_set(v, false)) cands.push_back({1, v, std::string("lagrangian window, tile ") + tile[v]});
            if (R == 3)
                for (int v = 0; v < 2; ++v)
                    if (lag_set(v, false))
                        cands.push_back({3, v, std::string("lagrangian window, tile ") + tile[v] + ", persistent"});
            for (int v = 0; v < 3; ++v)
                if (lag_set(v, true)) {
                    cands.push_back({2, v, std::string("lagrangian direct, tile ") + tile[v]});
                    break;
                }
        }
        int best = -1;
        double bms = 1e30;
        for (size_t i = 0; i < cands.size(); ++i) {
            double ms = 0;
            CONAN_TRY(dep_apply(cands[i]));
            CONAN_TRY(tune_time(save, a, da, &ms));
            tuned.push_back({"deposit", cands[i].name, ms, false});
            if (ms < bms) bms = ms, best = (int)i;
        }
        if (best >= 0) {
            CONAN_TRY(dep_apply(cands[best]));
            tuned[tuned.size() - cands.size() + best].chosen = true;
        }
        // (2) the gradient mesh (FD4 only)
        if (prm.gradient == CONAN_GRAD_FD4) {
            struct GC { bool zm; int block; std::string name; };
            std::vector<GC> g = {{false, 128, "thread per cell, 128"}, {false, 256, "thread per cell, 256"},
                                 {false, 512, "thread per cell, 512"}};
            if (grad_zm_fits()) g.push_back({true, 256, "z-marching columns"});
            best = -1;
            bms = 1e30;
            for (size_t i = 0; i < g.size(); ++i) {
                grad_zm = g[i].zm;
                grad_block = g[i].block;
                double ms = 0;
                CONAN_TRY(tune_time(save, a, da, &ms));
                tuned.push_back({"gradient", g[i].name, ms, false});
                if (ms < bms) bms = ms, best = (int)i;
            }
            grad_zm = g[best].zm;
            grad_block = g[best].block;
            tuned[tuned.size() - g.size() + best].chosen = true;
        }
        // (3) the z pass's lines per CTA (FP32 3D plane-transform solve)
        if (zpass && sizeof(T) == 4) {
            const std::vector<int> w = zpass_widths();
            best = -1;
            bms = 1e30;
            for (size_t i = 0; i < w.size(); ++i) {
                ztx = w[i];
                double ms = 0;
                CONAN_TRY(tune_time(save, a, da, &ms));
                char nm[64];
                if (w[i]) snprintf(nm, sizeof nm, "%d lines per CTA", w[i]);
                else snprintf(nm, sizeof nm, "default lines per CTA");
                tuned.push_back({"z pass", nm, ms, false});
                if (ms < bms) bms = ms, best = (int)i;
            }
            ztx = w[best];
            tuned[tuned.size() - w.size() + best].chosen = true;
        }
        // (4) the x and y transforms of the planes: thread-block clusters or
        // cuFFT's 2D plans
        if (plane && lag_on()) {
            struct PC { bool use, inv; int kc; std::string name; };
            std::vector<PC> pc = {{false, true, plane_kc, "cuFFT 2D plans"}};
            for (int kc : {16, 32})
                if (plane_kcs & (kc == 16 ? 1u : 2u)) {
                    const std::string cl = "thread-block clusters of " + std::to_string(mf.n / (2 * kc)) + " CTAs, " +
                                           std::to_string(kc) + " columns each";
                    pc.push_back({true, true, kc, cl});
                    pc.push_back({true, false, kc, cl + " (forward; cuFFT inverse)"});
                }
            best = -1;
            bms = 1e30;
            for (size_t i = 0; i < pc.size(); ++i) {
                plane_use = pc[i].use;
                plane_inv = pc[i].inv;
                plane_kc = pc[i].kc;
                double ms = 0;
                CONAN_TRY(tune_time(save, a, da, &ms));
                tuned.push_back({"plane transforms", pc[i].name, ms, false});
                if (ms < bms) bms = ms, best = (int)i;
            }
            plane_use = pc[best].use;
            plane_inv = pc[best].inv;
            plane_kc = pc[best].kc;
            tuned[tuned.size() - pc.size() + best].chosen = true;
        }
        return CONAN_OK;
    }

    std::string tune_report() const {
        std::string s = "[";
        for (size_t i = 0; i < tuned.size(); ++i) {
            char buf[256];
            snprintf(buf, sizeof buf, "%s{\"knob\": \"%s\", \"value\": \"%s\", \"ms_per_step\": %.4f, \"chosen\": %s}",
                     i ? ", " : "", tuned[i].knob.c_str(), tuned[i].value.c_str(), tuned[i].ms,
                     tuned[i].chosen ? "true" : "false");
            s += buf;
        }
        return s + "]";
    }

    int autotune(double a, double da, char *report, size_t len) override {
        CONAN_TRY(tune(a, da));
        if (report && len) {
            std::string r = tune_report();
            std::strncpy(report, r.c_str(), len - 1);
            report[len - 1] = 0;
            if (r.size() >= len) return set_error(CONAN_ERR_ARG, "report buffer too small (%zu bytes needed)", r.size() + 1);
        }
        return CONAN_OK;
    }

    // Kick and/or drift of every particle. rank_after: prepare the next
    // deposit (counting-sort ranks, or with the Lagrangian deposit and a
    // drift, the deposit itself in the same kernel).
    int gkd(bool kick, double ck, bool drift, double cd, bool rank_after) {
        const bool fuse = rank_after && drift && lag_on() && prm.gradient == CONAN_GRAD_FD4;
        const bool direct = rank_after && drift && direct_on();
        rank_after = rank_after && !lag_on() && !direct_on();  // these deposits need no ranks
        // ranks of positions about to move are stale either way
        if ((rank_after || drift) && ranks_pending) {
            CONAN_CUDA(cudaMemsetAsync(count, 0, mf.cells * sizeof(uint32_t), st));
            ranks_pending = false;
        }
        if (drift) CONAN_TRY(drop_lag_deposit());
        GKD c{ck, cd, kick ? 1 : 0, drift ? 1 : 0, rank_after ? 1 : 0, prm.periodic_gather ? 1 : 0};
        const char *name = kick ? (drift ? "gather_kick_drift" : "gather_kick") : "drift";
        if (fuse) {
            CONAN_TRY(launch_gkd_lag(c, kick ? "gather_kick_drift_deposit" : "drift_deposit"));
            lag_ready = true;
            return CONAN_OK;
        }
        // the last kick of a run (no drift, no deposit) on the same staged
        // tiles instead of the thread-per-particle kernel
        if (kick && !drift && !rank_after && lag_on() && prm.gradient == CONAN_GRAD_FD4) {
            c.deposit = 0;
            return launch_gkd_lag(c, name);
        }
        ulonglong2 *const da = direct ? dacc : nullptr;
        if (prm.gradient == CONAN_GRAD_SPECTRAL)
            CONAN_TIMED(prof, name, st,
                        (k_gkd<T, R, true><<<grid_p(), 256, 0, st>>>(P, mf, mesh, gm[0], gm[1], gm[2], grad, c,
                                                                     count, rank, da)));
        else
            CONAN_TIMED(prof, name, st,
                        (k_gkd<T, R, false><<<grid_p(), 256, 0, st>>>(P, mf, mesh, gm[0], gm[1], gm[2], grad, c,
                                                                      count, rank, da)));
        if (rank_after) ranks_pending = true;
        if (direct) lag_ready = true;
        return CONAN_OK;
    }

    double coef_drift(double a, double da) const {
        return da / (a * a * adot(prm.H0, prm.Omega_m, prm.Omega_L, a));
    }
    double coef_kick(double a, double da) const {
        return (da / adot(prm.H0, prm.Omega_m, prm.Omega_L, a)) / (res_f * res_f);
    }

    // --- API ---------------------------------------------------------------
    int init(const double *phi, double apos, double amom) override {
        if (!phi) return set_error(CONAN_ERR_ARG, "null potential");
        CONAN_TRY(upload_mesh(phi, mesh, mm.cells));
        double cdz = -apos / (res_m * res_f), cpz = -amom / (res_m * res_f);
        CONAN_TIMED(prof, "zeldovich", st, (k_zeldovich<T, R><<<grid_p(), 256, 0, st>>>(P, mesh, mm, cdz, cpz)));
        CONAN_TRY(positions_reset());
        mesh_holds = 0;
        a_pos = apos;
        a_mom = amom;
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }

    int drift(double a, double da) override {
        CONAN_TRY(gkd(false, 0, true, coef_drift(a, da), true));
        a_pos = a;
        return CONAN_OK;
    }

    int kick(double a, double da) override {
        CONAN_TRY(deposit_poisson(a));
        CONAN_TRY(gkd(true, coef_kick(a, da), false, 0, false));
        a_mom = a;
        return CONAN_OK;
    }

    // Steps [i0, i1) of a leapfrog run starting at a(i0) = a; the first drift
    // (left out unless `first`) is separate, every later drift is fused into
    // the previous kick, the last one too unless `last`.
    int steps(double &a, double da, unsigned i0, unsigned i1, bool first = true, bool last = true) {
        if (first) {
            CONAN_TRY(gkd(false, 0, true, coef_drift(a, da), true));
            a_pos = a;
        }
        for (unsigned i = i0; i < i1; ++i) {
            double am = a + da / 2;
            CONAN_TRY(deposit_poisson(am));
            const bool end = last && i + 1 == i1;
            double an = a + da;
            CONAN_TRY(gkd(true, coef_kick(am, da), !end, end ? 0 : coef_drift(an, da), !end));
            a_mom = am;
            a = an;
            if (!end) a_pos = a;
        }
        return CONAN_OK;
    }

    // A run segment is captured and launched as graphs of a few steps each, so
    // that the GPU works on one while the host captures the next (capturing
    // 100 steps of eleven launches first took the GPU's idle millisecond of a
    // 4.1 ms run). The instantiated graphs are kept by their shape (a piece of
    // the same shape holds the same launches with other scale-factor
    // coefficients, which an update in place exchanges; launches under way
    // keep theirs).
    static constexpr unsigned PIECE = 4;
    struct Piece {
        unsigned n;
        bool first, last;
        cudaGraphExec_t exec;
    };
    std::vector<Piece> pieces;

    int graph_piece(double &a, double da, unsigned i0, unsigned i1, bool first, bool last) {
        cudaGraph_t g = nullptr;
        CONAN_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
        int rc = steps(a, da, i0, i1, first, last);
        cudaError_t ce = cudaStreamEndCapture(st, &g);
        if (rc != CONAN_OK) {
            if (g) cudaGraphDestroy(g);
            return rc;
        }
        if (ce != cudaSuccess) return set_error(CONAN_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
        Piece *p = nullptr;
        for (auto &q : pieces)
            if (q.n == i1 - i0 && q.first == first && q.last == last) p = &q;
        cudaError_t ie = cudaSuccess;
        if (p) {
            cudaGraphExecUpdateResultInfo info{};
            if (cudaGraphExecUpdate(p->exec, g, &info) != cudaSuccess) {  // other launches: instantiate anew
                cudaGetLastError();
                cudaGraphExec_t fresh = nullptr;
                ie = graph_instantiate(&fresh, g);
                if (ie == cudaSuccess) {
                    cudaGraphExecDestroy(p->exec);
                    p->exec = fresh;
                }
            }
        } else {
            if (pieces.size() >= 8) {  // bounded: the oldest shape goes
                cudaGraphExecDestroy(pieces.front().exec);
                pieces.erase(pieces.begin());
            }
            cudaGraphExec_t fresh = nullptr;
            ie = graph_instantiate(&fresh, g);
            if (ie == cudaSuccess) {
                pieces.push_back({i1 - i0, first, last, fresh});
                p = &pieces.back();
            }
        }
        cudaGraphDestroy(g);
        if (ie != cudaSuccess) return set_error(CONAN_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ie));
        cudaError_t le = cudaGraphLaunch(p->exec, st);
        if (le != cudaSuccess) return set_error(CONAN_ERR_CUDA, "graph launch failed: %s", cudaGetErrorString(le));
        return CONAN_OK;
    }

    // Steps [i0, i1) as graphs; returns after they have run. A piece that fails
    // leaves the state and its scale factors as the pieces before it left them.
    int graph_segment(double &a, double da, unsigned i0, unsigned i1) {
        int rc = CONAN_OK;
        for (unsigned i = i0; i < i1 && rc == CONAN_OK;) {
            unsigned e = std::min(i1, i + PIECE);
            if (i1 - e < PIECE / 2) e = i1;  // no short last piece
            const double ap = a_pos, am = a_mom;
            rc = graph_piece(a, da, i, e, i == i0, e == i1);
            if (rc != CONAN_OK) {
                a_pos = ap;
                a_mom = am;
            }
            i = e;
        }
        cudaError_t se = cudaStreamSynchronize(st);
        if (rc != CONAN_OK) return rc;
        if (se != cudaSuccess) return set_error(CONAN_ERR_CUDA, "graph execution failed: %s", cudaGetErrorString(se));
        return CONAN_OK;
    }

    int run(conan_pm *h, const double *phi, double a0, double da, unsigned n, conan_step_cb cb,
            void *user) override {
        if (phi) CONAN_TRY(init(phi, a0, a0 + da / 2));
        double a = a0;
        unsigned i = 0;
        while (i < n) {
            unsigned seg_end = n;
            if (cb) {
                unsigned k = cb_every ? cb_every : 1;
                seg_end = ((i / k) + 1) * k;
                if (seg_end > n) seg_end = n;
            }
            const int rc = !prof.on && !debug_sync() ? graph_segment(a, da, i, seg_end) : steps(a, da, i, seg_end);
            if (rc != CONAN_OK) return failed(rc);
            i = seg_end;
            if (cb) {
                CONAN_CUDA(cudaStreamSynchronize(st));
                if (cb(h, i - 1, a, user) != 0)
                    return set_error(CONAN_ERR_STATE, "step callback stopped the run after step %u", i - 1);
            }
        }
        CONAN_CUDA(cudaStreamSynchronize(st));
        return check_err();
    }

    // Reads and clears the kernels' self-check word.
    int check_err() {
        int h = 0;
        CONAN_CUDA(cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st));
        CONAN_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
        CONAN_CUDA(cudaStreamSynchronize(st));
        return err_word_status(h);
    }

    int get_state(double *X, double *Pm) override {
        CONAN_TRY(export_state(P, np, X, Pm));
        return check_err();
    }

    int set_state(const double *X, const double *Pm, double apos, double amom) override {
        if (!X || !Pm) return set_error(CONAN_ERR_ARG, "null state");
        const size_t cp = stage_particles();
        for (size_t i0 = 0; i0 < np; i0 += cp) {
            const size_t cnt = std::min(cp, np - i0);
            CONAN_TRY(copy_to_device(stage[0], X + i0 * R, cnt * R * sizeof(double), st));
            CONAN_TRY(copy_to_device(stage[1], Pm + i0 * R, cnt * R * sizeof(double), st));
            CONAN_TIMED(prof, "import", st,
                        (k_import<T, R><<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(P, res_f, i0, cnt, stage[0],
                                                                                       stage[1])));
        }
        CONAN_TRY(positions_reset());
        a_pos = apos;
        a_mom = amom;
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }

    int mesh_out(double *out) {
        for (size_t c0 = 0, b = 0; c0 < mf.cells; c0 += stage_n, b ^= 1) {
            const size_t cnt = std::min(stage_n, mf.cells - c0);
            CONAN_TIMED(prof, "convert", st,
                        (k_convert<T, double><<<(unsigned)((cnt + 255) / 256), 256, 0, st>>>(mesh + c0, stage[b], cnt,
                                                                                          1.0, 0.0)));
            CONAN_TRY(copy_to_host(out + c0, stage[b], cnt * sizeof(double), st));
        }
        CONAN_CUDA(cudaStreamSynchronize(st));
        return check_err();
    }

    int density(double *out) override {
        CONAN_TRY(deposit());
        return mesh_out(out);
    }

    int potential(double *out) override {
        if (mesh_holds != 2) return set_error(CONAN_ERR_STATE, "no potential: call kick first");
        return mesh_out(out);
    }

    int power_spectrum(int nbins, double *k, double *Pk, double *cnt) override {
        if (nbins < 1) return set_error(CONAN_ERR_ARG, "nbins must be positive");
        CONAN_TRY(deposit());
        CONAN_TRY(full_spectrum());
        CONAN_TRY(spectrum_bins<T>(spec, mf, prm.size, nbins, k, Pk, cnt, st, this));
        return check_err();
    }

    int scale_factors(double *ap, double *am) override {
        if (ap) *ap = a_pos;
        if (am) *am = a_mom;
        return CONAN_OK;
    }
    int set_profiling(int on) override {
        prof.on = on != 0;
        return CONAN_OK;
    }
    int profile_entry(int i, char *name, int *launches, double *ms) override {
        CONAN_CUDA(cudaStreamSynchronize(st));
        CONAN_TRY(prof.collect());
        if (i < 0 || i >= (int)prof.names.size()) return set_error(CONAN_ERR_ARG, "no profile entry %d", i);
        if (name) {
            std::strncpy(name, prof.names[i].c_str(), 63);
            name[63] = 0;
        }
        if (launches) *launches = prof.launches[i];
        if (ms) *ms = prof.total_ms[i];
        return CONAN_OK;
    }
    int profile_reset() override {
        CONAN_CUDA(cudaStreamSynchronize(st));
        CONAN_TRY(prof.collect());
        prof.reset();
        return CONAN_OK;
    }
    int device_bytes(size_t *b) override {
        *b = bytes + fft.work_bytes * 0;
        return CONAN_OK;
    }
    int sync() override {
        CONAN_CUDA(cudaStreamSynchronize(st));
        return check_err();
    }
    int set_cb_every(unsigned k) override {
        cb_every = k ? k : 1;
        return CONAN_OK;
    }
    int device() const override { return prm.device; }
    void *stream() const override { return (void *)st; }
};

// Power-spectrum bins from a half spectrum (deterministic two-level sum).
__global__ void k_pk_final(const double *__restrict__ part, int nblocks, int nbins, double L, int R,
                           double ncells, double *__restrict__ out) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= 3 * nbins) return;
    double s = 0;
    for (int b = 0; b < nblocks; ++b) s += part[(size_t)b * 3 * nbins + j];
    out[j] = s;
}

template <typename T>
int spectrum_bins(const typename Cplx<T>::type *spec, const Mesh &m, double L, int nbins, double *k,
                  double *Pk, double *cnt, cudaStream_t st, PMBase *) {
    const int threads = 256, nblocks = 148 * 2;
    size_t sh = (size_t)(threads / 32) * 3 * nbins * sizeof(double);
    if (sh > 200 * 1024) return set_error(CONAN_ERR_ARG, "too many bins (%d)", nbins);
    double *part = nullptr, *out = nullptr;
    CONAN_CUDA(alloc_retry(
        [&] { return cudaMallocAsync((void **)&part, (size_t)nblocks * 3 * nbins * sizeof(double), st); }));
    CONAN_CUDA(alloc_retry([&] { return cudaMallocAsync((void **)&out, 3 * (size_t)nbins * sizeof(double), st); }));
    if (sh > 48 * 1024)
        CONAN_CUDA(cudaFuncSetAttribute(k_pk_partial<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sh));
    k_pk_partial<T><<<nblocks, threads, sh, st>>>(spec, m, nbins, part);
    CONAN_LAUNCHED();
    k_pk_final<<<(3 * nbins + 255) / 256, 256, 0, st>>>(part, nblocks, nbins, L, m.R, (double)m.cells, out);
    CONAN_LAUNCHED();
    std::vector<double> h(3 * (size_t)nbins);
    CONAN_CUDA(cudaMemcpyAsync(h.data(), out, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
    CONAN_CUDA(cudaFreeAsync(part, st));
    CONAN_CUDA(cudaFreeAsync(out, st));
    CONAN_CUDA(cudaStreamSynchronize(st));
    double norm = std::pow(L, m.R) / ((double)m.cells * (double)m.cells);
    for (int b = 0; b < nbins; ++b) {
        double c = h[2 * nbins + b];
        if (cnt) cnt[b] = c;
        if (k) k[b] = c > 0 ? h[nbins + b] / c * 2 * M_PI / L : 0;
        if (Pk) Pk[b] = c > 0 ? h[b] / c * norm : 0;
    }
    return CONAN_OK;
}

template int spectrum_bins<float>(const cufftComplex *, const Mesh &, double, int, double *, double *,
                                  double *, cudaStream_t, PMBase *);
template int spectrum_bins<double>(const cufftDoubleComplex *, const Mesh &, double, int, double *,
                                   double *, double *, cudaStream_t, PMBase *);

}  // namespace conan

#include "adjoint_impl.cuh"
#include "ensemble_impl.cuh"

namespace conan {

PMBase *make_pm(const conan_pm_params &p) {
    PMBase *b = nullptr;
    int rc = CONAN_OK;
#define MAKE(T, R)                     \
    {                                  \
        auto *x = new PM<T, R>();      \
        rc = x->create(p);             \
        b = x;                         \
    }
    if (p.precision == CONAN_FP32) {
        if (p.dim == 1) MAKE(float, 1) else if (p.dim == 2) MAKE(float, 2) else MAKE(float, 3)
    } else {
        if (p.dim == 1) MAKE(double, 1) else if (p.dim == 2) MAKE(double, 2) else MAKE(double, 3)
    }
#undef MAKE
    if (rc != CONAN_OK) {
        std::string msg = last_error();
        delete b;
        last_error() = msg;
        return nullptr;
    }
    return b;
}

}  // namespace conan

using namespace conan;

namespace conan {

// One CTA waits on a shared-memory barrier that nothing completes, with the
// bounded wait of the staged kernels; the wait must run out (bit 3).
__global__ void k_wait_selftest(int *err, unsigned polls) {
    __shared__ __align__(8) unsigned long long bar;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar)));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (threadIdx.x == 0 && !tma_wait(&bar, polls)) atomicOr(err, 8);
}

}  // namespace conan

struct conan_pm {
    PMBase *impl;
};

#define H_GUARD(h)                                                       \
    do {                                                                 \
        if (!(h) || !(h)->impl) return set_error(CONAN_ERR_ARG, "null handle"); \
        CONAN_TRY(device_guard((h)->impl->device()));                    \
    } while (0)

extern "C" {

const char *conan_last_error(void) { return last_error().c_str(); }
const char *conan_version(void) { return "conan_b200 1.0 (sm_100a)"; }

int conan_device_count(int *n) {
    if (!n) return set_error(CONAN_ERR_ARG, "null pointer");
    int c = 0;
    if (cudaGetDeviceCount(&c) != cudaSuccess) {
        cudaGetLastError();
        c = 0;
    }
    *n = c;
    return CONAN_OK;
}

int conan_selftest_fail_graph(int n) {
    g_fail_graph = n;
    return CONAN_OK;
}

int conan_selftest_bounded_wait(unsigned polls, void *stream) {
    int dev = 0;
    CONAN_CUDA(cudaGetDevice(&dev));
    CONAN_TRY(device_guard(dev));
    cudaStream_t st = (cudaStream_t)stream;
    int *err = nullptr, h = 0;
    CONAN_CUDA(cudaMalloc(&err, sizeof(int)));
    cudaError_t e = cudaMemsetAsync(err, 0, sizeof(int), st);
    if (e == cudaSuccess) {
        k_wait_selftest<<<1, 32, 0, st>>>(err, polls);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(err);
    if (e != cudaSuccess) return set_error(CONAN_ERR_CUDA, "bounded-wait self-test: %s", cudaGetErrorString(e));
    return err_word_status(h);
}

conan_pm *conan_pm_create(const conan_pm_params *p) {
    last_error().clear();
    if (check_pm_params(p) != CONAN_OK) return nullptr;
    if (device_guard(p->device) != CONAN_OK) return nullptr;
    PMBase *b = make_pm(*p);
    if (!b) return nullptr;
    return new conan_pm{b};
}

void conan_pm_destroy(conan_pm *h) {
    if (!h) return;
    if (h->impl) {
        cudaSetDevice(h->impl->device());
        delete h->impl;
    }
    delete h;
}

int conan_pm_init(conan_pm *h, const double *phi, double a_pos, double a_mom) {
    H_GUARD(h);
    return h->impl->init(phi, a_pos, a_mom);
}
int conan_pm_drift(conan_pm *h, double a, double da) {
    H_GUARD(h);
    return h->impl->drift(a, da);
}
int conan_pm_kick(conan_pm *h, double a, double da) {
    H_GUARD(h);
    return h->impl->kick(a, da);
}
int conan_pm_set_callback_interval(conan_pm *h, unsigned k) {
    H_GUARD(h);
    return h->impl->set_cb_every(k);
}
int conan_pm_set_deposit(conan_pm *h, int mode) {
    H_GUARD(h);
    return h->impl->set_deposit(mode);
}
int conan_pm_get_deposit(conan_pm *h, int *mode) {
    H_GUARD(h);
    return h->impl->get_deposit(mode);
}
int conan_pm_run(conan_pm *h, const double *phi, double a0, double da, unsigned n, conan_step_cb cb,
                 void *user) {
    H_GUARD(h);
    return h->impl->run(h, phi, a0, da, n, cb, user);
}
int conan_pm_get_state(conan_pm *h, double *X, double *P) {
    H_GUARD(h);
    return h->impl->get_state(X, P);
}
int conan_pm_set_state(conan_pm *h, const double *X, const double *P, double a_pos, double a_mom) {
    H_GUARD(h);
    return h->impl->set_state(X, P, a_pos, a_mom);
}
int conan_pm_scale_factors(conan_pm *h, double *a_pos, double *a_mom) {
    H_GUARD(h);
    return h->impl->scale_factors(a_pos, a_mom);
}
int conan_pm_density(conan_pm *h, double *delta_out) {
    H_GUARD(h);
    if (!delta_out) return set_error(CONAN_ERR_ARG, "null output");
    return h->impl->density(delta_out);
}
int conan_pm_potential(conan_pm *h, double *phi_out) {
    H_GUARD(h);
    if (!phi_out) return set_error(CONAN_ERR_ARG, "null output");
    return h->impl->potential(phi_out);
}
int conan_pm_power_spectrum(conan_pm *h, int nbins, double *k, double *P, double *count) {
    H_GUARD(h);
    return h->impl->power_spectrum(nbins, k, P, count);
}
int conan_pm_set_profiling(conan_pm *h, int enable) {
    H_GUARD(h);
    return h->impl->set_profiling(enable);
}
int conan_pm_profile_entry(conan_pm *h, int i, char *name, int *launches, double *total_ms) {
    H_GUARD(h);
    return h->impl->profile_entry(i, name, launches, total_ms);
}
int conan_pm_profile_reset(conan_pm *h) {
    H_GUARD(h);
    return h->impl->profile_reset();
}
int conan_pm_device_bytes(conan_pm *h, size_t *bytes) {
    H_GUARD(h);
    if (!bytes) return set_error(CONAN_ERR_ARG, "null pointer");
    return h->impl->device_bytes(bytes);
}
int conan_pm_sync(conan_pm *h) {
    H_GUARD(h);
    return h->impl->sync();
}
int conan_pm_autotune(conan_pm *h, double a, double da, char *report, size_t len) {
    H_GUARD(h);
    if (!(da > 0) || !(a > 0)) return set_error(CONAN_ERR_ARG, "need a > 0 and da > 0");
    return h->impl->autotune(a, da, report, len);
}
int conan_pm_get_stream(conan_pm *h, void **stream) {
    H_GUARD(h);
    if (!stream) return set_error(CONAN_ERR_ARG, "null pointer");
    *stream = h->impl->stream();
    return CONAN_OK;
}

}  // extern "C"

struct conan_diff {
    DiffBase *impl;
};

extern "C" {

conan_diff *conan_diff_create(const conan_diff_params *p) {
    last_error().clear();
    if (!p) {
        set_error(CONAN_ERR_ARG, "null parameters");
        return nullptr;
    }
    if (check_pm_params(&p->pm) != CONAN_OK || check_ic_params(&p->ic) != CONAN_OK) return nullptr;
    if (p->ic.dim != p->pm.dim || (1 << p->ic.mbits) != p->pm.n_mass) {
        set_error(CONAN_ERR_ARG, "ic and pm parameters disagree on dim / particles per side");
        return nullptr;
    }
    if (p->pm.gradient != CONAN_GRAD_FD4) {
        set_error(CONAN_ERR_UNSUPPORTED, "the adjoint supports the FD4 gradient only");
        return nullptr;
    }
    if (p->n < 1 || !(p->da > 0) || !(p->a0 > 0)) {
        set_error(CONAN_ERR_ARG, "need n >= 1, a0 > 0, da > 0");
        return nullptr;
    }
    if (device_guard(p->pm.device) != CONAN_OK) return nullptr;
    DiffBase *b = make_diff(*p);
    if (!b) return nullptr;
    return new conan_diff{b};
}

void conan_diff_destroy(conan_diff *h) {
    if (!h) return;
    if (h->impl) {
        cudaSetDevice(h->impl->device());
        delete h->impl;
    }
    delete h;
}

int conan_diff_forward(conan_diff *h, const void *noise_dev, void *density_out_dev, void *stream) {
    if (!h || !h->impl) return set_error(CONAN_ERR_ARG, "null handle");
    if (!noise_dev || !density_out_dev) return set_error(CONAN_ERR_ARG, "null buffer");
    CONAN_TRY(device_guard(h->impl->device()));
    return h->impl->forward(noise_dev, density_out_dev, stream);
}

int conan_diff_backward(conan_diff *h, const void *grad_density_dev, void *grad_noise_dev, void *stream) {
    if (!h || !h->impl) return set_error(CONAN_ERR_ARG, "null handle");
    if (!grad_density_dev || !grad_noise_dev) return set_error(CONAN_ERR_ARG, "null buffer");
    CONAN_TRY(device_guard(h->impl->device()));
    return h->impl->backward(grad_density_dev, grad_noise_dev, stream);
}

}  // extern "C"

struct conan_ens {
    EnsBase *impl;
};

#define ENS_GUARD(h)                                                              \
    do {                                                                          \
        if (!(h) || !(h)->impl) return set_error(CONAN_ERR_ARG, "null handle");   \
        CONAN_TRY(device_guard((h)->impl->device()));                             \
    } while (0)

extern "C" {

conan_ens *conan_ens_create(const conan_ens_params *p, int n_members, const conan_ens_member *m) {
    last_error().clear();
    if (!p || !m || n_members < 1) {
        set_error(CONAN_ERR_ARG, "need parameters and at least one member");
        return nullptr;
    }
    if (p->dim != 2 && p->dim != 3) {
        set_error(CONAN_ERR_UNSUPPORTED, "ensembles run in 2 or 3 dimensions");
        return nullptr;
    }
    if (p->n < 1 || !(p->a0 > 0) || !(p->da > 0) || !(p->H0 > 0) ||
        (p->precision != CONAN_FP32 && p->precision != CONAN_FP64)) {
        set_error(CONAN_ERR_ARG, "bad run parameters (n >= 1, a0, da, H0 > 0, precision)");
        return nullptr;
    }
    for (int i = 0; i < n_members; ++i)
        if (m[i].mbits < 3 || m[i].mbits > (p->dim == 3 ? 10 : 14) || !(m[i].size > 0)) {
            set_error(CONAN_ERR_ARG, "member %d: mbits %d / size %g out of range", i, m[i].mbits, m[i].size);
            return nullptr;
        }
    if (device_guard(p->device) != CONAN_OK) return nullptr;
    EnsBase *b = make_ens(*p, n_members, m);
    if (!b) return nullptr;
    return new conan_ens{b};
}

void conan_ens_destroy(conan_ens *h) {
    if (!h) return;
    if (h->impl) {
        cudaSetDevice(h->impl->device());
        delete h->impl;
    }
    delete h;
}

int conan_ens_init(conan_ens *h) {
    ENS_GUARD(h);
    return h->impl->init();
}
int conan_ens_run(conan_ens *h) {
    ENS_GUARD(h);
    return h->impl->run();
}
int conan_ens_forward_adjoint(conan_ens *h, double *loss_out) {
    ENS_GUARD(h);
    return h->impl->forward_adjoint(loss_out);
}
int conan_ens_power_spectrum(conan_ens *h, int member, int nbins, double *k, double *P, double *count) {
    ENS_GUARD(h);
    if (nbins < 1) return set_error(CONAN_ERR_ARG, "nbins must be positive");
    return h->impl->power_spectrum(member, nbins, k, P, count);
}
int conan_ens_state(conan_ens *h, int member, double *X, double *P) {
    ENS_GUARD(h);
    return h->impl->state(member, X, P);
}
int conan_ens_member_fields(conan_ens *h, int member, double *noise, double *target, double *gnoise) {
    ENS_GUARD(h);
    return h->impl->member_fields(member, noise, target, gnoise);
}
int conan_ens_last_ms(conan_ens *h, double *run_ms, double *adjoint_ms) {
    ENS_GUARD(h);
    return h->impl->last_ms(run_ms, adjoint_ms);
}
int conan_ens_total_particles(conan_ens *h, size_t *n) {
    ENS_GUARD(h);
    if (!n) return set_error(CONAN_ERR_ARG, "null pointer");
    *n = h->impl->total_particles();
    return CONAN_OK;
}
int conan_ens_describe(conan_ens *h, char *buf, size_t len) {
    ENS_GUARD(h);
    if (!buf || len == 0) return set_error(CONAN_ERR_ARG, "null buffer");
    std::string s = h->impl->describe();
    std::strncpy(buf, s.c_str(), len - 1);
    buf[len - 1] = 0;
    return s.size() < len ? CONAN_OK : set_error(CONAN_ERR_ARG, "buffer too small (%zu bytes needed)", s.size() + 1);
}

}  // extern "C"
