// fft_line64.cuh -- the last direction of the FP64 Poisson solve's transform in
// shared memory with the Green's function multiply in between, as fft_z.cuh does
// in FP32: forward complex FFT along y (2D meshes) or z (3D), multiply by gs /
// |k|^2 (DC = 0, the multiply of k_green), inverse FFT, so that the half
// spectrum crosses memory once between the transforms of the other axes and
// one launch takes the place of three or more.
//
// Stockham stages (see fft_z.cuh) with one radix-8 butterfly per thread and
// stage; the radix-2 or radix-4 stage of sizes that are no power of 8 comes
// first in the forward and last in the inverse transform. Every twiddle is read
// from the table of exp(-2 pi i k / n) (no recurrence in FP64). Lines are
// padded by one value in eight, so that the first stage's stride-8 writes
// spread over the banks.
#pragma once

#include "common.cuh"

namespace conan {

__device__ inline double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ inline double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ inline double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
// times -i (forward) or +i (inverse)
template <bool INV> __device__ inline double2 cmul_mi(double2 a) {
    return INV ? make_double2(-a.y, a.x) : make_double2(a.y, -a.x);
}

// In-register DFT of RAD = 2, 4 or 8 values, natural order in and out.
template <int RAD, bool INV> __device__ inline void dft_small(double2 *v) {
    if constexpr (RAD == 2) {
        const double2 a = v[0], b = v[1];
        v[0] = cadd(a, b);
        v[1] = csub(a, b);
    } else if constexpr (RAD == 4) {
        const double2 a0 = cadd(v[0], v[2]), a2 = csub(v[0], v[2]);
        const double2 a1 = cadd(v[1], v[3]), a3 = cmul_mi<INV>(csub(v[1], v[3]));
        v[0] = cadd(a0, a1);
        v[2] = csub(a0, a1);
        v[1] = cadd(a2, a3);
        v[3] = csub(a2, a3);
    } else {
        // two radix-4 transforms of the even and the odd values, then one
        // radix-2 level with W8^r = exp(-+ i pi r / 4)
        const double h = 0.70710678118654752440;
        double2 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
        dft_small<4, INV>(e);
        dft_small<4, INV>(o);
        o[1] = cmul(o[1], make_double2(h, INV ? h : -h));
        o[2] = cmul_mi<INV>(o[2]);
        o[3] = cmul(o[3], make_double2(-h, INV ? h : -h));
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            v[r] = cadd(e[r], o[r]);
            v[r + 4] = csub(e[r], o[r]);
        }
    }
}

// Lines per CTA: 3D meshes take 64 bytes or more of a row per access; 2D
// meshes have few lines (n/2 + 1), so two per CTA spread them over the SMs.
template <int N, int R> struct LineT {
    static constexpr int LT = N / 8;  // threads per line
    static constexpr int TX = R == 2 ? (N == 64 ? 4 : 2) : N >= 256 ? 4 : 1024 / N;
    static constexpr int THREADS = TX * LT;
    static constexpr int LINE = N + N / 8;
    static constexpr size_t SMEM = ((size_t)TX * LINE + N) * sizeof(double2);
    static constexpr int REST = N == 64 || N == 512 ? 1 : N == 256 ? 4 : 2;  // 64 .. 1024 points
};

// One stage of radix RAD, sub-length Ns: value e of line l is buf[pad(e) * TX
// + l], or g[e * zs + l] in memory (lines from `valid` on are zero and not
// written).
template <int N, int R, int RAD, bool INV, bool IN_G, bool OUT_G>
__device__ inline void line_stage(double2 *buf, double2 *g, size_t zs, int valid, int Ns, const double2 *tw) {
    typedef LineT<N, R> L;
    constexpr int NB = N / RAD, Q = NB / L::LT;
    const int l = (int)threadIdx.x % L::TX, j0 = (int)threadIdx.x / L::TX;
    auto at = [&](int e) -> double2 & { return buf[(e + (e >> 3)) * L::TX + l]; };
    double2 v[Q][RAD];
#pragma unroll
    for (int q = 0; q < Q; ++q)
#pragma unroll
        for (int r = 0; r < RAD; ++r) {
            const int e = j0 + q * L::LT + r * NB;
            if constexpr (IN_G) v[q][r] = l < valid ? g[(size_t)e * zs + l] : make_double2(0.0, 0.0);
            else v[q][r] = at(e);
        }
    if constexpr (!IN_G) __syncthreads();  // every input read before any output lands in place
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int j = j0 + q * L::LT, k = j % Ns, step = N / (Ns * RAD);
        if (Ns > 1) {  // the first stage's twiddles are all exactly 1
#pragma unroll
            for (int r = 1; r < RAD; ++r) {
                double2 w = tw[(k * step * r) & (N - 1)];
                if (INV) w.y = -w.y;
                v[q][r] = cmul(v[q][r], w);
            }
        }
        dft_small<RAD, INV>(v[q]);
        const int base = (j / Ns) * Ns * RAD + k;
#pragma unroll
        for (int r = 0; r < RAD; ++r) {
            const int e = base + r * Ns;
            if constexpr (OUT_G) {
                if (l < valid) g[(size_t)e * zs + l] = v[q][r];
            } else {
                at(e) = v[q][r];
            }
        }
    }
    if constexpr (!OUT_G) __syncthreads();
}

// Forward FFT, Green multiply and inverse FFT of TX lines of one row (3D: row
// ky = blockIdx.y, lines along z; 2D: lines along y) of member blockIdx.z, in
// place in the half spectrum spec.
template <int N, int R>
__global__ void __launch_bounds__(LineT<N, R>::THREADS)
    k_line_green64(double2 *spec, Mesh m, double gs, const double2 *__restrict__ twid) {
    typedef LineT<N, R> L;
    extern __shared__ __align__(16) double2 lsh[];
    double2 *tw = lsh + L::TX * L::LINE;
    for (int i = threadIdx.x; i < N; i += L::THREADS) tw[i] = twid[i];
    const int kx0 = (int)blockIdx.x * L::TX, row = R == 3 ? (int)blockIdx.y : 0;
    const size_t zs = R == 3 ? (size_t)m.n * m.nh : (size_t)m.nh;
    double2 *g = spec + (size_t)blockIdx.z * m.mspec + (size_t)row * m.nh + kx0;
    const int valid = m.nh - kx0, wy = R == 3 ? wave_index(row, m.n) : 0;
    __syncthreads();
    int Ns = 1;
    if constexpr (L::REST > 1) {
        line_stage<N, R, L::REST, false, true, false>(lsh, g, zs, valid, 1, tw);
        Ns = L::REST;
    } else {
        line_stage<N, R, 8, false, true, false>(lsh, g, zs, valid, 1, tw);
        Ns = 8;
    }
    for (; Ns < N / 8; Ns *= 8) line_stage<N, R, 8, false, false, false>(lsh, g, zs, valid, Ns, tw);
    {  // the last forward stage, the multiply and the first inverse stage in registers
        constexpr int NB = N / 8;
        const int l = (int)threadIdx.x % L::TX, j = (int)threadIdx.x / L::TX;
        auto at = [&](int e) -> double2 & { return lsh[(e + (e >> 3)) * L::TX + l]; };
        double2 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) v[r] = at(j + r * NB);
        __syncthreads();
#pragma unroll
        for (int r = 1; r < 8; ++r) v[r] = cmul(v[r], tw[(j * r) & (N - 1)]);
        dft_small<8, false>(v);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int kz = wave_index(j + r * NB, N);
            const long long k2 = (long long)(kx0 + l) * (kx0 + l) + (long long)wy * wy + (long long)kz * kz;
            const double f = k2 > 0 ? gs / (double)k2 : 0.0;
            v[r].x *= f;
            v[r].y *= f;
        }
        dft_small<8, true>(v);
#pragma unroll
        for (int r = 0; r < 8; ++r) at(8 * j + r) = v[r];
        __syncthreads();
    }
    Ns = 8;
    if constexpr (L::REST > 1) {
        for (; Ns < N / L::REST; Ns *= 8) line_stage<N, R, 8, true, false, false>(lsh, g, zs, valid, Ns, tw);
        line_stage<N, R, L::REST, true, false, true>(lsh, g, zs, valid, N / L::REST, tw);
    } else {
        for (; Ns < N / 8; Ns *= 8) line_stage<N, R, 8, true, false, false>(lsh, g, zs, valid, Ns, tw);
        line_stage<N, R, 8, true, false, true>(lsh, g, zs, valid, N / 8, tw);
    }
}

}  // namespace conan
