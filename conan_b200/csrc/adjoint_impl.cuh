// adjoint_impl.cuh -- the differentiable PM model (conan_diff_*): white noise
// -> initial conditions -> Zel'dovich start -> n leapfrog steps -> final CIC
// density, and its hand-written adjoint. Included by pm.cu after PM<T,R>.
//
// Forward step i (state s_i = (d_i, p_i) at the start of the step):
//   drift  d_{i+1} = d_i + cd_i p_i
//   kick   p_{i+1} = p_i - ck_i F(d_{i+1}),
//   F_j = sum_b W^g_b(x_j) G(c^g_b),  G = FD4(phi),  phi = Green * delta,
//   delta(c) = mass sum_j W^d(x_j, c) - 1
// (W^g: the gather's CIC weights with the reference's truncating origin,
// W^d: the deposit's weights). Adjoint of step i, given (dbar, pbar) of
// s_{i+1} and v = pbar:
//   dbar -= ck_i J^T v,   pbar = v + cd_i dbar,
//   (J^T v)_j = sum_b dW^g_b(x_j) (v_j . G(c^g_b))
//             + mass sum_b dW^d_b(x_j) rhobar(c^d_b),
//   rhobar = Green * ( -sum_k FD4_k(U_k) ),  U_k = gather-transpose deposit
//   of v_k (the Green operator is symmetric and FD4 antisymmetric).
// The state is run backwards reversibly (p_i = p_{i+1} + ck_i F(d_{i+1}),
// d_i = d_{i+1} - cd_i p_i) with the exact state restored from a checkpoint
// every k steps, which bounds the FP32 reversal error.
#pragma once

#include "ic.cuh"

namespace conan {

// dW_b/dx_k of the CIC weight of corner b, with a0 = 1 - a1 per axis.
template <typename T, int R> __device__ inline T dweight(const T *a0, const T *a1, int b, int k) {
    T z = ((b >> k) & 1) ? T(1) : T(-1);
#pragma unroll
    for (int l = 0; l < R; ++l)
        if (l != k) z *= ((b >> l) & 1) ? a1[l] : a0[l];
    return z;
}

// Deposit cell and weights of particle i exactly as the forward deposit
// forms them (the FP32 deposit position is rounded to 2^-21 cell).
template <typename T, int R>
__device__ inline void deposit_corner_frame(const Parts<T> &P, const Mesh &m, size_t i, const T *d, int *cell,
                                            T *a0, T *a1) {
    int q[3];
    lattice<T, R>(P, i, q);
#pragma unroll
    for (int k = 0; k < R; ++k) {
        if constexpr (sizeof(T) == 4) {
            uint32_t fr;
            Pay<float>::cell_frac(d[k], q[k], m.n - 1, &cell[k], &fr);
            a1[k] = (float)fr * 0x1p-21f;
        } else {
            double fr;
            Pay<double>::cell_frac(d[k], q[k], m.n - 1, &cell[k], &fr);
            a1[k] = fr;
        }
        a0[k] = T(1) - a1[k];
    }
}

template <int R> __device__ inline uint32_t corner_index(const int *o, int b, const Mesh &m) {
    uint32_t ci = 0;
#pragma unroll
    for (int k = R - 1; k >= 0; --k) ci = (ci << m.shift) | (uint32_t)((o[k] + ((b >> k) & 1)) & (m.n - 1));
    return ci;
}

// dbar_i = mass sum_b dW^d_b(x_i) deltabar(c_b): adjoint of the final deposit.
template <typename T, int R>
__global__ void k_adj_deposit_grad(Parts<T> P, Mesh m, const T *__restrict__ deltabar, double mass, T *db0, T *db1,
                                   T *db2) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.np) return;
    T d[3], a0[3], a1[3];
    int cell[3];
#pragma unroll
    for (int k = 0; k < R; ++k) d[k] = P.d[k][i];
    deposit_corner_frame<T, R>(P, m, i, d, cell, a0, a1);
    T g[3] = {T(0), T(0), T(0)};
    deltabar += cell_base(P, m, i);
#pragma unroll
    for (int b = 0; b < (1 << R); ++b) {
        T v = __ldg(deltabar + corner_index<R>(cell, b, m));
#pragma unroll
        for (int k = 0; k < R; ++k) g[k] += dweight<T, R>(a0, a1, b, k) * v;
    }
    T *db[3] = {db0, db1, db2};
#pragma unroll
    for (int k = 0; k < R; ++k) db[k][i] = (T)mass * g[k];
}

// Running maximum of |pbar|: the warps of k_adj_step reduce into ABS_SLOTS
// slots, one 32-byte sector each (a maximum does not depend on the order), as
// the bits of non-negative doubles, which order as integers.
constexpr int ABS_SLOTS = 128;

__device__ inline void absmax_add(unsigned long long *slots, unsigned lanes, unsigned slot, float v) {
    const float mx = __uint_as_float(__reduce_max_sync(lanes, __float_as_uint(v)));
    if ((threadIdx.x & 31) == 0)
        atomicMax(slots + 4 * slot, (unsigned long long)__double_as_longlong((double)mx));
}
__device__ inline void absmax_add(unsigned long long *slots, unsigned lanes, unsigned slot, double v) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mh = __reduce_max_sync(lanes, hi);
    const unsigned ml = __reduce_max_sync(lanes, hi == mh ? lo : 0u);
    if ((threadIdx.x & 31) == 0) atomicMax(slots + 4 * slot, ((unsigned long long)mh << 32) | ml);
}

// Fixed-point exponent S for the vector deposit of values up to the slots'
// maximum: every cell sum of |v| w 2^S stays below 2^61 (gather weights with
// the truncating origin can reach 3 per axis). Clears the slots.
__global__ void __launch_bounds__(ABS_SLOTS) k_fix_exponent(unsigned long long *slots, double np, int R, int *S) {
    __shared__ unsigned long long part[ABS_SLOTS];
    part[threadIdx.x] = slots[4 * threadIdx.x];
    slots[4 * threadIdx.x] = 0ull;
    for (int h = ABS_SLOTS / 2; h > 0; h >>= 1) {
        __syncthreads();
        if ((int)threadIdx.x < h) part[threadIdx.x] = max(part[threadIdx.x], part[threadIdx.x + h]);
    }
    if (threadIdx.x != 0) return;
    const double mx = __longlong_as_double((long long)part[0]);
    int s = 0;
    if (mx > 0) {
        const double lg = log2(mx) + log2(np) + 2.0 * R;
        s = max(-1000, min(1000, (int)floor(61.0 - lg)));
    }
    *S = s;
}

// U_k(c) += v_k W^g_b for every particle and gather corner, in 64-bit
// fixed point (integer atomics: the sums are exact and order-independent).
// Bound by the load/store units' and L2's 64-bit reductions (2^R R adds of 8
// bytes per particle). MERGE: fewer of them reach the L2. One thread takes
// two particles that follow each other along the slowest axis; where the
// second sits one cell further along that axis, the first's upper corners are
// the second's lower ones and their integers are added in registers. Likewise
// along x: a lane whose origin is one cell beyond the lane before it adds that
// lane's upper-x values (shuffles) to its own lower-x ones. Integer sums, so
// the same bits. 256^3 particles, a = 0.3: 795 -> 600 us; without the x
// merge 690, with four or eight particles per thread 650, one 640.
template <typename T, int R, bool MERGE>
__global__ void __launch_bounds__(256)
    k_adj_vec_deposit(Parts<T> P, Mesh m, const T *__restrict__ v0, const T *__restrict__ v1, const T *__restrict__ v2,
                      int periodic, const int *__restrict__ S, unsigned long long *U0, unsigned long long *U1,
                      unsigned long long *U2) {
    constexpr int NZ = MERGE ? 2 : 1;
    const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.np / NZ) return;
    const int ls = (R - 1) * P.mshift;  // log2 of the particles per layer of the slowest axis
    const size_t i0 = (t & (((size_t)1 << ls) - 1)) | ((t >> ls) * NZ << ls);
    const T *vv[3] = {v0, v1, v2};
    const size_t cb = cell_base(P, m, i0);  // the NZ particles belong to one member
    unsigned long long *U[3] = {U0 + cb, U1 + cb, U2 + cb};
    const double sc = ldexp(1.0, *S);  // a power of two: v z sc is exact in double for FP32
    // rn(x sc): for 2^18 particles and more the fixed-point exponent keeps
    // |x sc| below 2^43, so one fused multiply-add onto 1.5 2^52 leaves the
    // rounded integer in the mantissa (the conversion instruction runs at a
    // quarter of that rate)
    auto fix = [&](double x) -> long long {
        if constexpr (MERGE)
            return __double_as_longlong(__fma_rn(x, sc, 6755399441055744.0)) - 0x4338000000000000LL;
        else
            return __double2ll_rn(x * sc);
    };
    constexpr int HALF = 1 << (R - 1);
    auto emit = [&](const int *o, int b, const long long *q) {
        const uint32_t ci = corner_index<R>(o, b, m);
#pragma unroll
        for (int k = 0; k < R; ++k)
            if (q[k]) atomicAdd(U[k] + ci, (unsigned long long)q[k]);
    };
    int po[3] = {0, 0, 0};
    long long pend[HALF][R];
#pragma unroll
    for (int j = 0; j < NZ; ++j) {
        const size_t i = i0 + ((size_t)j << ls);
        int q[3], o[3] = {0, 0, 0};
        T a0[3], a1[3], v[3];
        lattice<T, R>(P, i, q);
#pragma unroll
        for (int k = 0; k < R; ++k) {
            gather_axis<T>(P.d[k][i], q[k], periodic != 0, &o[k], &a1[k]);
            a0[k] = T(1) - a1[k];
            v[k] = vv[k][i];
        }
        bool meet = j > 0 && o[R - 1] == po[R - 1] + 1;
#pragma unroll
        for (int k = 0; k < R - 1; ++k) meet = meet && o[k] == po[k];
        // the lane before this one sits one cell back along x: its
        // upper-x corners are this lane's lower-x corners
        bool take = false, give = false;
        if constexpr (MERGE) {
            take = (threadIdx.x & 31) != 0;
#pragma unroll
            for (int k = 0; k < R; ++k) {
                const int ok = __shfl_up_sync(FULL, o[k], 1);
                take = take && ok + (k == 0 ? 1 : 0) == o[k];
            }
            give = __shfl_down_sync(FULL, (int)take, 1) != 0 && (threadIdx.x & 31) != 31;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // the lower, then the upper layer
            long long w[HALF][R];
#pragma unroll
            for (int b = 0; b < HALF; ++b) {
                const int c = h * HALF + b;
                T z = 1;
#pragma unroll
                for (int k = 0; k < R; ++k) z *= ((c >> k) & 1) ? a1[k] : a0[k];
#pragma unroll
                for (int k = 0; k < R; ++k) w[b][k] = fix((double)v[k] * (double)z);
            }
            if (h == 0 && j > 0) {
                if (meet) {
#pragma unroll
                    for (int b = 0; b < HALF; ++b)
#pragma unroll
                        for (int k = 0; k < R; ++k) w[b][k] += pend[b][k];
                } else {
#pragma unroll
                    for (int b = 0; b < HALF; ++b) emit(po, HALF + b, pend[b]);
                }
            }
            if (h == 0 || j + 1 == NZ) {
                if constexpr (MERGE) {
#pragma unroll
                    for (int b = 0; b < HALF; b += 2)
#pragma unroll
                        for (int k = 0; k < R; ++k) {
                            const long long u = __shfl_up_sync(FULL, w[b + 1][k], 1);
                            if (take) w[b][k] += u;
                        }
                }
#pragma unroll
                for (int b = 0; b < HALF; ++b)
                    if (!MERGE || !(b & 1) || !give) emit(o, h * HALF + b, w[b]);
            } else {
#pragma unroll
                for (int b = 0; b < HALF; ++b)
#pragma unroll
                    for (int k = 0; k < R; ++k) pend[b][k] = w[b][k];
            }
        }
#pragma unroll
        for (int k = 0; k < R; ++k) po[k] = o[k];
    }
}

// out(c) = -sum_k FD4_k(U_k)(c): the adjoint of the FD4 gradient, from the
// fixed-point meshes (scale 2^-S) or from real meshes (S == nullptr).
template <typename T, int R, typename UT>
__global__ void k_neg_div(const UT *__restrict__ U0, const UT *__restrict__ U1, const UT *__restrict__ U2,
                          const int *__restrict__ S, T *__restrict__ out, Mesh m) {
    uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.cells) return;
    const UT *U[3] = {U0, U1, U2};
    const uint32_t mask = m.n - 1;
    const double sc = S ? ldexp(1.0, -*S) : 1.0;
    double acc = 0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const int sh = k * m.shift;
        uint32_t ck = (c >> sh) & mask, rest = c & ~(mask << sh);
        auto at = [&](int o) -> double {
            UT x = U[k][rest | (((ck + o) & mask) << sh)];
            if constexpr (sizeof(UT) == 8 && !std::is_floating_point<UT>::value)
                return (double)(long long)x;
            else
                return (double)x;
        };
        acc += (at(-2) - at(2)) / 12.0 + (at(1) - at(-1)) * (2.0 / 3.0);
    }
    out[c] = (T)(-acc * sc);
}

// 12 FD4 of the values at -2, -1, 1, 2 of a line. Fixed-point values are
// combined as integers: the exponent keeps a component's sum over all cells
// below 2^60, so |u(-2) - u(2) + 8 (u(1) - u(-1))| < 2^63 for four distinct
// cells: exact, and one conversion instead of four.
__device__ inline double fd4_x12(unsigned long long m2, unsigned long long m1, unsigned long long p1,
                                 unsigned long long p2) {
    return (double)(long long)((m2 - p2) + ((p1 - m1) << 3));
}
template <typename T> __device__ inline double fd4_x12(T m2, T m1, T p1, T p2) {
    return ((double)m2 - (double)p2) + 8.0 * ((double)p1 - (double)m1);
}

// The same for 3D meshes of 32 cells per side and more: a block of 32 x 8
// threads marches NDZ planes along z, so that each thread keeps its column's
// five U2 values in registers and the rows it reads for y stay in L1. Bound
// by the L2 reads of the thread-per-cell form (nine mesh values per cell
// instead of three); fixed-point meshes, 128^3 21 -> 14 us, 256^3 161 -> 114
// (with 16 planes 24 and 125, with 4 14 and 110 but 126 instead of 82 us for
// real meshes).
constexpr int NDZ = 8;
template <typename T, typename UT>
__global__ void __launch_bounds__(256)
    k_neg_div_z(const UT *__restrict__ U0, const UT *__restrict__ U1, const UT *__restrict__ U2,
                const int *__restrict__ S, T *__restrict__ out, Mesh m) {
    const uint32_t mask = (uint32_t)m.n - 1;
    const int s = m.shift;
    unsigned b = blockIdx.x;
    const uint32_t x = (b & ((1u << (s - 5)) - 1)) * 32 + (threadIdx.x & 31);
    b >>= s - 5;
    const uint32_t y = (b & ((1u << (s - 3)) - 1)) * 8 + (threadIdx.x >> 5);
    b >>= s - 3;
    const uint32_t nz = (unsigned)m.n / NDZ;
    const uint32_t z0 = (b & (nz - 1)) * NDZ;
    const size_t mb = (size_t)(b / nz) << m.cshift;
    U0 += mb;
    U1 += mb;
    U2 += mb;
    out += mb;
    const uint32_t col = (y << s) | x;
    uint32_t rx[5], ry[5];  // offsets of the x and y neighbours in a plane
#pragma unroll
    for (int o = 0; o < 5; ++o) {
        rx[o] = (y << s) | ((x + o - 2) & mask);
        ry[o] = (((y + o - 2) & mask) << s) | x;
    }
    auto plane = [&](uint32_t z) { return (z & mask) << (2 * s); };
    UT q[5];  // this column at z - 2 .. z + 2
#pragma unroll
    for (int j = 0; j < 4; ++j) q[j] = __ldg(U2 + (plane(z0 + j - 2) | col));
    const double sc = (S ? ldexp(1.0, -*S) : 1.0) * (-1.0 / 12.0);
#pragma unroll 4
    for (int zi = 0; zi < NDZ; ++zi) {
        const uint32_t z = z0 + zi, pz = plane(z);
        q[4] = __ldg(U2 + (plane(z + 2) | col));
        const UT *__restrict__ a = U0 + pz, *__restrict__ c = U1 + pz;
        double acc = fd4_x12(__ldg(a + rx[0]), __ldg(a + rx[1]), __ldg(a + rx[3]), __ldg(a + rx[4]));
        acc += fd4_x12(__ldg(c + ry[0]), __ldg(c + ry[1]), __ldg(c + ry[3]), __ldg(c + ry[4]));
        acc += fd4_x12(q[0], q[1], q[3], q[4]);
        out[pz | col] = (T)(acc * sc);
#pragma unroll
        for (int j = 0; j < 4; ++j) q[j] = q[j + 1];
    }
}

// One adjoint step (see the file comment): updates dbar, pbar and runs the
// state back from s_{i+1} to s_i, using G = FD4 gradient at d_{i+1} and
// rhobar = Green * div (null: zero); the maximum of the new |pbar| goes into
// absmax (a pass of its own over pbar before: 160 us per step at 256^3).
// Bound by the chain of its twelve streams and 16 corner loads: in FP32 the
// register budget of four blocks per SM takes 450 us at 256^3, three 547, five
// 524. FP64 in 3D spills within four (84 bytes) and takes three: a backward of
// four steps at 256^3 13.34 -> 12.90 ms (two 13.35), of eight at 128^3 3.92 ->
// 3.80; 2D fits four. Walking the lattice in 16 x 4 x 4 tiles 578 (half-used sectors of the
// streams cost more than the corner reads' locality gains), streaming loads
// and stores 457.
template <typename T, int R>
__global__ void __launch_bounds__(256, sizeof(T) == 8 && R == 3 ? 3 : 4)
    k_adj_step(Parts<T> P, Mesh m, const G4<T> *__restrict__ G, const T *__restrict__ rhobar, T *pb0, T *pb1, T *pb2,
               T *db0, T *db1, T *db2, double ck, double cd, double mass, int periodic, unsigned long long *absmax) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned lanes = __ballot_sync(FULL, i < P.np);
    if (i >= P.np) return;
    T *pbv[3] = {pb0, pb1, pb2}, *dbv[3] = {db0, db1, db2};
    T d[3], p[3], v[3], dbar[3];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        d[k] = P.d[k][i];
        p[k] = P.p[k][i];
        v[k] = pbv[k][i];
        dbar[k] = dbv[k][i];
    }
    int q[3], o[3], cell[3];
    T a0[3], a1[3], b0[3], b1[3];
    lattice<T, R>(P, i, q);
#pragma unroll
    for (int k = 0; k < R; ++k) {
        gather_axis<T>(d[k], q[k], periodic != 0, &o[k], &a1[k]);
        a0[k] = T(1) - a1[k];
    }
    T F[3] = {T(0), T(0), T(0)}, t1[3] = {T(0), T(0), T(0)}, t2[3] = {T(0), T(0), T(0)};
    const size_t cb = cell_base(P, m, i);
    G += cb;
#pragma unroll
    for (int b = 0; b < (1 << R); ++b) {
        G4<T> g = load_g4(G + corner_index<R>(o, b, m));
        T gv[3] = {g.x, g.y, g.z};
        T z = 1, vg = 0;
#pragma unroll
        for (int k = 0; k < R; ++k) {
            z *= ((b >> k) & 1) ? a1[k] : a0[k];
            vg += v[k] * gv[k];
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            F[k] += gv[k] * z;
            t1[k] += dweight<T, R>(a0, a1, b, k) * vg;
        }
    }
    if (rhobar) {
        rhobar += cb;
        deposit_corner_frame<T, R>(P, m, i, d, cell, b0, b1);
#pragma unroll
        for (int b = 0; b < (1 << R); ++b) {
            T r = __ldg(rhobar + corner_index<R>(cell, b, m));
#pragma unroll
            for (int k = 0; k < R; ++k) t2[k] += dweight<T, R>(b0, b1, b, k) * r;
        }
    }
    T mx = T(0);
    const T tck = (T)ck, tcd = (T)cd, tm = (T)mass;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        T dbn = dbar[k] - tck * (t1[k] + tm * t2[k]);
        T pbn = v[k] + tcd * dbn;
        dbv[k][i] = dbn;
        pbv[k][i] = pbn;
        mx = fmax(mx, fabs(pbn));
        T pold = p[k] + tck * F[k];
        P.p[k][i] = pold;
        P.d[k][i] = d[k] - tcd * pold;
    }
    absmax_add(absmax, lanes, (blockIdx.x * 8 + (threadIdx.x >> 5)) % ABS_SLOTS, mx);
}

// ubar_k = cdz dbar_k + cpz pbar_k in place in dbar (particle i = mass cell
// i), all axes in one launch.
template <typename T, int R> struct ZaArrays {
    T *db[3];
    const T *pb[3];
};
template <typename T, int R>
__global__ void __launch_bounds__(256) k_za_adjoint(ZaArrays<T, R> a, size_t n, double cdz, double cpz) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    T d[R], p[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
        d[k] = a.db[k][i];
        p[k] = a.pb[k][i];
    }
#pragma unroll
    for (int k = 0; k < R; ++k) a.db[k][i] = (T)(cdz * (double)d[k] + cpz * (double)p[k]);
}

// R arrays of n values copied at once, 16 bytes per thread and array
// (cudaMalloc'd arrays). One launch instead of R copies, and faster than a
// graph's copy nodes (a 512^3 model with two checkpoints: 39.5 ms against 40.9).
template <typename T> struct CopyArrays {
    const T *src[3];
    T *dst[3];
};
template <typename T, int R> __global__ void __launch_bounds__(256) k_copy_arrays(CopyArrays<T> a, size_t n) {
    constexpr int V = 16 / sizeof(T);
    const size_t i = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) * V;
    if (i + V <= n) {
        uint4 v[R];
#pragma unroll
        for (int k = 0; k < R; ++k) v[k] = __ldcs(reinterpret_cast<const uint4 *>(a.src[k] + i));
#pragma unroll
        for (int k = 0; k < R; ++k) __stcs(reinterpret_cast<uint4 *>(a.dst[k] + i), v[k]);
    } else {
        for (int k = 0; k < R; ++k)
            for (size_t j = i; j < n; ++j) a.dst[k][j] = a.src[k][j];
    }
}

struct DiffBase {
    virtual ~DiffBase() {}
    virtual int forward(const void *noise, void *density, void *stream) = 0;
    virtual int backward(const void *gdens, void *gnoise, void *stream) = 0;
    virtual int device() const = 0;
};

template <typename T, int R> struct Diff : DiffBase {
    typedef typename Cplx<T>::type CT;
    conan_diff_params prm{};
    PM<T, R> pm;
    Mesh mm{}, mm1{};  // mass meshes of the batch and of one member
    std::vector<conan_ic_params> ic;
    // initial conditions on the mass mesh
    T *w = nullptr, *ict = nullptr, *ict2 = nullptr;
    CT *ics = nullptr, *ics2 = nullptr;
    void *icwork = nullptr;
    FFTPair icfft;
    double *part = nullptr;
    // adjoint state
    T *db[3] = {nullptr, nullptr, nullptr}, *pb[3] = {nullptr, nullptr, nullptr};
    unsigned long long *U[3] = {nullptr, nullptr, nullptr};
    T *rhobar = nullptr;
    int *S = nullptr;           // fixed-point exponent of the vector deposit
    unsigned long long *absmax = nullptr;  // slots of the running |pbar| maximum
    std::vector<T *> ckpt;  // per checkpoint: d[0..R), p[0..R)
    std::vector<double> a_start;
    cudaEvent_t ev = nullptr;
    bool have_forward = false;  // the checkpoints are those of a forward that was enqueued whole
    // the state is the final one and the gradient mesh that of the last step,
    // as forward leaves them and backward starts from (it ends at the initial
    // state)
    bool at_final = false;
    // Calls that a caller captures run when the graph does, as often as it does,
    // which the host does not see: the capture (0: none) that set at_final, and
    // whether any call was captured.
    unsigned long long final_capture = 0;
    bool captured = false;
    // The launches of a pass between the caller's buffers, captured as graphs
    // from a handle's second pass on (a few microseconds of host time per
    // launch, and there are hundreds). Forward and backward by launches, in the
    // pass that builds the graphs and by them: 32^3, 8 steps 1.61, 1.98, 1.01
    // ms; 64^3, 10 steps 1.86, 2.15, 1.27; 128^3, 16 steps 7.3, 7.5, 6.3; 256^3,
    // 6 steps 16.6, 16.7, 16.1: building costs at most two thirds of what each
    // pass gains afterwards, and waits for the second since many handles make
    // only one. Everything in them belongs to the handle.
    enum { G_STEPS, G_LAST, G_BACK, G_COUNT };
    cudaGraphExec_t graphs[G_COUNT] = {};
    unsigned graph_config = 0, passes[G_COUNT] = {};

    ~Diff() override {
        if (pm.st) cudaStreamSynchronize(pm.st);
        drop_graphs();
        icfft.destroy();
        if (ev) cudaEventDestroy(ev);
    }

    // `batch` equal boxes; member b's initial conditions use member_ic[b]
    // (default: p.ic for every member).
    int create(const conan_diff_params &p, int batch = 1,
               const std::vector<conan_ic_params> *member_ic = nullptr) {
        prm = p;
        CONAN_TRY(pm.create(p.pm, batch));
        mm = make_mesh(R, p.pm.n_mass, batch);
        mm1 = make_mesh(R, p.pm.n_mass, 1);
        ic.assign(batch, p.ic);
        if (member_ic) ic = *member_ic;
        CONAN_TRY(pm.alloc(&w, mm.cells));
        CONAN_TRY(pm.alloc(&ict, mm.cells));
        CONAN_TRY(pm.alloc(&ict2, mm.cells));
        CONAN_TRY(pm.alloc(&ics, mm.spec));
        CONAN_TRY(pm.alloc(&ics2, mm.spec));
        CONAN_TRY(pm.alloc(&part, ic_scratch(mm1)));
        CONAN_TRY(icfft.create(mm1, sizeof(T) == 8, 1));
        CONAN_TRY(pm.alloc((char **)&icwork, icfft.work_bytes ? icfft.work_bytes : 16));
        CONAN_TRY(icfft.bind(icwork, pm.st));
        // pb and U in one piece each: one memset clears all their axes
        CONAN_TRY(pm.alloc(&pb[0], R * pm.np));
        CONAN_TRY(pm.alloc(&U[0], R * pm.mf.cells));
        for (int k = 0; k < R; ++k) {
            CONAN_TRY(pm.alloc(&db[k], pm.np));
            pb[k] = pb[0] + k * pm.np;
            U[k] = U[0] + k * pm.mf.cells;
        }
        CONAN_TRY(pm.alloc(&rhobar, pm.mf.cells));
        CONAN_TRY(pm.alloc(&S, 1));
        CONAN_TRY(pm.alloc(&absmax, 4 * ABS_SLOTS));
        for (size_t i = 0; i < p.n; i += kev())  // the state before every kev()-th step
            for (int c = 0; c < 2 * R; ++c) {
                T *b = nullptr;
                CONAN_TRY(pm.alloc(&b, pm.np));
                ckpt.push_back(b);
            }
        a_start.resize(p.n + 1);
        double a = p.a0;
        for (unsigned i = 0; i <= p.n; ++i) {
            a_start[i] = a;
            a += p.da;  // LeapFrog::run accumulates a += da
        }
        CONAN_CUDA(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        return CONAN_OK;
    }
    int device() const override { return prm.pm.device; }
    unsigned kev() const { return prm.checkpoint_every ? prm.checkpoint_every : 1; }
    dim3 gp() const { return dim3((unsigned)((pm.np + 255) / 256)); }

    void drop_graphs() {
        for (auto &g : graphs) {
            if (g) cudaGraphExecDestroy(g);
            g = nullptr;
        }
    }

    // Enqueues what `body` launches on the handle's stream: directly the first
    // time, as graph `which` from then on. body must leave the solver's host
    // state as it finds it, apart from what the caller sets itself.
    template <typename F> int replay(int which, F body) {
        if (graph_config != pm.config) {  // other kernels were chosen meanwhile
            drop_graphs();
            graph_config = pm.config;
        }
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;  // a caller's capture takes the launches themselves
        CONAN_CUDA(cudaStreamIsCapturing(pm.st, &cs));
        if (debug_sync() || cs != cudaStreamCaptureStatusNone || passes[which]++ == 0) return body();
        if (!graphs[which]) {
            cudaGraph_t g = nullptr;
            CONAN_CUDA(cudaStreamBeginCapture(pm.st, cudaStreamCaptureModeThreadLocal));
            const int rc = body();
            const cudaError_t ce = cudaStreamEndCapture(pm.st, &g);
            if (rc != CONAN_OK) {
                if (g) cudaGraphDestroy(g);
                return rc;
            }
            if (ce != cudaSuccess) return set_error(CONAN_ERR_CUDA, "graph capture failed: %s", cudaGetErrorString(ce));
            const cudaError_t ie = graph_instantiate(&graphs[which], g);
            cudaGraphDestroy(g);
            if (ie != cudaSuccess) {
                graphs[which] = nullptr;
                return set_error(CONAN_ERR_CUDA, "graph instantiate failed: %s", cudaGetErrorString(ie));
            }
        }
        CONAN_CUDA(cudaGraphLaunch(graphs[which], pm.st));
        return CONAN_OK;
    }

    // The caller's capture that the handle's stream takes part in (0: none).
    int capture_id(unsigned long long *id) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        unsigned long long v = 0;
        CONAN_CUDA(cudaStreamGetCaptureInfo(pm.st, &cs, &v));
        *id = cs == cudaStreamCaptureStatusNone ? 0 : v;
        captured = captured || *id;
        return CONAN_OK;
    }
    // Whether this call (of capture `id`) finds the final state on the device:
    // if the forward that left it there belongs to the same capture, or if
    // neither it nor any other call of the handle was captured.
    bool final_known(unsigned long long id) const {
        return at_final && final_capture == id && (id || !captured);
    }

    // Orders the handle's stream after the caller's work. NULL is the legacy
    // default stream (where torch enqueues unless told otherwise), which a
    // non-blocking stream does not wait for by itself.
    int enter(void *stream) {
        CONAN_CUDA(cudaEventRecord(ev, stream ? (cudaStream_t)stream : cudaStreamLegacy));
        CONAN_CUDA(cudaStreamWaitEvent(pm.st, ev, 0));
        return CONAN_OK;
    }
    int leave(void *stream) {
        if (stream) {
            CONAN_CUDA(cudaEventRecord(ev, pm.st));
            CONAN_CUDA(cudaStreamWaitEvent((cudaStream_t)stream, ev, 0));
            return CONAN_OK;
        }
        CONAN_CUDA(cudaStreamSynchronize(pm.st));
        return pm.check_err();
    }
    int copy_arrays(T *const *dst, T *const *src) {
        CopyArrays<T> c{};
        for (int k = 0; k < R; ++k) {
            c.src[k] = src[k];
            c.dst[k] = dst[k];
        }
        const size_t nt = (pm.np * sizeof(T) + 15) / 16;
        k_copy_arrays<T, R><<<(unsigned)((nt + 255) / 256), 256, 0, pm.st>>>(c, pm.np);
        CONAN_LAUNCHED();
        return CONAN_OK;
    }
    // Positions (mom = false) or momenta of the current state into a slot.
    int save_ckpt(unsigned slot, bool mom) {
        return copy_arrays(&ckpt[slot * 2 * R + (mom ? R : 0)], mom ? pm.P.p : pm.P.d);
    }
    int load_ckpt(unsigned slot) {
        CONAN_TRY(pm.positions_reset());
        CONAN_TRY(copy_arrays(pm.P.d, &ckpt[slot * 2 * R]));
        return copy_arrays(pm.P.p, &ckpt[slot * 2 * R + R]);
    }
    double cdz() const { return -prm.a0 / (pm.res_m * pm.res_f); }
    double cpz() const { return -(prm.a0 + prm.da / 2) / (pm.res_m * pm.res_f); }

    // The noise (device, batch) into the handle; what the solver had pending of
    // other positions is dropped.
    int take_noise(const void *noise) {
        have_forward = at_final = false;
        CONAN_CUDA(cudaMemcpyAsync(w, noise, mm.cells * sizeof(T), cudaMemcpyDeviceToDevice, pm.st));
        CONAN_TRY(pm.positions_reset());
        pm.a_pos = prm.a0;
        pm.a_mom = prm.a0 + prm.da / 2;
        return CONAN_OK;
    }
    // Initial conditions of every member from the handle's noise and the
    // Zel'dovich start of the particle state at (a0, a0 + da/2).
    int start_state() {
        cudaStream_t st = pm.st;
        for (int b = 0; b < mm.batch; ++b) {  // initial conditions, member by member
            T *x = ict + member_cells(mm, b);
            CONAN_TRY(grf_device<T>(ic[b], mm1, w + member_cells(mm, b), x, ics, icfft, part, st));
            CONAN_TRY(potential_device<T>(mm1, ic[b].size, x, ics, icfft, st));
        }
        k_zeldovich<T, R><<<gp(), 256, 0, st>>>(pm.P, ict, mm, cdz(), cpz());
        CONAN_LAUNCHED();
        return CONAN_OK;
    }
    int initial_state(const void *noise) {
        CONAN_TRY(take_noise(noise));
        return start_state();
    }

    // From the state before step i0 up to the last deposit. The kick of a step
    // and the drift (with its deposit) of the next are one launch, as in a run;
    // a checkpoint between them takes the positions before it (a kick moves
    // none) and the momenta after it (a drift changes none).
    int steps_from(unsigned i0) {
        CONAN_TRY(pm.gkd(false, 0, true, pm.coef_drift(a_start[i0], prm.da), true));
        for (unsigned i = i0; i + 1 < prm.n; ++i) {
            const double am = a_start[i] + prm.da / 2;
            const bool save = (i + 1) % kev() == 0;
            CONAN_TRY(pm.deposit_poisson(am));
            if (save) CONAN_TRY(save_ckpt((i + 1) / kev(), false));
            CONAN_TRY(pm.gkd(true, pm.coef_kick(am, prm.da), true, pm.coef_drift(a_start[i + 1], prm.da), true));
            if (save) CONAN_TRY(save_ckpt((i + 1) / kev(), true));
        }
        return pm.deposit_for_solve();
    }
    int forward_steps() {
        CONAN_TRY(start_state());
        CONAN_TRY(save_ckpt(0, false));
        CONAN_TRY(save_ckpt(0, true));
        return steps_from(0);
    }
    int forward_last() {
        const double am = a_start[prm.n - 1] + prm.da / 2;
        CONAN_TRY(pm.solve_deposited(am));
        return pm.gkd(true, pm.coef_kick(am, prm.da), false, 0, false);
    }
    // The final state again, from the last checkpoint: the forward's own
    // launches from there, so its bits.
    int restore_final() {
        const unsigned slot = (prm.n - 1) / kev();
        CONAN_TRY(load_ckpt(slot));
        CONAN_TRY(steps_from(slot * kev()));
        return forward_last();
    }

    int forward(const void *noise, void *density, void *stream) override {
        const int rc = forward_pass(noise, density, stream);
        return rc == CONAN_OK ? rc : pm.failed(rc);
    }
    int forward_pass(const void *noise, void *density, void *stream) {
        CONAN_TRY(enter(stream));
        unsigned long long cap = 0;
        CONAN_TRY(capture_id(&cap));
        CONAN_TRY(take_noise(noise));
        CONAN_TRY(replay(G_STEPS, [&] { return forward_steps(); }));
        // the positions of the last deposit are the final ones: its density
        // is the output
        CONAN_TRY(pm.deposited_density((T *)density));
        CONAN_TRY(replay(G_LAST, [&] { return forward_last(); }));
        pm.mesh_holds = 2;
        at_final = have_forward = true;
        final_capture = cap;
        return leave(stream);
    }

    template <typename UT> int neg_div(UT *const *u, const int *exps, T *out, const Mesh &m) {
        if constexpr (R == 3) {
            if (m.n >= 32) {
                const unsigned blocks = (unsigned)(m.cells / (256 * NDZ));
                k_neg_div_z<T, UT><<<blocks, 256, 0, pm.st>>>(u[0], u[1], u[2], exps, out, m);
                CONAN_LAUNCHED();
                return CONAN_OK;
            }
        }
        k_neg_div<T, R, UT><<<(unsigned)((m.cells + 255) / 256), 256, 0, pm.st>>>(u[0], u[1], u[2], exps, out, m);
        CONAN_LAUNCHED();
        return CONAN_OK;
    }

    // rhobar = Green(a) * (-sum_k FD4_k(U_k)) without touching the gradient mesh
    int adjoint_poisson(double am) {
        CONAN_TRY(neg_div(U, S, rhobar, pm.mf));
        const double gsc = pm.poisson_scale(am);
        if (pm.zpass) {  // the forward solve's plane transforms and z pass
            CONAN_TRY(pm.fft2.forward(rhobar, pm.spec));
            CONAN_TRY(pm.green_z(gsc));
            CONAN_TRY(pm.fft2.inverse(pm.spec, rhobar));
            return CONAN_OK;
        }
        CONAN_TRY(pm.fft.forward(rhobar, pm.spec));
        CONAN_TRY(pm.green(pm.spec, gsc));
        CONAN_TRY(pm.fft.inverse(pm.spec, rhobar));
        return CONAN_OK;
    }

    // U = gather-transpose deposit of pb. The merging kernel needs whole warps
    // within one member (8 particles per side) and, for its one-instruction
    // rounding, a fixed-point exponent that leaves particles below 2^51 units:
    // 2^18 particles are enough for both (and smaller lattices are launch-bound
    // either way).
    int vec_deposit() {
        cudaStream_t st = pm.st;
        if (R > 1 && mm.n >= 8 && pm.np >= ((size_t)1 << 18)) {
            const size_t nt = pm.np / 2;
            k_adj_vec_deposit<T, R, (R > 1)><<<(unsigned)((nt + 255) / 256), 256, 0, st>>>(
                pm.P, pm.mf, pb[0], pb[1], pb[2], prm.pm.periodic_gather, S, U[0], U[1], U[2]);
        } else {
            k_adj_vec_deposit<T, R, false><<<gp(), 256, 0, st>>>(pm.P, pm.mf, pb[0], pb[1], pb[2],
                                                                 prm.pm.periodic_gather, S, U[0], U[1], U[2]);
        }
        CONAN_LAUNCHED();
        return CONAN_OK;
    }

    // Every adjoint step from the density's adjoint in db, the final state
    // and its gradient mesh back to the initial state.
    int backward_steps() {
        cudaStream_t st = pm.st;
        const Mesh &mf = pm.mf;
        CONAN_CUDA(cudaMemsetAsync(pb[0], 0, R * pm.np * sizeof(T), st));
        // the previous backward's first step left its maximum behind
        CONAN_CUDA(cudaMemsetAsync(absmax, 0, 4 * ABS_SLOTS * sizeof(unsigned long long), st));
        for (int i = (int)prm.n - 1; i >= 0; --i) {
            double a = a_start[i], am = a + prm.da / 2;
            double ck = pm.coef_kick(am, prm.da), cd = pm.coef_drift(a, prm.da);
            // forward force at d_{i+1}: deposit, potential, gradient mesh (the
            // last step's is there). U = gather-transpose deposit of v = pbar
            // and the density's adjoint rhobar; pbar is zero in the last step
            // (the loss sees positions only), and so is rhobar
            const bool vz = i == (int)prm.n - 1;
            if (!vz) {
                CONAN_TRY(pm.deposit_poisson(am));
                k_fix_exponent<<<1, ABS_SLOTS, 0, st>>>(absmax, (double)pm.np, R, S);
                CONAN_LAUNCHED();
                CONAN_CUDA(cudaMemsetAsync(U[0], 0, R * mf.cells * sizeof(unsigned long long), st));
                CONAN_TRY(vec_deposit());
                CONAN_TRY(adjoint_poisson(am));
            }
            k_adj_step<T, R><<<gp(), 256, 0, st>>>(pm.P, mf, pm.grad, vz ? nullptr : rhobar, pb[0], pb[1], pb[2],
                                                   db[0], db[1], db[2], ck, cd, pm.mass, prm.pm.periodic_gather, absmax);
            CONAN_LAUNCHED();
            if ((unsigned)i % kev() == 0) CONAN_TRY(load_ckpt((unsigned)i / kev()));
        }
        return CONAN_OK;
    }

    int backward(const void *gdens, void *gnoise, void *stream) override {
        if (!have_forward) return set_error(CONAN_ERR_STATE, "backward without a forward call");
        const int rc = backward_pass(gdens, gnoise, stream);
        return rc == CONAN_OK ? rc : pm.failed(rc);
    }
    int backward_pass(const void *gdens, void *gnoise, void *stream) {
        CONAN_TRY(enter(stream));
        cudaStream_t st = pm.st;
        unsigned long long cap = 0;
        CONAN_TRY(capture_id(&cap));
        if (!final_known(cap)) CONAN_TRY(restore_final());  // a further gradient of the same forward
        at_final = false;
        // the density adjoint through the final deposit
        k_adj_deposit_grad<T, R><<<gp(), 256, 0, st>>>(pm.P, pm.mf, (const T *)gdens, pm.mass, db[0], db[1], db[2]);
        CONAN_LAUNCHED();
        CONAN_TRY(replay(G_BACK, [&] { return backward_steps(); }));
        pm.mesh_holds = 2;
        // Zel'dovich, potential and random-field adjoints on the mass mesh
        unsigned gm = (unsigned)((mm.cells + 255) / 256);
        ZaArrays<T, R> za{};
        for (int k = 0; k < R; ++k) {
            za.db[k] = db[k];
            za.pb[k] = pb[k];
        }
        k_za_adjoint<T, R><<<gm, 256, 0, st>>>(za, mm.cells, cdz(), cpz());
        CONAN_LAUNCHED();
        CONAN_TRY(neg_div(db, nullptr, ict, mm));
        for (int b = 0; b < mm.batch; ++b) {
            const size_t o = member_cells(mm, b);
            CONAN_TRY(potential_device<T>(mm1, ic[b].size, ict + o, ics, icfft, st));
            CONAN_TRY(grf_adjoint_device<T>(ic[b], mm1, w + o, ict + o, (T *)gnoise + o, ics, ics2, ict2, icfft,
                                            part, st));
        }
        return leave(stream);
    }
};

inline DiffBase *make_diff(const conan_diff_params &p) {
    DiffBase *b = nullptr;
    int rc = CONAN_OK;
#define MAKE_DIFF(T, R)               \
    {                                 \
        auto *x = new Diff<T, R>();   \
        rc = x->create(p);            \
        b = x;                        \
    }
    if (p.pm.precision == CONAN_FP32) {
        if (p.pm.dim == 1) MAKE_DIFF(float, 1) else if (p.pm.dim == 2) MAKE_DIFF(float, 2) else MAKE_DIFF(float, 3)
    } else {
        if (p.pm.dim == 1) MAKE_DIFF(double, 1) else if (p.pm.dim == 2) MAKE_DIFF(double, 2) else MAKE_DIFF(double, 3)
    }
#undef MAKE_DIFF
    if (rc != CONAN_OK) {
        std::string msg = last_error();
        delete b;
        last_error() = msg;
        return nullptr;
    }
    return b;
}

}  // namespace conan
