// fof.cu -- the `fof` tool on the GPU: friends-of-friends groups of a
// snapshot's particles, fof_run<R> (src/fof/fof.cc:164-279).
//
// The reference links two particles when the squared length of their raw
// coordinate difference, wrapped once per axis into [-L/2, L/2] (Proximity,
// src/fof/fof.cc:71-99), is at most the squared linking length, and numbers
// the connected groups from 1 in the order of their lowest particle index
// (the flood fill started from every untagged particle in index order,
// src/fof/fof.cc:183-231). The result is a partition plus that numbering, so
// any order of discovery gives the same tags. Here:
//   keys     every particle's row -- its cell in the transverse axes (y, or
//            y and z) on a grid of cells no smaller than the linking length,
//            wrapped coordinates -- and its wrapped x quantised to 2^16
//            steps, as one 64-bit key; an integer count per row;
//   sort     counting sort by row (offsets from the counts; one 64-bit value
//            of x and particle index per particle), then every row sorted by
//            it: across the lanes of a warp up to 32 particles (four rows of up
//            to 8 at once), in shared memory up to 4096; a longer row sends
//            the whole array through a stable radix sort of (key, particle
//            index) instead (radix.cuh). Either way: rows in order, x
//            ascending inside a row, ties in particle order;
//   gather   coordinates (one array per axis) in sorted order;
//   link     every sorted particle is tested, in its own row, against the
//            particles ahead of it in cyclic x order within the linking
//            length, and in the forward half of the neighbouring rows
//            ((3^(R-1) - 1) / 2 rows) against those within the linking length
//            in x, found by binary search; a warp shares the candidates of its
//            32 particles evenly among its lanes; every pair within reach is
//            tested exactly once, in FP64 with the reference's operation order
//            and no fused multiply-add. A linked pair joins two trees of a
//            lock-free union-find over the sorted positions (neighbours in
//            memory) that always hooks the larger root under the smaller one;
//   roots    every position's root (a read-only walk once the links are in),
//            every tree's lowest particle index;
//   number   exclusive scan over the particles of the flags of those lowest
//            particles = group number - 1.
// Against cubic cells, the row-and-window search tests candidates from a
// volume of 2 ll x (3 ll)^(R-1) around each particle instead of (3 h)^R with
// cells h >= ll; inside halos that is most of the work.
#include <algorithm>
#include <cmath>

#include "hostio.cuh"
#include "pm.cuh"
#include "radix.cuh"
#include "scan.cuh"

namespace conan {
namespace {

constexpr int FOF_T = 256;
constexpr int FOF_UNITE_LIMIT = 1 << 24;  // retries of one union (each one is another thread's hook)
constexpr int FOF_XB = 16;                 // bits of the quantised x in the sort key
constexpr uint32_t FOF_XN = 1u << FOF_XB;
constexpr uint64_t FOF_XMASK = FOF_XN - 1;

struct FofGrid {
    int nr;         // row cells per transverse axis (1 or >= 3)
    int wq;         // x window in quanta; whole rows when 2 wq + 1 >= 2^16
    double L;       // box size
    double half;    // L / 2
    double inv_h;   // nr / L
    double xscale;  // 2^16 / L
    double rsqr;    // linking length squared
};

// Wrapped coordinate in [0, L], explicitly rounded.
__device__ inline double fof_wrap(double x, const FofGrid &g) {
    return __dsub_rn(x, __dmul_rn(floor(__ddiv_rn(x, g.L)), g.L));
}

// Row of a position (transverse cells, highest axis most significant) and
// its key: row << 16 | quantised x.
template <int R>
__device__ inline uint64_t fof_key(const double *x, const FofGrid &g, uint32_t *row_out) {
    uint32_t row = 0;
#pragma unroll
    for (int k = R - 1; k >= 1; --k) {
        int ck = (int)__dmul_rn(fof_wrap(x[k], g), g.inv_h);
        ck = ck < 0 ? 0 : (ck >= g.nr ? g.nr - 1 : ck);
        row = row * (uint32_t)g.nr + (uint32_t)ck;
    }
    long long q = (long long)__dmul_rn(fof_wrap(x[0], g), g.xscale);
    q = q < 0 ? 0 : (q >= (long long)FOF_XN ? (long long)FOF_XN - 1 : q);
    *row_out = row;
    return ((uint64_t)row << FOF_XB) | (uint64_t)q;
}

// Proximity::operator()(size_t), src/fof/fof.cc:85-99: b = x_j - x_i, one
// wrap per axis, d.sqr() summed in axis order, compared with r * r.
template <int R>
__device__ inline bool fof_linked(const double *a, const double *b, const FofGrid &g) {
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < R; ++k) {
        const double e = __dsub_rn(b[k], a[k]);
        const double d = e > g.half ? __dsub_rn(e, g.L) : (e < -g.half ? __dadd_rn(e, g.L) : e);
        v = __dadd_rn(v, __dmul_rn(d, d));
    }
    return v <= g.rsqr;
}

// Root of x with path halving. Parents always point to lower indices, so the
// walk ends; a halving store writes an ancestor of x, which stays valid
// whatever other threads do to the tree meanwhile. Loads bypass L1 so that
// hooks made by other SMs are seen.
__device__ inline uint32_t fof_find(uint32_t *par, uint32_t x) {
    for (;;) {
        const uint32_t p = __ldcg(par + x);
        if (p == x) return x;
        const uint32_t g = __ldcg(par + p);
        if (g == p) return p;
        __stcg(par + x, g);
        x = g;
    }
}

// Joins the trees of a and b: the larger root is hooked under the smaller
// one with a compare-and-swap that only succeeds while it is still a root.
// Pairs that share a parent are in one tree already (most pairs inside a
// halo). False if it gave up.
__device__ inline bool fof_unite(uint32_t *par, uint32_t a, uint32_t b) {
    for (int it = 0; it < FOF_UNITE_LIMIT; ++it) {
        a = fof_find(par, a);
        b = fof_find(par, b);
        if (a == b) return true;
        const uint32_t hi = a > b ? a : b, lo = a > b ? b : a;
        const uint32_t old = atomicCAS(par + hi, hi, lo);
        if (old == hi) return true;
        a = old;  // hi was hooked by another thread meanwhile: continue from there
        b = lo;
    }
    return false;
}

// Key of every particle (particle order) and its rank in its row from an
// integer counter.
template <int R>
__global__ void __launch_bounds__(FOF_T) k_fof_keys(const double *__restrict__ X, size_t n, FofGrid g,
                                                    uint64_t *__restrict__ keys, uint32_t *__restrict__ slot,
                                                    uint32_t *__restrict__ rowcount) {
    const size_t i = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    if (i >= n) return;
    double x[3];
#pragma unroll
    for (int k = 0; k < R; ++k) x[k] = X[i * R + k];
    uint32_t row;
    keys[i] = fof_key<R>(x, g, &row);
    slot[i] = atomicAdd(rowcount + row, 1u);
}

// Counting sort by row: every particle's sort value -- quantised x above the
// particle index (unique, and the order a stable sort by key from particle
// order would give) -- at its row's offset plus its rank. One scattered
// 8-byte store per particle; the row sorts put the order inside a row right and
// write the keys and indices out.
__global__ void __launch_bounds__(FOF_T) k_fof_place(const uint64_t *__restrict__ kp, const uint32_t *__restrict__ slot,
                                                     const uint32_t *__restrict__ rowoff, size_t n,
                                                     uint64_t *__restrict__ val) {
    const size_t i = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    if (i >= n) return;
    const uint64_t key = kp[i];
    val[(size_t)rowoff[key >> FOF_XB] + slot[i]] = ((key & FOF_XMASK) << 32) | (uint64_t)i;
}

constexpr int FOF_BIG = 4096;                    // longest row sorted in shared memory
constexpr int FOF_WARP_ROW = FOF_BIG / (256 / 32);  // longest row one warp sorts in its share of it

// One compare-exchange step of a bitonic network across the lanes.
__device__ inline uint64_t fof_exchange(uint64_t v, int j, int k) {
    const int lane = threadIdx.x & 31;
    const uint64_t o = __shfl_xor_sync(FULL, v, j);
    const bool keep_min = ((lane & j) == 0) == ((lane & k) == 0);
    return keep_min ? (v < o ? v : o) : (v > o ? v : o);
}

// Sort values in, keys and particle indices out (keys in place). One warp per
// four rows: four rows of up to 8 particles are sorted at once, one per
// quarter of the warp, else each of up to 32 across the lanes; longer rows are
// queued for k_fof_rowsort_big (up to FOF_BIG) or flagged in nbig[1]
// (longer). One row per warp and step before, with three dependent loads each
// and 25 of 32 lanes idle on 7 particles per row: 256 -> 145 us for 0.83
// million rows.
__global__ void __launch_bounds__(256) k_fof_rowsort_small(uint64_t *__restrict__ keys, uint32_t *__restrict__ order,
                                                           const uint32_t *__restrict__ rowoff, size_t rows,
                                                           uint32_t *__restrict__ big, uint32_t *__restrict__ nbig) {
    const int lane = threadIdx.x & 31;
    const size_t nw = (size_t)gridDim.x * (256 / 32);
    for (size_t r0 = 4 * (((size_t)blockIdx.x * 256 + threadIdx.x) >> 5); r0 < rows; r0 += 4 * nw) {
        const size_t ro = r0 + lane < rows ? r0 + lane : rows;  // rows beyond the last are empty
        const uint32_t off = lane < 5 ? rowoff[ro] : 0u;
        const uint32_t qs = __shfl_sync(FULL, off, lane >> 3), qm = __shfl_sync(FULL, off, (lane >> 3) + 1) - qs;
        if (__all_sync(FULL, qm <= 8)) {
            const uint32_t l = lane & 7;
            uint64_t v = l < qm ? keys[qs + l] : ~0ull;
#pragma unroll
            for (int k = 2; k <= 8; k <<= 1)
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) v = fof_exchange(v, j, k == 8 ? 32 : k);
            if (l < qm) {
                keys[qs + l] = ((uint64_t)(r0 + (lane >> 3)) << FOF_XB) | (v >> 32);
                order[qs + l] = (uint32_t)v;
            }
            continue;
        }
        for (int q = 0; q < 4; ++q) {
            const uint32_t rs = __shfl_sync(FULL, off, q), m = __shfl_sync(FULL, off, q + 1) - rs;
            const size_t r = r0 + q;
            if (m > 32) {
                if (lane == 0) {
                    if (m > (uint32_t)FOF_BIG) atomicOr(nbig + 1, 1u);
                    else big[atomicAdd(nbig, 1u)] = (uint32_t)r;
                }
                continue;
            }
            uint64_t v = (uint32_t)lane < m ? keys[rs + lane] : ~0ull;
            if (m > 1) {
#pragma unroll
                for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
                    for (int j = k >> 1; j > 0; j >>= 1) v = fof_exchange(v, j, k);
            }
            if ((uint32_t)lane < m) {
                keys[rs + lane] = ((uint64_t)r << FOF_XB) | (v >> 32);
                order[rs + lane] = (uint32_t)v;
            }
        }
    }
}

// Bitonic sort of m values of row r (at rs) in shared memory over the next
// power of two, padded with the largest value, by `T` threads of index x0.
template <int T, typename Sync>
__device__ inline void fof_rowsort(uint64_t *sv, uint64_t *keys, uint32_t *order, uint32_t r, uint32_t rs, uint32_t m,
                                   uint32_t x0, Sync sync) {
    uint32_t P = 64;
    while (P < m) P <<= 1;
    for (uint32_t j = x0; j < P; j += T) sv[j] = j < m ? keys[rs + j] : ~0ull;
    sync();
    for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t h = x0; h < P / 2; h += T) {  // pair (x, x + j), bit j of x clear
                const uint32_t x = ((h & ~(j - 1)) << 1) | (h & (j - 1)), y = x + j;
                const uint64_t a = sv[x], c = sv[y];
                if ((a > c) == ((x & k) == 0)) {
                    sv[x] = c;
                    sv[y] = a;
                }
            }
            sync();
        }
    }
    for (uint32_t j = x0; j < m; j += T) {
        const uint64_t v = sv[j];
        keys[rs + j] = ((uint64_t)r << FOF_XB) | (v >> 32);
        order[rs + j] = (uint32_t)v;
    }
    sync();
}

// The queued rows (33 .. FOF_BIG particles): those of up to FOF_WARP_ROW by
// one warp each in its share of the shared memory (no block barriers), the
// rest by one CTA each (146 -> 61 us for the whole queue).
__global__ void __launch_bounds__(256) k_fof_rowsort_big(uint64_t *__restrict__ keys, uint32_t *__restrict__ order,
                                                         const uint32_t *__restrict__ rowoff,
                                                         const uint32_t *__restrict__ big,
                                                         const uint32_t *__restrict__ nbig) {
    __shared__ uint64_t sv[FOF_BIG];
    const uint32_t nq = nbig[0], w = threadIdx.x >> 5;
    for (uint32_t b = blockIdx.x * 8 + w; b < nq; b += gridDim.x * 8) {
        const uint32_t r = big[b], rs = rowoff[r], m = rowoff[r + 1] - rs;
        if (m <= (uint32_t)FOF_WARP_ROW)
            fof_rowsort<32>(sv + w * FOF_WARP_ROW, keys, order, r, rs, m, threadIdx.x & 31, [] { __syncwarp(); });
    }
    __syncthreads();
    for (uint32_t b = blockIdx.x; b < nq; b += gridDim.x) {
        const uint32_t r = big[b], rs = rowoff[r], m = rowoff[r + 1] - rs;
        if (m > (uint32_t)FOF_WARP_ROW)
            fof_rowsort<256>(sv, keys, order, r, rs, m, threadIdx.x, [] { __syncthreads(); });
    }
}

__global__ void __launch_bounds__(FOF_T) k_fof_iota(uint32_t *__restrict__ v, size_t n) {
    const size_t i = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    if (i < n) v[i] = (uint32_t)i;
}

template <int R>
__global__ void __launch_bounds__(FOF_T) k_fof_gather(const double *__restrict__ X, size_t n,
                                                      const uint32_t *__restrict__ order, double *__restrict__ S,
                                                      uint32_t *__restrict__ par) {
    const size_t t = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    if (t >= n) return;
    const uint32_t i = order[t];
#pragma unroll
    for (int k = 0; k < R; ++k) S[(size_t)k * n + t] = X[(size_t)i * R + k];
    par[t] = (uint32_t)t;  // every sorted position its own parent
}

struct FofLink {
    const double *S;
    const uint64_t *keys;
    const uint32_t *rowoff;
    size_t n;
    FofGrid g;
    uint32_t *par;
    int *err;
};

// First sorted position in [lo, hi) whose key is >= k.
__device__ inline uint32_t fof_lower(const uint64_t *__restrict__ keys, uint32_t lo, uint32_t hi, uint64_t k) {
    while (lo < hi) {
        const uint32_t mid = lo + ((hi - lo) >> 1);
        if (__ldg(keys + mid) < k) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Candidates of one particle in one row: sorted positions [b0, b0 + n0) and,
// where the x window wraps around the box, [b1, b1 + n1).
struct FofRange {
    uint32_t b0, n0, b1, n1;
};

// The positions of row [rs, re) (row key rk) whose quantised x lies in [qa, qb].
__device__ inline void fof_segment(const FofLink &a, uint32_t rs, uint32_t re, uint64_t rk, long long qa, long long qb,
                                   uint32_t *b, uint32_t *n) {
    *b = fof_lower(a.keys, rs, re, rk | (uint64_t)qa);
    *n = fof_lower(a.keys, *b, re, (rk | (uint64_t)qb) + 1) - *b;
}

// Tests every candidate of the warp's 32 particles (lane l: particle t0 + l
// with range r, coordinates in shared memory) and joins the linked pairs. The
// candidates of all lanes form one list that the lanes take in turn, 32 at a
// time, so that a particle in a dense row does not leave the others waiting.
template <int R, bool LONG>
__device__ inline void fof_test_all(const FofLink &a, const double (*sx)[32], uint32_t t0, const FofRange &r) {
    const int lane = threadIdx.x & 31;
    const uint32_t cnt = r.n0 + r.n1;
    auto test = [&](int o, uint32_t u) {  // particle t0 + o against sorted position u
        if (__ldcg(a.par + t0 + o) == __ldcg(a.par + u)) return;  // in one tree already
        double xi[3], xj[3];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            xi[q] = sx[q][o];
            xj[q] = __ldg(a.S + (size_t)q * a.n + u);
        }
        if (fof_linked<R>(xi, xj, a.g) && !fof_unite(a.par, t0 + o, u)) atomicOr(a.err, 1);
    };
    // the shared list is counted in 32 bits; LONG: rows of over FOF_BIG
    // particles exist, so a list may be too long for that
    if (LONG && __any_sync(FULL, cnt >= (1u << 26))) {
        for (uint32_t k = 0; k < cnt; ++k) test(lane, k < r.n0 ? r.b0 + k : r.b1 + (k - r.n0));
        return;
    }
    uint32_t inc = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, inc, o);
        if (lane >= o) inc += v;
    }
    const uint32_t total = __shfl_sync(FULL, inc, 31), pre = inc - cnt;
    const bool wraps = __any_sync(FULL, r.n1 != 0);
    for (uint32_t c = 0; c < total; c += 32) {
        const uint32_t k = c + lane;
        // owner: the last lane whose list starts at or before item k
        int o = 0;
#pragma unroll
        for (int st = 16; st > 0; st >>= 1)
            if (__shfl_sync(FULL, pre, o + st) <= k) o += st;
        const uint32_t off = k - __shfl_sync(FULL, pre, o);
        uint32_t u = __shfl_sync(FULL, r.b0, o) + off;
        if (wraps) {
            const uint32_t n0 = __shfl_sync(FULL, r.n0, o), b1 = __shfl_sync(FULL, r.b1, o);
            if (off >= n0) u = b1 + (off - n0);
        }
        if (k < total) test(o, u);
    }
}

// One warp links 32 particles that follow each other in sorted order. Before
// the candidates were shared among the lanes (fof_test_all), every lane
// walked its own: 3 of 32 lanes were active per instruction on a clustered
// set (half of 6 million particles in halos), 3.9 ms against 1.0 now. Half of
// the pairs share a parent already and need no distance (1.11 ms without that
// check).
template <int R, bool LONG>
__global__ void __launch_bounds__(FOF_T) k_fof_link(FofLink a) {
    __shared__ double sxs[FOF_T / 32][R][32];
    const uint32_t t = blockIdx.x * FOF_T + threadIdx.x;  // n < 2^32 - 1
    const int lane = threadIdx.x & 31;
    double(*sx)[32] = sxs[threadIdx.x >> 5];
    const uint32_t t0 = t - lane;
    const bool act = t < a.n;
    uint64_t key = 0;
    if (act) {
#pragma unroll
        for (int k = 0; k < R; ++k) sx[k][lane] = a.S[(size_t)k * a.n + t];
        key = a.keys[t];
    }
    __syncwarp();
    const uint32_t row = (uint32_t)(key >> FOF_XB);
    const long long xq = (long long)(key & FOF_XMASK), N = FOF_XN;
    const long long lo = xq - a.g.wq, hi = xq + a.g.wq;
    const bool whole = 2 * (long long)a.g.wq + 1 >= N;
    // own row: the particles ahead of t in cyclic x order, up to wq ahead
    FofRange r{0, 0, 0, 0};
    if (act) {
        const uint32_t rs = a.rowoff[row], re = a.rowoff[row + 1];
        const uint64_t rk = (uint64_t)row << FOF_XB;
        r.b0 = t + 1;
        if (whole) {
            r.n0 = re - r.b0;
        } else {
            r.n0 = fof_lower(a.keys, t + 1, re, (rk | (uint64_t)(hi < N ? hi : N - 1)) + 1) - r.b0;
            if (hi >= N) {
                r.b1 = rs;
                r.n1 = fof_lower(a.keys, rs, t, (rk | (uint64_t)(hi - N)) + 1) - rs;
            }
        }
    }
    fof_test_all<R, LONG>(a, sx, t0, r);
    if (a.g.nr == 1) return;
    // the forward half of the neighbouring rows: y + 1 (2D); (y+-1, z+1),
    // (y, z+1), (y+1, z) (3D)
    const int nr = a.g.nr;
    const int cy = (int)(row % (uint32_t)nr), cz = R == 3 ? (int)(row / (uint32_t)nr) : 0;
    constexpr int NF = R == 2 ? 1 : 4;
    const int dy[4] = {1, -1, 0, 1}, dz[4] = {0, 1, 1, 1};
#pragma unroll 1
    for (int f = 0; f < NF; ++f) {
        int y = cy + dy[f], z = cz + dz[f];
        y = y < 0 ? y + nr : (y >= nr ? y - nr : y);
        z = z >= nr ? z - nr : z;
        const uint32_t nrow = R == 2 ? (uint32_t)y : (uint32_t)z * (uint32_t)nr + (uint32_t)y;
        r = FofRange{0, 0, 0, 0};
        if (act) {
            const uint32_t rs = a.rowoff[nrow], re = a.rowoff[nrow + 1];
            const uint64_t rk = (uint64_t)nrow << FOF_XB;
            if (rs == re) {
            } else if (whole) {
                r.b0 = rs;
                r.n0 = re - rs;
            } else if (lo < 0) {
                fof_segment(a, rs, re, rk, lo + N, N - 1, &r.b0, &r.n0);
                fof_segment(a, rs, re, rk, 0, hi, &r.b1, &r.n1);
            } else if (hi >= N) {
                fof_segment(a, rs, re, rk, lo, N - 1, &r.b0, &r.n0);
                fof_segment(a, rs, re, rk, 0, hi - N, &r.b1, &r.n1);
            } else {
                fof_segment(a, rs, re, rk, lo, hi, &r.b0, &r.n0);
            }
        }
        fof_test_all<R, LONG>(a, sx, t0, r);
    }
}

// Every sorted position's root into a separate array, and the lowest particle
// index of every tree into low[root]. The walk only reads the parents: a
// path-halving store in this pass could overwrite a root another thread has
// just written with an older ancestor. Lanes with the same root (neighbours
// in a halo) send one minimum.
__global__ void __launch_bounds__(FOF_T) k_fof_roots(const uint32_t *__restrict__ par,
                                                     const uint32_t *__restrict__ order, size_t n,
                                                     uint32_t *__restrict__ root, uint32_t *__restrict__ low) {
    const size_t t = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    const unsigned lanes = __ballot_sync(FULL, t < n);
    if (t >= n) return;
    uint32_t r = (uint32_t)t, p = par[r];
    while (p != r) {
        r = p;
        p = par[r];
    }
    root[t] = r;
    const unsigned same = __match_any_sync(lanes, r);
    const uint32_t mn = __reduce_min_sync(same, order[t]);
    if ((int)(threadIdx.x & 31) == __ffs(same) - 1) atomicMin(low + r, mn);
}

// flag = 1 for the lowest particle of every tree (cleared before).
__global__ void __launch_bounds__(FOF_T) k_fof_leaders(const uint32_t *__restrict__ root,
                                                       const uint32_t *__restrict__ low, size_t n,
                                                       uint32_t *__restrict__ flag) {
    const size_t t = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    if (t < n && root[t] == (uint32_t)t) flag[low[t]] = 1u;
}

__global__ void __launch_bounds__(FOF_T) k_fof_tags(const uint32_t *__restrict__ root,
                                                    const uint32_t *__restrict__ low,
                                                    const uint32_t *__restrict__ gnum,
                                                    const uint32_t *__restrict__ order, size_t n,
                                                    unsigned long long *__restrict__ tags) {
    const size_t t = (size_t)blockIdx.x * FOF_T + threadIdx.x;
    if (t >= n) return;
    tags[order[t]] = (unsigned long long)gnum[low[root[t]]] + 1ull;
}

inline unsigned blocks(size_t n) { return (unsigned)((n + FOF_T - 1) / FOF_T); }

}  // namespace

// Grid and device buffers of one problem size; reused across runs.
struct FofEngine {
    int R = 3, device = 0, key_bits = 0;
    size_t n = 0, rows = 0;
    FofGrid g{};
    cudaStream_t st = nullptr;
    double *X = nullptr, *S = nullptr;
    uint64_t *keys[2] = {nullptr, nullptr};
    uint32_t *vals[2] = {nullptr, nullptr};
    uint32_t *par = nullptr, *rowcount = nullptr, *rowoff = nullptr, *flag = nullptr, *gnum = nullptr,
             *bh = nullptr, *boff = nullptr, *bsum = nullptr, *bigrows = nullptr, *nbig = nullptr;
    unsigned long long *tags = nullptr;
    uint32_t *ngroups_h = nullptr, *nbig_h = nullptr;  // pinned
    int *err = nullptr;
    int sort_blocks = 0;
    bool used_radix = false;  // the last run's rows were too long for the row sorts

    ~FofEngine() {
        if (st) cudaStreamSynchronize(st);
        for (void *q : {(void *)X, (void *)S, (void *)keys[0], (void *)keys[1], (void *)vals[0], (void *)vals[1],
                        (void *)par, (void *)rowcount, (void *)rowoff, (void *)flag, (void *)gnum, (void *)bh,
                        (void *)boff, (void *)bsum, (void *)tags, (void *)err, (void *)bigrows, (void *)nbig})
            cudaFree(q);
        cudaFreeHost(ngroups_h);
        cudaFreeHost(nbig_h);
        if (st) cudaStreamDestroy(st);
    }

    int init(const conan_fof_params &p) {
        R = p.dim;
        device = p.device;
        n = (size_t)p.n_particles;
        // transverse cells no smaller than the linking length (with a margin
        // far above the rounding of the wrap), at most about eight rows per
        // particle
        const double q = p.size / (p.linking_length * (1.0 + 1e-9));
        long long nr = q >= 2147483647.0 ? 2147483647LL : (long long)q;
        long long cap = 1;
        while (true) {
            long long c1 = cap + 1, v = 1;
            for (int k = 1; k < R; ++k) v *= c1;
            if (v > 8 * (long long)std::max<size_t>(n, 27) || v > (1LL << 26)) break;
            cap = c1;
        }
        nr = std::min(nr, cap);
        if (nr < 3) nr = 1;
        g.nr = (int)nr;
        g.L = p.size;
        g.half = p.size / 2;
        g.inv_h = (double)nr / p.size;
        g.xscale = (double)FOF_XN / p.size;
        g.rsqr = p.linking_length * p.linking_length;
        const double wq = std::ceil(p.linking_length * g.xscale) + 2.0;
        g.wq = wq >= (double)FOF_XN ? (int)FOF_XN : (int)wq;
        rows = 1;
        for (int k = 1; k < R; ++k) rows *= (size_t)nr;
        int rb = 0;
        while (((size_t)1 << rb) < rows) ++rb;
        key_bits = FOF_XB + rb;
        const size_t tiles = radix_tiles(n), m = 256 * tiles;
        const size_t nb = (std::max(std::max(m, rows), n) + SCAN_CHUNK - 1) / SCAN_CHUNK;
        CONAN_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
        CONAN_CUDA(device_alloc(&X, n * R * sizeof(double)));
        CONAN_CUDA(device_alloc(&S, n * R * sizeof(double)));
        for (int b = 0; b < 2; ++b) {
            CONAN_CUDA(device_alloc(&keys[b], n * sizeof(uint64_t)));
            CONAN_CUDA(device_alloc(&vals[b], n * sizeof(uint32_t)));
        }
        CONAN_CUDA(device_alloc(&par, n * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&flag, n * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&gnum, (n + 1) * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&rowcount, rows * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&rowoff, (rows + 1) * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&bh, m * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&boff, (m + 1) * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&bsum, nb * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&tags, n * sizeof(unsigned long long)));
        CONAN_CUDA(device_alloc(&err, sizeof(int)));
        CONAN_CUDA(cudaMallocHost(&ngroups_h, 2 * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&bigrows, std::min(rows, n / 33 + 1) * sizeof(uint32_t)));
        CONAN_CUDA(device_alloc(&nbig, 2 * sizeof(uint32_t)));
        CONAN_CUDA(cudaMallocHost(&nbig_h, 2 * sizeof(uint32_t)));
        int sms = 0;
        CONAN_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
        sort_blocks = 8 * sms;
        CONAN_CUDA(cudaFuncSetAttribute(k_rs_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RS_SMEM));
        CONAN_CUDA(cudaMemsetAsync(rowcount, 0, rows * sizeof(uint32_t), st));
        CONAN_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }

    void scan(uint32_t *cnt, size_t m, uint32_t *out, cudaStream_t s) { scan_exclusive(cnt, m, bsum, out, s); }

    // Groups of the positions in Xd (device, n x R doubles); tags into tg
    // (device, n values). Enqueued on `s`; the group count is read back.
    template <int RR> int run_t(const double *Xd, unsigned long long *tg, cudaStream_t s, uint64_t *ngroups) {
        // per-particle keys into keys[1], ranks in the rows into `flag`
        k_fof_keys<RR><<<blocks(n), FOF_T, 0, s>>>(Xd, n, g, keys[1], flag, rowcount);
        scan(rowcount, rows, rowoff, s);  // also clears the counts for the next run
        // counting sort by row, then every row sorted by (x, index)
        CONAN_CUDA(cudaMemsetAsync(nbig, 0, 2 * sizeof(uint32_t), s));
        k_fof_place<<<blocks(n), FOF_T, 0, s>>>(keys[1], flag, rowoff, n, keys[0]);
        k_fof_rowsort_small<<<(unsigned)sort_blocks, 256, 0, s>>>(keys[0], vals[0], rowoff, rows, bigrows, nbig);
        k_fof_rowsort_big<<<(unsigned)sort_blocks, 256, 0, s>>>(keys[0], vals[0], rowoff, bigrows, nbig);
        CONAN_CUDA(cudaMemcpyAsync(nbig_h, nbig, 2 * sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        CONAN_CUDA(cudaStreamSynchronize(s));
        uint64_t *sk = keys[0];
        uint32_t *order = vals[0], *root = vals[1];
        used_radix = nbig_h[1] != 0;
        if (used_radix) {
            // a row longer than FOF_BIG: radix sort of (key, index) from particle order instead
            k_fof_iota<<<blocks(n), FOF_T, 0, s>>>(vals[1], n);
            uint64_t *kk[2] = {keys[1], keys[0]};
            uint32_t *vv[2] = {vals[1], vals[0]};
            const int w = radix_sort_pairs(kk, vv, n, key_bits, bh, boff, bsum, s);
            sk = kk[w];
            order = vv[w];
            root = vv[w ^ 1];
        }
        k_fof_gather<RR><<<blocks(n), FOF_T, 0, s>>>(Xd, n, order, S, par);
        FofLink a{S, sk, rowoff, n, g, par, err};
        if (used_radix) k_fof_link<RR, true><<<blocks(n), FOF_T, 0, s>>>(a);
        else k_fof_link<RR, false><<<blocks(n), FOF_T, 0, s>>>(a);
        // roots into the free value buffer, the trees' lowest particles into
        // the free key buffer, leader flags and group numbers by particle
        uint32_t *low = reinterpret_cast<uint32_t *>(sk == keys[0] ? keys[1] : keys[0]);
        CONAN_CUDA(cudaMemsetAsync(low, 0xff, n * sizeof(uint32_t), s));
        CONAN_CUDA(cudaMemsetAsync(flag, 0, n * sizeof(uint32_t), s));
        k_fof_roots<<<blocks(n), FOF_T, 0, s>>>(par, order, n, root, low);
        k_fof_leaders<<<blocks(n), FOF_T, 0, s>>>(root, low, n, flag);
        scan(flag, n, gnum, s);
        k_fof_tags<<<blocks(n), FOF_T, 0, s>>>(root, low, gnum, order, n, tg);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            return set_error(CONAN_ERR_CUDA, "fof kernel launch failed: %s", cudaGetErrorString(e));
        int herr = 0;
        CONAN_CUDA(cudaMemcpyAsync(ngroups_h, gnum + n, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
        CONAN_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, s));
        CONAN_CUDA(cudaMemsetAsync(err, 0, sizeof(int), s));
        CONAN_CUDA(cudaStreamSynchronize(s));
        if (herr)
            return set_error(CONAN_ERR_STATE, "fof: a union did not finish within %d retries", FOF_UNITE_LIMIT);
        if (ngroups) *ngroups = ngroups_h[0];
        return CONAN_OK;
    }

    int run_device(const double *Xd, unsigned long long *tg, cudaStream_t s, uint64_t *ngroups) {
        return R == 2 ? run_t<2>(Xd, tg, s, ngroups) : run_t<3>(Xd, tg, s, ngroups);
    }

    int run_host(const double *Xh, unsigned long long *tg_h, uint64_t *ngroups) {
        CONAN_TRY(copy_to_device(X, Xh, n * R * sizeof(double), st));
        CONAN_TRY(run_device(X, tags, st, ngroups));
        CONAN_TRY(copy_to_host(tg_h, tags, n * sizeof(unsigned long long), st));
        CONAN_CUDA(cudaStreamSynchronize(st));
        return CONAN_OK;
    }
};

int check_fof_params(const conan_fof_params *p) {
    if (!p) return set_error(CONAN_ERR_ARG, "null parameters");
    if (p->dim != 2 && p->dim != 3) return set_error(CONAN_ERR_UNSUPPORTED, "fof: dim = %d (2 or 3)", p->dim);
    if (p->n_particles < 1 || p->n_particles >= (1ULL << 32) - 1)
        return set_error(CONAN_ERR_ARG, "fof: particle count %llu outside 1 .. 2^32 - 2", p->n_particles);
    if (!(p->size > 0) || !std::isfinite(p->size)) return set_error(CONAN_ERR_ARG, "fof: box size must be positive");
    if (!(p->linking_length > 0) || !std::isfinite(p->linking_length))
        return set_error(CONAN_ERR_ARG, "fof: linking length must be positive");
    return CONAN_OK;
}

}  // namespace conan

using namespace conan;

struct conan_fof_engine {
    FofEngine e;
};

extern "C" conan_fof_engine *conan_fof_create(const conan_fof_params *p) {
    if (check_fof_params(p) != CONAN_OK) return nullptr;
    if (device_guard(p->device) != CONAN_OK) return nullptr;
    conan_fof_engine *h = new conan_fof_engine;
    if (h->e.init(*p) != CONAN_OK) {
        std::string msg = last_error();
        delete h;
        set_error(CONAN_ERR_ALLOC, "%s", msg.c_str());
        return nullptr;
    }
    return h;
}

extern "C" void conan_fof_destroy(conan_fof_engine *h) {
    if (!h) return;
    cudaSetDevice(h->e.device);
    delete h;
}

extern "C" int conan_fof_run(conan_fof_engine *h, const double *X, unsigned long long *tags, unsigned long long *n_groups) {
    if (!h) return set_error(CONAN_ERR_ARG, "null fof handle");
    if (!X || !tags) return set_error(CONAN_ERR_ARG, "fof: null positions or tags");
    CONAN_TRY(device_guard(h->e.device));
    uint64_t ng = 0;
    CONAN_TRY(h->e.run_host(X, tags, &ng));
    if (n_groups) *n_groups = ng;
    return CONAN_OK;
}

extern "C" int conan_fof_run_device(conan_fof_engine *h, const double *X, unsigned long long *tags,
                                    unsigned long long *n_groups, void *stream) {
    if (!h) return set_error(CONAN_ERR_ARG, "null fof handle");
    if (!X || !tags) return set_error(CONAN_ERR_ARG, "fof: null positions or tags");
    CONAN_TRY(device_guard(h->e.device));
    uint64_t ng = 0;
    CONAN_TRY(h->e.run_device(X, tags, (cudaStream_t)stream, &ng));
    if (n_groups) *n_groups = ng;
    return CONAN_OK;
}

extern "C" int conan_fof(const conan_fof_params *p, const double *X, unsigned long long *tags,
                         unsigned long long *n_groups) {
    CONAN_TRY(check_fof_params(p));
    if (!X || !tags) return set_error(CONAN_ERR_ARG, "fof: null positions or tags");
    conan_fof_engine *h = conan_fof_create(p);
    if (!h) return CONAN_ERR_ALLOC;
    int rc = conan_fof_run(h, X, tags, n_groups);
    conan_fof_destroy(h);
    return rc;
}
