// LQ preconditioning of the sector SVDs: W <- W Q, rot <- Q with W Q lower trapezoidal on
// its rows in order of falling norm, so that the one-sided Jacobi that follows runs on the
// columns of a triangular factor whose rows are graded.
//
// One-sided Jacobi converges slowly on the matrices a DMRG truncation decomposes (rows and
// columns graded over 8 to 14 decades): 15 to 30 sweeps.  On the columns of L -- the rows of R
// in A^T P = Q R, with the rows of A sorted by norm -- it needs about 7 whatever the grading (Drmac
// and Veselic's preconditioning, SIAM J. Matrix Anal. Appl. 29 (2008), with one sorted instead of a
// pivoted factorisation; unsorted it gains nothing).  Q is a product of Householder reflections, each
// orthogonal to working precision at any magnitude of its row (scale_row), and any orthogonal start gives an exact SVD: the factorisation decides the speed alone.
//
// All sectors go through one cooperative launch in panels of NB = 8 reflections.  The vectors
// (the p rows of W and the q rows of the identity, q long, contiguous in X) are independent under
// a panel's block reflection x <- x - V T^T (V^T x), one warp each; the next panel's eight rows go
// first, on the CTA that owns the sector, which factors them (a warp per row) while the other CTAs
// apply the current panel to the rest.  So a panel costs one grid barrier, and the chain of a
// panel's eight reflections is hidden behind the update where that is the longer of the two.
// Work is 10/3 q^3 + 4 (p - q) q^2 FLOP per sector, a third to a half of one Jacobi sweep.
#include <cooperative_groups.h>

#include <atomic>

#include "kernels.h"
#include "qtt_core.h"

namespace cg = cooperative_groups;

namespace qtt {
namespace {
constexpr int NB = 8, LT = 256;  // reflections per panel, threads per CTA (a warp per reflection)

template <class T>
struct LqParams {
    T *x;             // vectors
    T *v;             // per sector 2 x (NB x q + NB x NB): reflectors and T, by panel parity
    const LqSec *secs;
    const int *order;  // rows of W by falling norm
    int *next;         // per panel: update items claimed (zero on entry)
    const int *np;     // panels of each sector (0: left as it is), then the most of any
    int nsec, chunk, max_q;
};

__device__ __forceinline__ double lsum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float lsum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ __forceinline__ int panels_of(int q) { return (q - 1 + NB - 1) / NB; }

// Eight per-lane sums reduced over the warp in nine additions: lane l gets the total of number
// 4 (l >> 4) + 2 (l >> 3 & 1) + (l >> 2 & 1).
template <class T>
__device__ __forceinline__ T sum8(T (&a)[NB], int lane) {
    const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const T send = h4 ? a[i] : a[i + 4], keep = h4 ? a[i + 4] : a[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const T send = h3 ? a[i] : a[i + 2], keep = h3 ? a[i + 2] : a[i];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
    const T send = h2 ? a[0] : a[1], keep = h2 ? a[1] : a[0];
    T s = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}
__device__ __forceinline__ int lane_of(int c) { return (c & 4) << 2 | (c & 2) << 2 | (c & 1) << 2; }

// x <- x - V T^T (V^T x) on x[0 .. len), one warp: V (NB x len) and T (NB x NB, row-major) in
// shared memory.
template <class T>
__device__ __forceinline__ void apply_panel(T *x, const T *V, const T *Tm, int len, int lane) {
    T a[NB];
#pragma unroll
    for (int c = 0; c < NB; ++c) a[c] = T(0);
    for (int k = lane; k < len; k += 32) {
        const T y = x[k];
#pragma unroll
        for (int c = 0; c < NB; ++c) a[c] = fma(V[c * len + k], y, a[c]);
    }
    const T d = sum8(a, lane);
    // w = T^T d on the lanes of component c
    const int c = (lane >> 4) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
    T w = T(0);
#pragma unroll
    for (int i = 0; i < NB; ++i) w = fma(Tm[i * NB + c], __shfl_sync(0xffffffffu, d, lane_of(i)), w);
    T wv[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) wv[i] = __shfl_sync(0xffffffffu, w, lane_of(i));
    for (int k = lane; k < len; k += 32) {
        T y = x[k];
#pragma unroll
        for (int i = 0; i < NB; ++i) y = fma(-V[i * len + k], wv[i], y);
        x[k] = y;
    }
}

// The exact powers of two that bring a row's largest |x| to about 1 and back (scale_row: false where there
// is nothing to reflect by: zeros, an infinity or a NaN).  Sums of squares of the row as it is leave the work type's
// range long before its elements do -- FP32 elements of 1e-20 have subnormal squares -- and a reflection from an inexact
// sum is not orthogonal.
__device__ __forceinline__ bool scale_row(const float *x, int first, int len, int lane, float &up, float &down) {
    uint32_t m = 0;
    for (int k = first + lane; k < len; k += 32) m = max(m, __float_as_uint(x[k]) & 0x7FFFFFFFu);
    m = __reduce_max_sync(0xffffffffu, m);
    const uint32_t f = 253u - min(m >> 23, 252u);
    up = __uint_as_float(f << 23);
    down = __uint_as_float((254u - f) << 23);
    return m != 0 && m < 0x7F800000u;
}
__device__ __forceinline__ bool scale_row(const double *x, int first, int len, int lane, double &up, double &down) {
    uint32_t m = 0;  // by the high words
    for (int k = first + lane; k < len; k += 32) m = max(m, uint32_t(__double2hiint(x[k])) & 0x7FFFFFFFu);
    m = __reduce_max_sync(0xffffffffu, m);
    const uint32_t f = 2045u - min(m >> 20, 2044u);
    up = __hiloint2double(int(f << 20), 0);
    down = __hiloint2double(int((2046u - f) << 20), 0);
    return m != 0 && m < 0x7FF00000u;
}

// Whether a sum of squares lost nothing to the ends of the work type's range (false with a NaN): squares that do are
// at least 2^-60 times smaller than the sum.  Scaling every row took svd D = 600 from 10.80 to 10.93 ms.
__device__ __forceinline__ bool squares_fit(float total) { return total >= 0x1p-80f && total <= 0x1p+120f; }
__device__ __forceinline__ bool squares_fit(double total) { return total >= 0x1p-900 && total <= 0x1p+1000; }

// Factors the NB rows held in xs (`pitch` apart, len long; nr of them exist): row c's reflection
// zeroes its elements beyond c.  vs receives the reflectors (zero before their
// first element), Tm the triangular factor.  All 8 warps of the CTA, one per row.
template <class T>
__device__ void factor_panel(T *xs, int pitch, T *vs, T *Tm, T *gram, T *tau, int len, int nr, int warp, int lane) {
    for (int c = 0; c < NB; ++c) {
        T *v = vs + c * len;
        if (warp == c) {
            T *x = xs + c * pitch;
            T s = T(0), up = T(1), down = T(1);
            bool real = c < nr && c + 1 < len;
            if (real)
                for (int k = c + 1 + lane; k < len; k += 32) s = fma(x[k], x[k], s);
            s = lsum(s);
            if (real && !squares_fit(fma(x[c], x[c], s))) {
                real = scale_row(x, c, len, lane, up, down);
                s = T(0);
                if (real)
                    for (int k = c + 1 + lane; k < len; k += 32) s = fma(x[k] * up, x[k] * up, s);
                s = lsum(s);
            }
            T t = T(0), scale = T(0), beta = T(0);
            if (real && s > T(0)) {
                const T alpha = x[c] * up;
                beta = -copysign(sqrt(fma(alpha, alpha, s)), alpha);
                t = (beta - alpha) / beta;
                scale = T(1) / (alpha - beta);
                beta *= down;
            }
            for (int k = lane; k < len; k += 32) {
                const T y = t != T(0) && k > c ? x[k] * up * scale : (k == c && t != T(0) ? T(1) : T(0));
                v[k] = y;
                if (t != T(0)) {
                    if (k == c) x[k] = beta;
                    if (k > c) x[k] = T(0);
                }
            }
            if (lane == 0) tau[c] = t;
        }
        __syncthreads();
        const T t = tau[c];
        if (warp > c) {
            if (t != T(0) && warp < nr) {
                T *x = xs + warp * pitch;
                T d = T(0);
                for (int k = c + lane; k < len; k += 32) d = fma(v[k], x[k], d);
                d = lsum(d) * t;
                for (int k = c + lane; k < len; k += 32) x[k] = fma(-d, v[k], x[k]);
            }
        } else if (warp < c) {
            const T *u = vs + warp * len;
            T d = T(0);
            for (int k = c + lane; k < len; k += 32) d = fma(u[k], v[k], d);
            d = lsum(d);
            if (lane == 0) gram[warp * NB + c] = d;
        }
        __syncwarp();
    }
    __syncthreads();
    // T = [T', -tau T' (V'^T v); 0, tau], column by column; thread i holds row i
    if (threadIdx.x < NB) {
        const int i = threadIdx.x;
        T row[NB];
        for (int c = 0; c < NB; ++c) {
            T acc = T(0);
            for (int l = i; l < c; ++l) acc = fma(row[l], gram[l * NB + c], acc);
            row[c] = c < i ? T(0) : (c == i ? tau[c] : -tau[c] * acc);
            Tm[i * NB + c] = row[c];
        }
    }
    __syncthreads();
}

template <class T>
__global__ void __launch_bounds__(LT) k_lq(LqParams<T> P) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ __align__(16) unsigned char lsh[];
    T *buf = reinterpret_cast<T *>(lsh);       // NB x max_q: rows of a panel, or a vector per warp
    T *vs = buf + NB * P.max_q;                // NB x max_q reflectors
    T *Tm = vs + NB * P.max_q;                 // NB x NB
    T *gram = Tm + NB * NB, *tau = gram + NB * NB;
    int *start = reinterpret_cast<int *>(tau + NB);  // nsec + 1 prefix sums of update items
    __shared__ int item_sh;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // first sorted row beyond panel k's and, where there is one, panel k + 1's
    // (of a sector that is factored)
    auto first_row = [&](const LqSec &s, int k) { return min(s.q, (k + 1 + (k + 1 < panels_of(s.q))) * NB); };
    const int panels = P.np[P.nsec];
    auto vbuf = [&](const LqSec &s, int k) { return P.v + s.v_off + int64_t(k & 1) * (NB * (s.q + NB)); };

    // the panel k of sector s, its rows in xs; leaves reflectors and T in the panel's buffer
    auto factor = [&](const LqSec &s, int k, T *xs, int pitch) {
        const int j = k * NB, len = s.q - j, nr = min(NB, s.q - j);
        factor_panel(xs, pitch, vs, Tm, gram, tau, len, nr, warp, lane);
        T *dst = vbuf(s, k);
        for (int e = tid; e < NB * len; e += LT) dst[e] = vs[e];
        for (int e = tid; e < NB * NB; e += LT) dst[NB * s.q + e] = Tm[e];
        if (warp < nr) {
            T *x = P.x + s.x_off + int64_t(P.order[s.o_off + j + warp]) * s.q + j;
            for (int e = lane; e < len; e += 32) x[e] = xs[warp * pitch + e];
        }
        __syncthreads();
    };
    auto load_v = [&](const LqSec &s, int k) {
        const int len = s.q - k * NB;
        const T *src = vbuf(s, k);
        for (int e = tid; e < NB * len; e += LT) vs[e] = __ldcg(src + e);
        for (int e = tid; e < NB * NB; e += LT) Tm[e] = __ldcg(src + NB * s.q + e);
    };

    for (int i = blockIdx.x; i < P.nsec; i += gridDim.x) {
        const LqSec s = P.secs[i];
        if (P.np[i] < 1) continue;
        const int nr = min(NB, s.q);
        if (warp < nr) {
            const T *x = P.x + s.x_off + int64_t(P.order[s.o_off + warp]) * s.q;
            for (int e = lane; e < s.q; e += 32) buf[warp * s.q + e] = __ldcg(x + e);
        }
        __syncthreads();
        factor(s, 0, buf, s.q);
    }
    grid.sync();
    for (int k = 0; k < panels; ++k) {
        const int j = k * NB;
        // owners: panel k on the rows of panel k + 1, then that panel's factorisation
        for (int i = blockIdx.x; i < P.nsec; i += gridDim.x) {
            const LqSec s = P.secs[i];
            if (k + 1 >= P.np[i]) continue;
            const int len = s.q - j, nr = min(NB, s.q - j - NB);
            load_v(s, k);
            T *x = buf + warp * len;
            if (warp < nr) {
                const T *src = P.x + s.x_off + int64_t(P.order[s.o_off + j + NB + warp]) * s.q + j;
                for (int e = lane; e < len; e += 32) x[e] = __ldcg(src + e);
            }
            __syncthreads();
            if (warp < nr) {
                apply_panel(x, vs, Tm, len, lane);
                // the elements of panel k are final
                T *dst = P.x + s.x_off + int64_t(P.order[s.o_off + j + NB + warp]) * s.q + j;
                if (lane < NB) dst[lane] = x[lane];
            }
            __syncthreads();
            factor(s, k + 1, buf + NB, len);
        }
        // the other vectors: items of `chunk` vectors, claimed by whichever CTA is free
        __syncthreads();
        if (warp == 0) {
            int carry = 0;
            for (int base = 0; base < P.nsec; base += 32) {
                const int i = base + lane;
                int n = 0;
                if (i < P.nsec) {
                    const LqSec &s = P.secs[i];
                    if (k < P.np[i]) n = (s.p - first_row(s, k) + s.q + P.chunk - 1) / P.chunk;
                }
                int v = n;
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, v, o);
                    if (lane >= o) v += u;
                }
                if (i < P.nsec) start[i + 1] = v + carry;
                carry += __shfl_sync(0xffffffffu, v, 31);
            }
            if (lane == 0) start[0] = 0;
        }
        __syncthreads();
        const int total = start[P.nsec];
        int have = -1;  // sector whose reflectors are in shared memory
        for (;;) {
            if (tid == 0) item_sh = atomicAdd(P.next + k, 1);
            __syncthreads();
            const int item = item_sh;
            if (item >= total) break;
            int lo = 0, hi = P.nsec - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (start[mid] <= item)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const LqSec s = P.secs[lo];
            const int len = s.q - j;
            if (have != lo) load_v(s, k);
            have = lo;
            __syncthreads();
            const int first = first_row(s, k), nw = s.p - first, nv = nw + s.q;
            const int v0 = (item - start[lo]) * P.chunk, v1 = min(nv, v0 + P.chunk);
            T *y = buf + warp * len;
            for (int v = v0 + warp; v < v1; v += LT / 32) {
                const int64_t vec = v < nw ? P.order[s.o_off + first + v] : int64_t(s.p) + (v - nw);
                T *x = P.x + s.x_off + vec * s.q + j;
                for (int e = lane; e < len; e += 32) y[e] = __ldcg(x + e);
                __syncwarp();
                apply_panel(y, vs, Tm, len, lane);
                __syncwarp();
                for (int e = lane; e < len; e += 32) x[e] = y[e];
                __syncwarp();
            }
            __syncthreads();
        }
        grid.sync();
    }
}

// Transposed copies between the column-major work / rotation matrices and the vectors X, in 32 x 32
// tiles through shared memory: rows of W (store == 0: X <- W, else W <- X) and the rotation's rows
// (store == 0: X <- identity; else rot <- X).
template <class T>
__global__ void __launch_bounds__(256) k_lq_move(T *__restrict__ work, T *__restrict__ rot, T *__restrict__ x,
                                                 const LqSec *__restrict__ secs, int store) {
    __shared__ T tile[32][33];
    const LqSec s = secs[blockIdx.y];
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int nr = (s.p + 31) / 32 + (s.q + 31) / 32, nc = (s.q + 31) / 32;
    for (int t = blockIdx.x; t < nr * nc; t += gridDim.x) {
        const int rt = t / nc, c0 = (t - rt * nc) * 32;
        const bool w = rt < (s.p + 31) / 32;
        const int r0 = (w ? rt : rt - (s.p + 31) / 32) * 32, rows = w ? s.p : s.q;
        T *m = w ? work + s.w_off : rot + s.rot_off;          // rows x q, column-major
        T *v = x + s.x_off + (w ? 0 : int64_t(s.p) * s.q);    // rows vectors of q
        for (int i = ty; i < 32; i += 8) {
            if (store) {
                const int r = r0 + i, c = c0 + tx;
                tile[i][tx] = r < rows && c < s.q ? v[int64_t(r) * s.q + c] : T(0);
            } else {
                const int r = r0 + tx, c = c0 + i;
                tile[tx][i] = r < rows && c < s.q ? (w ? m[int64_t(c) * rows + r] : (r == c ? T(1) : T(0))) : T(0);
            }
        }
        __syncthreads();
        for (int i = ty; i < 32; i += 8) {
            if (store) {
                const int r = r0 + tx, c = c0 + i;
                if (r < rows && c < s.q) m[int64_t(c) * rows + r] = tile[tx][i];
            } else {
                const int r = r0 + i, c = c0 + tx;
                if (r < rows && c < s.q) v[int64_t(r) * s.q + c] = tile[i][tx];
            }
        }
        __syncthreads();
    }
}

// Squared norms of W's rows (one warp each).
template <class T>
__global__ void __launch_bounds__(256) k_lq_norms(const T *__restrict__ x, const LqSec *__restrict__ secs,
                                                  double *__restrict__ norms) {
    const LqSec s = secs[blockIdx.y];
    const int lane = threadIdx.x & 31, r = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (r >= s.p) return;
    const T *v = x + s.x_off + int64_t(r) * s.q;
    float f = 0.0f;  // an order is all that is wanted, but of values over the whole FP64 range
    double d = 0.0;
    if (sizeof(T) == 4) {
        for (int e = lane; e < s.q; e += 32) f = fmaf(float(v[e]), float(v[e]), f);
        d = double(lsum(f));
    } else {
        for (int e = lane; e < s.q; e += 32) d = fma(double(v[e]), double(v[e]), d);
        d = lsum(d);
    }
    if (lane == 0) norms[s.o_off + r] = d;
}

// order <- the rows by falling norm: ranks in bit order (a permutation also with NaN).  np <- the sector's panels, none
// if it is tall (p >= 1.5 q) and its largest squared row norm is at most `graded` times the smallest.
__global__ void __launch_bounds__(256) k_lq_rank(const double *__restrict__ norms, const LqSec *__restrict__ secs,
                                                 int *__restrict__ order, int *__restrict__ np, double graded) {
    const LqSec s = secs[blockIdx.y];
    const int r = blockIdx.x * 256 + threadIdx.x;
    __shared__ long long keys[256];
    const long long mine = r < s.p ? __double_as_longlong(norms[s.o_off + r]) : 0;
    int rank = 0;
    long long low = __double_as_longlong(norms[s.o_off]), high = low;
    for (int b = 0; b < s.p; b += 256) {
        __syncthreads();
        if (b + int(threadIdx.x) < s.p) keys[threadIdx.x] = __double_as_longlong(norms[s.o_off + b + threadIdx.x]);
        __syncthreads();
        const int n = min(256, s.p - b);
        for (int i = 0; i < n; ++i) {
            rank += keys[i] > mine || (keys[i] == mine && b + i < r);
            low = min(low, keys[i]);
            high = max(high, keys[i]);
        }
    }
    if (r == 0) {
        const bool left = 2 * s.p >= 3 * s.q && !(__longlong_as_double(high) > graded * __longlong_as_double(low));
        const int n = left ? 0 : panels_of(s.q);
        np[blockIdx.y] = n;
        atomicMax(np + gridDim.y, n);
    }
    if (r < s.p) order[s.o_off + rank] = r;
}

template <class T>
BufPtr lq_impl(T *work, T *rot, const std::vector<LqSec> &host, double graded) {
    std::vector<LqSec> secs = host;
    int64_t xs = 0, vs = 0, os = 0;
    int max_q = 0, max_p = 0;
    for (LqSec &s : secs) {
        s.x_off = xs;
        s.v_off = vs;
        s.o_off = os;
        xs += int64_t(s.p + s.q) * s.q;
        vs += 2 * int64_t(NB) * (s.q + NB);
        os += s.p;
        max_q = std::max(max_q, int(s.q));
        max_p = std::max(max_p, int(s.p));
    }
    const int nsec = int(secs.size()), panels = (max_q - 1 + NB - 1) / NB;
    const cudaStream_t st = ctx().stream;
    // one buffer for vectors, reflectors, norms and order, one for the panels and the counters
    const size_t xb = (size_t(xs) * sizeof(T) + 255) & ~size_t(255), vb = (size_t(vs) * sizeof(T) + 255) & ~size_t(255);
    const size_t nb = (size_t(os) * 8 + 255) & ~size_t(255), ob = (size_t(os) * 4 + 255) & ~size_t(255);
    const size_t counters = size_t(panels + 1 + nsec + 1) * 4;
    BufPtr buf = dev_alloc(xb + vb + nb + ob), ints = dev_alloc(counters);
    char *p = static_cast<char *>(buf->p);
    T *x = reinterpret_cast<T *>(p);
    double *norms = reinterpret_cast<double *>(p + xb + vb);
    int *order = reinterpret_cast<int *>(p + xb + vb + nb);
    int *np = static_cast<int *>(ints->p), *next = np + nsec + 1;
    cuda_check(cudaMemsetAsync(np, 0, counters, st), "cudaMemsetAsync(LQ counters)");
    const LqSec *dsecs = upload_vec(secs);
    const int tiles = ((max_p + 31) / 32 + (max_q + 31) / 32) * ((max_q + 31) / 32);
    const dim3 mv(unsigned(std::min(tiles, 4096)), unsigned(nsec));
    k_lq_move<T><<<mv, 256, 0, st>>>(work, rot, x, dsecs, 0);
    k_lq_norms<T><<<dim3(unsigned((max_p + 7) / 8), unsigned(nsec)), 256, 0, st>>>(x, dsecs, norms);
    k_lq_rank<<<dim3(unsigned((max_p + 255) / 256), unsigned(nsec)), 256, 0, st>>>(norms, dsecs, order, np, graded);
    const size_t smem = (size_t(2) * NB * max_q + 2 * NB * NB + NB) * sizeof(T) + size_t(nsec + 1) * sizeof(int);
    static std::atomic<uint64_t> attr{0};
    once_per_device(attr, [] {
        cuda_check(cudaFuncSetAttribute(k_lq<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(LQ_SMEM_MAX)),
                   "LQ smem attribute");
    });
    int occ = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_lq<T>, LT, smem), "occupancy");
    if (occ < 1) fail(ERR_RUNTIME, "the LQ kernel cannot be resident on an SM");
    int64_t vectors = 0;
    for (const LqSec &s : secs) vectors += s.p + s.q;
    // two CTAs an SM at most, one per eight vectors; items of one round of them
    const int sms = device_sm_count();
    const int grid = int(std::max<int64_t>(1, std::min<int64_t>(int64_t(sms) * std::min(occ, 2), (vectors + 7) / 8)));
    LqParams<T> P;
    P.x = x;
    P.v = reinterpret_cast<T *>(p + xb);
    P.secs = dsecs;
    P.order = order;
    P.next = next;
    P.nsec = nsec;
    P.np = np;
    P.chunk = int(std::max<int64_t>(8, (vectors + grid - 1) / grid / 8 * 8));
    P.max_q = max_q;
    void *args[] = {&P};
    cuda_check(cudaLaunchCooperativeKernel((void *)k_lq<T>, dim3(grid), dim3(LT), args, smem, st), "cooperative LQ launch");
    k_lq_move<T><<<mv, 256, 0, st>>>(work, rot, x, dsecs, 1);
    count_launch(5);
    cuda_check(cudaGetLastError(), "LQ kernel launch");
    return ints;
}
}  // namespace

int lq_max_q(int f32, int nsec) {
    const size_t es = f32 ? 4 : 8;
    const size_t fixed = (2 * NB * NB + NB) * es + size_t(nsec + 1) * sizeof(int);
    return fixed >= LQ_SMEM_MAX ? 0 : int((LQ_SMEM_MAX - fixed) / (2 * NB * es));
}

BufPtr launch_lq(void *work, void *rot, const std::vector<LqSec> &secs, int f32, double graded) {
    if (secs.empty()) return nullptr;
    return f32 ? lq_impl(static_cast<float *>(work), static_cast<float *>(rot), secs, graded)
               : lq_impl(static_cast<double *>(work), static_cast<double *>(rot), secs, graded);
}

}  // namespace qtt
