// FP64 refinement of the mixed path's sector SVDs.
//
// QuantiT decomposes every sector in FP64 (torch::svd, sources/btensor_linalg.cpp:483).
// The mixed path keeps that accuracy while doing most sweeps in FP32: the one-sided
// Jacobi first runs on an FP32 copy of each sector (FP32 runs at 64x the FP64 rate on
// GB300's CUDA cores), and its accumulated rotation V0 then starts an FP64 Jacobi on
// the FP64 sector matrix:
//
//   1. V0 is orthogonal only to ~1e-6 (FP32 accumulation).  Two Newton-Schulz steps
//      V <- V + V E, E = (I - V^T V) / 2, in FP64 make it orthogonal to FP64 precision (each
//      step squares the departure from orthogonality: 1e-6 -> 1e-12 -> 1e-16).
//   2. W1 = W V in FP64 from the FP64 sector matrix W.
//   3. The FP64 Jacobi sweeps run on (W1, V).  Any orthogonal V gives an exact SVD of
//      W (W V = U S Vt^T => W = U S (V Vt)^T), so the factors are an FP64 SVD; from the
//      near-diagonal W1 the columns FP32 resolved converge in a sweep or two.
//
// The Gram matrices and W V are FP64 products of the grouped block GEMM (gemm_f64.cu), all sectors
// of a decomposition in one launch.  The correction V E is formed in FP32: E is at most 1e-6 (then
// 1e-12), so its relative error of 1e-7 leaves 1e-13 behind in the first step, which the second
// removes with the rest, and 1e-19 in the second.  That leaves 2 q^3 of 6 q^3 FP64 FLOP to the
// orthogonalisation; with it and the finer tiles of the Grams' upper halves (64 x 64 tiles of a q ~
// 900 sector left the SMs a last wave of a few) the five products of the cylinder theta at D = 2048
// went from 19.3 to 7.7 ms (its whole decomposition from 70 to 58 ms).
#include "kernels.h"
#include "qtt_core.h"

namespace qtt {
namespace {

constexpr int CT = 64, CK = 16;  // FP32 correction: tile and K slab

// out = V + 0.5 V (I - G) per sector (q x q, column-major); G's elements below the diagonal are
// read from above it (G[min + max q]).
struct Correction {
    int64_t off;
    int32_t q, tile_start;
};

template <class TV>
__global__ void __launch_bounds__(256) k_ns_correct(const TV *__restrict__ V, const double *__restrict__ G,
                                                    double *__restrict__ out, const Correction *__restrict__ cs, int n) {
    __shared__ float As[CK][CT + 1];
    __shared__ float Bs[CK][CT + 1];
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (cs[mid].tile_start <= int(blockIdx.x))
            lo = mid;
        else
            hi = mid - 1;
    }
    const Correction c = cs[lo];
    const int q = c.q, tm = (q + CT - 1) / CT, t = int(blockIdx.x) - c.tile_start;
    const int r0 = (t % tm) * CT, c0 = (t / tm) * CT;
    const TV *v = V + c.off;
    const double *g = G + c.off;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
    for (int k0 = 0; k0 < q; k0 += CK) {
        for (int e = threadIdx.x; e < CK * CT; e += 256) {
            const int i = e % CT, kk = e / CT, r = r0 + i, k = k0 + kk;
            As[kk][i] = r < q && k < q ? float(v[int64_t(k) * q + r]) : 0.0f;
            const int kb = e % CK, jj = e / CK, col = c0 + jj, kq = k0 + kb;
            float x = 0.0f;
            if (col < q && kq < q) x = float((kq == col ? 1.0 : 0.0) - g[int64_t(max(kq, col)) * q + min(kq, col)]);
            Bs[kb][jj] = x;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < CK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][tx + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][ty + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int col = c0 + ty + 16 * j;
        if (col >= q) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = r0 + tx + 16 * i;
            if (row < q) out[c.off + int64_t(col) * q + row] = double(v[int64_t(col) * q + row]) + 0.5 * double(acc[i][j]);
        }
    }
}

template <class TV>
void ns_correct(const TV *V, const double *G, double *out, const std::vector<SectorDesc> &secs) {
    std::vector<Correction> cs;
    int tiles = 0;
    for (const SectorDesc &s : secs) {
        if (s.q <= 0) continue;
        cs.push_back(Correction{s.rot_off, s.q, tiles});
        const int t = (s.q + CT - 1) / CT;
        tiles += t * t;
    }
    if (cs.empty()) return;
    k_ns_correct<TV><<<tiles, 256, 0, ctx().stream>>>(V, G, out, upload_vec(cs), int(cs.size()));
    count_launch();
    cuda_check(cudaGetLastError(), "Newton-Schulz correction launch");
}

// G <- 1.5 I - G / 2 with G's elements below the diagonal read from above it: the factor of a Newton-Schulz step
// taken as one FP64 product, V <- V (3 I - V^T V) / 2.
__global__ void __launch_bounds__(256) k_ns_factor(double *__restrict__ G, const SectorDesc *__restrict__ secs) {
    const int q = secs[blockIdx.y].q;
    double *g = G + secs[blockIdx.y].rot_off;
    for (int64_t e = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; e < int64_t(q) * q; e += int64_t(gridDim.x) * blockDim.x) {
        const int64_t r = e % q, c = e / q;
        if (r > c) continue;
        const double v = (r == c ? 1.5 : 0.0) - 0.5 * g[e];
        g[e] = v;
        g[r * q + c] = v;
    }
}

// One FP64 product per task in one launch of the grouped block GEMM, column-major:
// C (M x N, ldc = M) = op(A) B, A M x K (a_trans: stored K x M), B K x N.  upper: C is symmetric, tiles
// strictly below the diagonal are left out.
struct Product {
    int64_t a_off, b_off, c_off;
    int32_t M, N, K;
    bool a_trans, upper;
};
void products(const double *A, const double *B, double *C, const std::vector<Product> &tasks) {
    // the GEMM writes row-major: C^T = B^T op(A)^T, so its rows are our columns
    std::vector<F64Pair> pairs;
    std::vector<GemmOut> outs;
    std::vector<GemmTile> tiles;
    int64_t square = 0;
    double area = 0, volume = 0;
    for (const Product &t : tasks) {
        square += ((int64_t(t.M) + 31) / 32) * ((int64_t(t.N) + 31) / 32);
        area += double(t.M) * t.N;
        volume += double(t.M) * t.N * t.K;
    }
    const bool fine = gemm_f64_fine(square, volume / std::max(area, 1.0));
    for (const Product &t : tasks) {
        if (t.M <= 0 || t.N <= 0 || t.K <= 0) continue;
        F64Pair p{};
        p.a_off = t.b_off;
        p.b_off = t.a_off;
        p.k1 = 1;
        p.k2 = t.K;
        p.ak2 = 1;
        p.bk2 = t.a_trans ? 1 : t.M;
        p.am2 = t.N;
        p.as2 = t.K;
        p.bn2 = t.M;
        p.bs2 = t.a_trans ? t.K : 1;
        GemmOut o{};
        o.c_off = t.c_off;
        o.add_off = -1;
        o.M = t.N;
        o.N = t.M;
        o.p0 = int32_t(pairs.size());
        o.p1 = o.p0 + 1;
        int tm, tn;
        const int cls = gemm_f64_class(o.M, o.N, t.K, &tm, &tn, fine);
        for (int m0 = 0; m0 < o.M; m0 += tm)
            for (int n0 = 0; n0 < o.N; n0 += tn) {
                // (row of C^T = column of C) a tile is needed if it reaches the diagonal or above
                if (t.upper && n0 > m0 + tm - 1) continue;
                tiles.push_back(GemmTile{int32_t(outs.size()), m0, n0, cls});
            }
        pairs.push_back(p);
        outs.push_back(o);
    }
    if (tiles.empty()) return;
    std::stable_sort(tiles.begin(), tiles.end(), [&](const GemmTile &x, const GemmTile &y) {
        return pairs[x.out].k2 > pairs[y.out].k2;
    });
    F64Args g;
    g.A = B;
    g.B = A;
    g.C = C;
    g.Cadd = nullptr;
    const BufPtr tables = upload_many({table(pairs, g.pairs), table(outs, g.outs), table(tiles, g.tiles)});
    g.ntiles = int32_t(tiles.size());
    g.b_strided = tasks.front().a_trans ? 1 : 0;
    g.alpha = 1.0;
    g.beta = 0.0;
    launch_gemm_f64(g);
}

// Squared column norms of every sector matrix (one warp per column); amax: of the sectors as they were before k_pack scaled
// them.
template <class T>
__global__ void k_col_norms(const T *__restrict__ W, const SectorDesc *__restrict__ secs,
                            double *__restrict__ out, const uint32_t *__restrict__ amax) {
    const SectorDesc sd = secs[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const int col = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (col >= sd.q) return;
    const T *w = W + sd.w_off + int64_t(col) * sd.p;
    double acc = 0.0;
    for (int r = lane; r < sd.p; r += 32) acc = fma(double(w[r]), double(w[r]), acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) out[sd.s_off + col] = amax ? ldexp(acc, 2 * sector_exponent(amax[blockIdx.y])) : acc;
}

template <class T>
__global__ void __launch_bounds__(256) k_col_copy(const T *__restrict__ src, T *__restrict__ dst,
                                                  const ColCopy *__restrict__ cc, int n) {
    for (int c = blockIdx.x; c < n; c += gridDim.x) {
        const ColCopy e = cc[c];
        for (int r = threadIdx.x; r < e.len; r += blockDim.x) dst[e.dst_off + r] = src[e.src_off + r];
    }
}

}  // namespace

void launch_col_copy(const void *src, void *dst, const std::vector<ColCopy> &cols, int f32) {
    if (cols.empty()) return;
    const ColCopy *d = upload_vec(cols);
    const int grid = int(std::min<size_t>(cols.size(), 8192));
    if (f32)
        k_col_copy<float><<<grid, 256, 0, ctx().stream>>>(static_cast<const float *>(src), static_cast<float *>(dst), d,
                                                          int(cols.size()));
    else
        k_col_copy<double><<<grid, 256, 0, ctx().stream>>>(static_cast<const double *>(src), static_cast<double *>(dst), d,
                                                           int(cols.size()));
    count_launch();
    cuda_check(cudaGetLastError(), "column copy launch");
}

void launch_rot_product(const double *vg, const double *r, double *vn, const std::vector<RotProduct> &t) {
    std::vector<Product> g;
    for (const RotProduct &e : t) g.push_back({e.vg_off, e.r_off, e.vn_off, e.vrows, e.k, e.k, false, false});
    products(vg, r, vn, g);
}

void launch_col_norms(const void *W, const SectorDesc *secs, int nsec, int max_q, double *out, int f32, const uint32_t *amax) {
    if (nsec <= 0 || max_q <= 0) return;
    const dim3 grid(unsigned((max_q + 7) / 8), unsigned(nsec));
    if (f32)
        k_col_norms<float><<<grid, 256, 0, ctx().stream>>>(static_cast<const float *>(W), secs, out, amax);
    else
        k_col_norms<double><<<grid, 256, 0, ctx().stream>>>(static_cast<const double *>(W), secs, out, amax);
    count_launch();
    cuda_check(cudaGetLastError(), "column norm launch");
}

void launch_svd_refine(const float *rot32, int64_t rot_size, const double *w64, double *w1, double *va, double *vb,
                       double *g, const std::vector<SectorDesc> &secs, bool exact) {
    std::vector<Product> gram, wv, ns;
    int max_q = 0;
    for (const SectorDesc &s : secs) {
        max_q = std::max(max_q, int(s.q));
        ns.push_back({s.rot_off, s.rot_off, s.rot_off, s.q, s.q, s.q, false, false});
        gram.push_back({s.rot_off, s.rot_off, s.rot_off, s.q, s.q, s.q, true, true});
        wv.push_back({s.w_off, s.rot_off, s.w_off, s.p, s.q, s.q, false, false});
    }
    // step 1 from the FP32 rotation (widened into vb): va = V0 + V0 (I - V0^T V0) / 2
    launch_convert(rot32, vb, rot_size, 0, 1);
    products(vb, vb, g, gram);
    if (exact && max_q > 0) {
        // all FP64, as whole products: the values do not depend on how the correction is cut
        const dim3 grid(unsigned(std::min<int64_t>((int64_t(max_q) * max_q + 2047) / 2048, 1024)), unsigned(secs.size()));
        const SectorDesc *dsec = upload_vec(secs);
        auto factor = [&] {
            k_ns_factor<<<grid, 256, 0, ctx().stream>>>(g, dsec);
            count_launch();
            cuda_check(cudaGetLastError(), "Newton-Schulz factor launch");
        };
        factor();
        products(vb, g, va, ns);
        products(va, va, g, gram);
        factor();
        products(va, g, vb, ns);
    } else {
        ns_correct(rot32, g, va, secs);
        // step 2: vb = va + va (I - va^T va) / 2
        products(va, va, g, gram);
        ns_correct(static_cast<const double *>(va), g, vb, secs);
    }
    products(w64, vb, w1, wv);
}

}  // namespace qtt
