// Grouped FP64 block GEMM: every charge-matched block product of one
// contraction in one launch (btensor::tensordot's mm / addmm_ loop,
// sources/btensor.cpp:2057-2114).  One CTA computes a tile of one output block
// and accumulates all of that block's matching (A, B) pairs in registers, in pair
// order and with K ascending, before a single store, so no output block is written
// twice and the sums do not depend on the tile shape.
//
// FP64 has no tcgen05 kind and GB300's FP64 pipe retires about 2 FMA per clock and SM
// (a warp's FMA occupies it for 16 clocks), so the kernel is built around not issuing
// an FMA that is not needed rather than around feeding the pipe:
//  * Operands are read where they lie, through L1, with no shared-memory staging: a
//    2 x 2 register tile needs 4 loads for 64 clocks of FMA.  That leaves no CTA
//    barrier in the loop, no padding of K, and any leg order whose free and contracted
//    legs each fold to two strides needs no packed copy of the operand first (f64_square: warps of either shape).
//  * The tile follows the block: 32 x 32, 16 x 16 where that leaves SMs idle (gemm_f64_fine) or most of
//    the tile outside the block, and 256 x 8 / 8 x 256 strips for the thin products of
//    an MPO tensor (N or M of a few, K of a few), which are bound by memory.
// Against 64 x 64 x 16 tiles staged in shared memory (17 us of FP64 pipe for any tile,
// however small the block), same sums to the last bit: theta pair contraction at D = 2048
// 1787 -> 1192 us (1.07 TFLOP/s, 89% of what independent FMAs reach; mma.sync FP64 runs on the same pipe at
// 1.05 against their 1.20 TFLOP/s); the matvec of a Hubbard chain at D = 512 2584 -> 771 us, of which its kernels
// take 124 and the host's planning the rest; an environment update of a spin chain at D = 777
// 1271 -> 315 us; a 24-dimensional site pair 34 -> 15 us.
#include "kernels.h"
#include "qtt_core.h"

namespace qtt {
namespace {
constexpr int THREADS = 256;
constexpr int PBATCH = 32;  // pair descriptors staged in shared memory at a time

// Copies np pair descriptors to shared memory.
__device__ __forceinline__ void stage_pairs(F64Pair *sp, const F64Pair *pairs, int np) {
    __syncthreads();
    const int4 *src = reinterpret_cast<const int4 *>(pairs);
    int4 *dst = reinterpret_cast<int4 *>(sp);
    for (int e = threadIdx.x; e < np * int(sizeof(F64Pair) / 16); e += THREADS) dst[e] = src[e];
    __syncthreads();
}

__device__ __forceinline__ void store_out(const F64Args &g, const GemmOut &o, int64_t idx, double acc) {
    double v = g.alpha * acc;
    if (o.add_off >= 0) v += g.beta * g.Cadd[o.add_off + idx];
    g.C[o.c_off + idx] = v;
}

// A square tile: RT x RT outputs per thread, 16 x 16 threads.  A warp covers 2 rows x 16 columns, whose loads of B are one
// line, or 8 x 4 where B's columns are strided (its last leg is contracted) and every one of them is a line of its own:
// 12 instead of 18 lines a k where a warp's FMA takes 16 clocks.  M = N = K = 576 722 -> 366 us, 600 x 600 x 4000 5639 ->
// 2670; with 8 x 4 for contiguous columns too the lines would be 9 instead of 3.
template <int RT, int U>
__device__ __forceinline__ void f64_square(const F64Args &g, const GemmTile &t, const GemmOut &o, F64Pair *sp) {
    constexpr int RM = RT, RN = RT, TX = 16, TY = 16;
    const int tid = threadIdx.x;
    const int tx = g.b_strided ? (tid & 3) | (tid >> 3 & 12) : tid % TX;
    const int ty = g.b_strided ? (tid >> 2 & 7) | (tid >> 4 & 8) : tid / TX;
    // rows / columns of the register tile that the block reaches (the same for every thread)
    const int rm = min(RM, (o.M - t.m0 + TY - 1) / TY), rn = min(RN, (o.N - t.n0 + TX - 1) / TX);
    int m[RM], n[RN];
#pragma unroll
    for (int i = 0; i < RM; ++i) m[i] = min(t.m0 + ty + TY * i, o.M - 1);
#pragma unroll
    for (int j = 0; j < RN; ++j) n[j] = min(t.n0 + tx + TX * j, o.N - 1);
    double acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.0;

    for (int pb = o.p0; pb < o.p1; pb += PBATCH) {
        const int np = min(PBATCH, o.p1 - pb);
        stage_pairs(sp, g.pairs + pb, np);
        for (int p = 0; p < np; ++p) {
            const F64Pair &pr = sp[p];
            const double *pa[RM], *pB[RN];
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const int q = m[i] / pr.am2, r = m[i] - q * pr.am2;
                pa[i] = g.A + pr.a_off + int64_t(q) * pr.as1 + int64_t(r) * pr.as2;
            }
#pragma unroll
            for (int j = 0; j < RN; ++j) {
                const int q = n[j] / pr.bn2, r = n[j] - q * pr.bn2;
                pB[j] = g.B + pr.b_off + int64_t(q) * pr.bs1 + int64_t(r) * pr.bs2;
            }
            const int K1 = pr.k1, K2 = pr.k2;
            const int64_t ak = pr.ak2, bk = pr.bk2;
            for (int k1 = 0; k1 < K1; ++k1) {
                const int64_t oa = int64_t(k1) * pr.ak1, ob = int64_t(k1) * pr.bk1;
                int k = 0;
                for (; k + U <= K2; k += U) {
                    double a[U][RM], b[U][RN];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
#pragma unroll
                        for (int i = 0; i < RM; ++i)
                            if (i < rm) a[u][i] = *(pa[i] + oa + (k + u) * ak);
#pragma unroll
                        for (int j = 0; j < RN; ++j)
                            if (j < rn) b[u][j] = *(pB[j] + ob + (k + u) * bk);
                    }
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int i = 0; i < RM; ++i)
                            if (i < rm)
#pragma unroll
                                for (int j = 0; j < RN; ++j)
                                    if (j < rn) acc[i][j] = fma(a[u][i], b[u][j], acc[i][j]);
                }
                for (; k < K2; ++k) {
                    double a[RM], b[RN];
#pragma unroll
                    for (int i = 0; i < RM; ++i)
                        if (i < rm) a[i] = *(pa[i] + oa + k * ak);
#pragma unroll
                    for (int j = 0; j < RN; ++j)
                        if (j < rn) b[j] = *(pB[j] + ob + k * bk);
#pragma unroll
                    for (int i = 0; i < RM; ++i)
                        if (i < rm)
#pragma unroll
                            for (int j = 0; j < RN; ++j)
                                if (j < rn) acc[i][j] = fma(a[i], b[j], acc[i][j]);
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int gm = t.m0 + ty + TY * i;
        if (gm >= o.M) continue;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
            const int gn = t.n0 + tx + TX * j;
            if (gn >= o.N) continue;
            store_out(g, o, int64_t(gm) * o.N + gn, acc[i][j]);
        }
    }
}

// A strip: one row (TALL) or column per thread and the block's up to 8 columns (rows),
// whose operand values are the same for every thread.
template <bool TALL, int U>
__device__ __forceinline__ void f64_strip(const F64Args &g, const GemmTile &t, const GemmOut &o, F64Pair *sp) {
    constexpr int S = F64_STRIP;
    const int tid = threadIdx.x;
    const int l0 = (TALL ? t.m0 : t.n0) + tid, len = TALL ? o.M : o.N, ns = TALL ? o.N : o.M;
    const int l = min(l0, len - 1);
    const double *L = TALL ? g.A : g.B, *Sh = TALL ? g.B : g.A;  // long and short side
    double acc[S];
#pragma unroll
    for (int j = 0; j < S; ++j) acc[j] = 0.0;
    for (int pb = o.p0; pb < o.p1; pb += PBATCH) {
        const int np = min(PBATCH, o.p1 - pb);
        stage_pairs(sp, g.pairs + pb, np);
        for (int p = 0; p < np; ++p) {
            const F64Pair &pr = sp[p];
            const int l2 = TALL ? pr.am2 : pr.bn2, s2 = TALL ? pr.bn2 : pr.am2;
            const int q = l / l2, r = l - q * l2;
            const double *pl = L + (TALL ? pr.a_off : pr.b_off) + int64_t(q) * (TALL ? pr.as1 : pr.bs1) +
                               int64_t(r) * (TALL ? pr.as2 : pr.bs2);
            const double *ps = Sh + (TALL ? pr.b_off : pr.a_off);
            int off[S];
#pragma unroll
            for (int j = 0; j < S; ++j) {
                const int js = min(j, ns - 1), q1 = js / s2;
                off[j] = q1 * (TALL ? pr.bs1 : pr.as1) + (js - q1 * s2) * (TALL ? pr.bs2 : pr.as2);
            }
            const int64_t lk = TALL ? pr.ak2 : pr.bk2, sk = TALL ? pr.bk2 : pr.ak2;
            const int K1 = pr.k1, K2 = pr.k2;
            for (int k1 = 0; k1 < K1; ++k1) {
                const double *xl = pl + int64_t(k1) * (TALL ? pr.ak1 : pr.bk1);
                const double *xs = ps + int64_t(k1) * (TALL ? pr.bk1 : pr.ak1);
                int k = 0;
                for (; k + U <= K2; k += U) {
                    double v[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) v[u] = *(xl + (k + u) * lk);
#pragma unroll
                    for (int u = 0; u < U; ++u)
#pragma unroll
                        for (int j = 0; j < S; ++j)
                            if (j < ns) {
                                const double w = *(xs + (k + u) * sk + off[j]);
                                acc[j] = TALL ? fma(v[u], w, acc[j]) : fma(w, v[u], acc[j]);
                            }
                }
                for (; k < K2; ++k) {
                    const double v = *(xl + k * lk);
#pragma unroll
                    for (int j = 0; j < S; ++j)
                        if (j < ns) {
                            const double w = *(xs + k * sk + off[j]);
                            acc[j] = TALL ? fma(v, w, acc[j]) : fma(w, v, acc[j]);
                        }
                }
            }
        }
    }
    if (l0 >= len) return;
#pragma unroll
    for (int j = 0; j < S; ++j)
        if (j < ns) store_out(g, o, TALL ? int64_t(l0) * o.N + j : int64_t(j) * o.N + l0, acc[j]);
}

__global__ void __launch_bounds__(THREADS, 3) k_gemm_f64(F64Args g) {
    __shared__ __align__(16) F64Pair sp[PBATCH];
    const GemmTile t = g.tiles[blockIdx.x];
    const GemmOut o = g.outs[t.out];
    switch (t.cls) {
        case F64_SQUARE: f64_square<2, 4>(g, t, o, sp); break;
        case F64_SMALL: f64_square<1, 4>(g, t, o, sp); break;
        case F64_TALL: f64_strip<true, 4>(g, t, o, sp); break;
        default: f64_strip<false, 4>(g, t, o, sp); break;
    }
}
}  // namespace

// 16 x 16 tiles take as long per FMA as 32 x 32 ones (the FP64 pipe is busy either way) and share out more evenly
// over three CTAs an SM, until the lines that they load four times as often are what counts.  32 x 32 and 16 x 16,
// us: M = N = K = 800 1045, 914; 1000 2298, 1781; 1700 8988, 8296; 2200 18244, 17714 (4761 tiles); 3000 44636,
// 45546; 3500 71090, 74046; 3000 x 300 x 2000 4541, 3116; an environment of the cylinder at D = 1024 (4974 tiles, K
// ~136) 2364, 2482.  Short sums store more than they load: 1400 x 1400 x 64 272, 282; the matvec of a cylinder at D = 512
// 752, 784.
bool gemm_f64_fine(int64_t square_tiles, double mean_k) {
    return square_tiles < 4 * device_sm_count() || (square_tiles < 30 * device_sm_count() && mean_k >= 128.0);
}

int gemm_f64_class(int64_t M, int64_t N, int64_t K, int *tm, int *tn, bool fine) {
    // (a strip's short-side offsets are 32-bit)
    const bool strip = K <= (int64_t(1) << 27);
    if (strip && N <= F64_STRIP && M >= 64) {
        *tm = THREADS;
        *tn = F64_STRIP;
        return F64_TALL;
    }
    if (strip && M <= F64_STRIP && N >= 64) {
        *tm = F64_STRIP;
        *tn = THREADS;
        return F64_WIDE;
    }
    const int e = fine || (M <= 16 && N <= 16) ? 16 : 32;
    *tm = *tn = e;
    return e == 16 ? F64_SMALL : F64_SQUARE;
}

void launch_gemm_f64(const F64Args &a) {
    if (a.ntiles <= 0) return;
    k_gemm_f64<<<a.ntiles, THREADS, 0, ctx().stream>>>(a);
    count_launch();
    cuda_check(cudaGetLastError(), "grouped FP64 GEMM launch");
}

}  // namespace qtt
