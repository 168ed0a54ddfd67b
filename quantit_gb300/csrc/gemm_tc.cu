// Grouped block GEMM on the 5th-generation tensor cores (tcgen05) with split operands:
// every FP64 operand element x, scaled by a power of two, is split into a few terms of
// a tensor-core type, and each output tile accumulates the products of the leading
// orders in FP32 in tensor memory (TMEM); everything outside the block GEMMs stays FP64.
//
//  * TF32X3: hi = tf32(x), lo = tf32(x - hi); A_hi B_lo + A_lo B_hi + A_hi B_hi.  The
//    dropped A_lo B_lo term and the FP32 accumulation leave about FP32 accuracy.
//  * BF16X3: hi = bf16(x), mid = bf16(x - hi), lo = bf16(x - hi - mid), 24 significant
//    bits together; the six products of order <= 2, smallest first.  Six BF16 products
//    cost the tensor time of three TF32 products.
//
// Three kernels, two of them templates over the schemes:
//  * k_amax: per CTA maxima of |x| of both operands (their scales), in one launch.
//  * k_split: both operands in one launch, straight into the layout the GEMM copies:
//    a block's K is cut into chunks of CKB bytes per row and term; a chunk holds its rows in
//    groups of 8, a group its terms one after the other, a term its 16-byte columns as core
//    matrices (8 rows x 16 bytes).  The rows of an output tile are then ONE contiguous
//    piece of a chunk, terms included: two bulk copies a stage.  Rows are padded to 8 and
//    K to a k-step of 32 bytes by the kernel itself.  A thread writes whole 16-byte rows of
//    core matrices, a warp 512 contiguous bytes.  Bound by memory (4.5 TB/s with the maxima)
//    since the FP64 -> FP32 conversion takes eight integer instructions and flat layouts no
//    division; at 40 instructions an element it was bound by the ALUs.  A CTA's first elements
//    are loaded before it reduces the maxima, of which there are two an SM and operand: 429 -> 392 us for
//    the three splits of the cylinder matvec at D = 2048.
//  * k_gemm_tc: persistent, CTAS_PER_SM CTAs per SM over the longest-first tile list in
//    boustrophedon order, warp-specialised:
//      - warp 0 (producer) fills a ring of stages with bulk asynchronous copies counted on
//        the stage's "full" mbarrier.  A stage takes CKB bytes of K per row from one or
//        several pairs: the thin contractions with an MPO tensor have many pairs of K = 1
//        to 8 per tile.  Tile and pair descriptors are fetched 32 at a time, one per lane.
//      - one thread of warp 1 issues the stage's tcgen05.mma (32 bytes of K each, N
//        rounded up to 16) and commits them to the stage's "empty" mbarrier; the
//        stage's word in shared memory says which units it holds, so this thread reads no
//        table.  A tile accumulates in TMEM buffer i % 2.
//      - warps 2-5 run tile i's epilogue from that buffer (tcgen05.ld, transposed through
//        shared memory so that a warp stores contiguous rows of C) during tile i + 1's MMAs.
//    What bounds it is the one thread's issue (about 900 clocks a stage of six TF32 MMAs that
//    take 450) and, for thin tiles, the epilogue; hence two CTAs per SM, each with half the
//    ring: 88 against 121 us at the D = 4096 theta pair with one CTA and twice the stages,
//    921 against 1518 us for the three contractions of the cylinder matvec at D = 2048.  Launches of no more
//    tiles than SMs have one CTA an SM and stages of twice the K (split_chunk_bytes).
//
// Against row groups outermost (64 or 96 copies of 1 KB a stage), one pair per stage, one CTA
// per SM, five launches and as many memsets: theta pair D = 4096, TF32X3 436 -> 162 us (gemm
// 252 -> 82); D = 1531, BF16X3 130 -> 49 us; cylinder matvec D = 2048, TF32X3 5974 -> 1418 us
// (its MPO contraction alone 2606 -> 357), all to the same last bit.  The epilogue also gives the
// largest result of each CTA, from which the next contraction of a chain takes its operand's scale: reading the
// product again for it was 1543 us instead of 1418.
//
// The order of the MMAs of a tile is that of its pairs and k-steps whatever the stages
// hold, so results do not depend on the grid or the ring.
//
// Every mbarrier wait is bounded (the epilogue's by its tile's K); on timeout the kernel records an error code in
// a device word that the host checks, drains (bounded) the copies and MMAs it
// issued and frees its TMEM before returning.
#include <cstdint>
#include <mutex>

#include "kernels.h"
#include "qtt_core.h"
#include "tc_common.cuh"

namespace qtt {
namespace {
using namespace tc;

constexpr int TBM = 128, TBN = 128;
constexpr int TTHREADS = 192;             // producer, MMA and four epilogue warps
constexpr int CTAS_PER_SM = 2;
constexpr int AMAX_THREADS = 512;
constexpr int TMEM_COLS = 128;            // FP32 accumulator columns of one tile
constexpr int EPI_COLS = 16, EPI_PITCH = EPI_COLS + 1;  // an epilogue warp's 32 x 16 patch (floats)
constexpr int EPI_BYTES = 4 * 32 * EPI_PITCH * 4;

__device__ __forceinline__ uint32_t to_tf32(float x) {
    uint32_t r;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ uint32_t to_bf16(float x) {
    uint16_t r;
    asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float from_bf16(uint32_t h) { return __uint_as_float(h << 16); }

struct Tf32x3 {
    static constexpr int NC = 2, ELEM = 4, NSTAGE = 3, ERR = 1;
    // D = F32, A = B = TF32, both K-major, M = 128
    static __device__ __forceinline__ uint32_t idesc(int n16) {
        return (1u << 4) | (2u << 7) | (2u << 10) | (uint32_t(n16 * 2) << 17) | (uint32_t(TBM >> 4) << 24);
    }
    static __device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.b32 q, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, q;\n}\n" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc));
    }
    // one k-step: small terms first, then the leading product
    static __device__ __forceinline__ void step(uint32_t d, const uint64_t (&a)[NC], const uint64_t (&b)[NC],
                                                uint32_t idesc, uint32_t acc) {
        mma(d, a[0], b[1], idesc, acc);
        mma(d, a[1], b[0], idesc, 1u);
        mma(d, a[0], b[0], idesc, 1u);
    }
    static __device__ __forceinline__ void split(const float (&x)[16 / ELEM], uint4 (&out)[NC]) {
        uint32_t h[4], l[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            h[i] = to_tf32(x[i]);
            l[i] = to_tf32(x[i] - __uint_as_float(h[i]));
        }
        out[0] = make_uint4(h[0], h[1], h[2], h[3]);
        out[1] = make_uint4(l[0], l[1], l[2], l[3]);
    }
};

struct Bf16x3 {
    static constexpr int NC = 3, ELEM = 2, NSTAGE = 2, ERR = 3;
    // D = F32, A = B = BF16, both K-major, M = 128
    static __device__ __forceinline__ uint32_t idesc(int n16) {
        return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(n16 * 2) << 17) | (uint32_t(TBM >> 4) << 24);
    }
    static __device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
        asm volatile(
            "{\n .reg .pred q;\n setp.ne.b32 q, %4, 0;\n"
            " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, q;\n}\n" ::"r"(d),
            "l"(a), "l"(b), "r"(idesc), "r"(acc));
    }
    // one k-step: second-order terms first, then first order, then the leading product
    static __device__ __forceinline__ void step(uint32_t d, const uint64_t (&a)[NC], const uint64_t (&b)[NC],
                                                uint32_t idesc, uint32_t acc) {
        mma(d, a[0], b[2], idesc, acc);
        mma(d, a[1], b[1], idesc, 1u);
        mma(d, a[2], b[0], idesc, 1u);
        mma(d, a[0], b[1], idesc, 1u);
        mma(d, a[1], b[0], idesc, 1u);
        mma(d, a[0], b[0], idesc, 1u);
    }
    static __device__ __forceinline__ void split(const float (&x)[16 / ELEM], uint4 (&out)[NC]) {
        uint32_t w[NC][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t t[2][NC];
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float v = x[2 * i + j];
                t[j][0] = to_bf16(v);
                const float r = v - from_bf16(t[j][0]);
                t[j][1] = to_bf16(r);
                t[j][2] = to_bf16(r - from_bf16(t[j][1]));
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) w[c][i] = t[0][c] | (t[1][c] << 16);
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) out[c] = make_uint4(w[c][0], w[c][1], w[c][2], w[c][3]);
    }
};

// CKB: bytes of K per row and stage (split_chunk_bytes); one operand copy of a stage takes 128 rows of them
constexpr int stage_bytes(int nc, int ckb) { return 2 * nc * 128 * ckb; }
constexpr int smem_bytes(int nc, int nstage, int ckb) { return nstage * stage_bytes(nc, ckb) + EPI_BYTES; }

// Maxima of |x| as bit patterns (bit order = value order for non-negative doubles), one
// per CTA; operand b's CTAs follow operand a's.
__global__ void __launch_bounds__(AMAX_THREADS) k_amax(AmaxArgs g) {
    constexpr int VEC = 8, SPAN = AMAX_THREADS * VEC;
    const int which = int(blockIdx.x) >= g.parts[0];
    const double *__restrict__ x = g.x[which];
    const int64_t n = g.n[which];
    const int64_t first = int64_t(blockIdx.x) - (which ? g.parts[0] : 0), step = int64_t(g.parts[which]) * SPAN;
    unsigned long long m = 0;
    auto take = [&](double v) {
        const unsigned long long u = static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFull;
        m = u > m ? u : m;
    };
    // plain loads: the same loop over __ldg / __ldcg reaches 3.7 TB/s instead of 6.4
    for (int64_t b = first * SPAN + threadIdx.x; b < n; b += step) {
        double v[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) v[j] = b + j * AMAX_THREADS < n ? x[b + j * AMAX_THREADS] : 0.0;
#pragma unroll
        for (int j = 0; j < VEC; ++j) take(v[j]);
    }
    __shared__ unsigned long long red[AMAX_THREADS / 32];
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, m, o);
        m = u > m ? u : m;
    }
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < AMAX_THREADS / 32; ++w) m = red[w] > m ? red[w] : m;
        g.out[blockIdx.x] = m;
    }
}

// The largest of the per-CTA maxima of one operand (every thread of the CTA gets it).
__device__ __forceinline__ unsigned long long amax_of(const unsigned long long *parts, int n, unsigned long long *red) {
    unsigned long long m = 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const unsigned long long u = parts[i];
        m = u > m ? u : m;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long u = __shfl_xor_sync(0xffffffffu, m, o);
        m = u > m ? u : m;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = red[0];
    for (int w = 1; w < int(blockDim.x >> 5); ++w) m = red[w] > m ? red[w] : m;
    return m;
}

// FLAT: every entry's rows have one stride and its K one (no index arithmetic but two
// products); otherwise rows and K of two strides each, or any legs.
template <class S, int CKB, bool FLAT>
__global__ void __launch_bounds__(256) k_split(SplitArgs g) {
    constexpr int EV = 16 / S::ELEM;  // elements of a core matrix row
    __shared__ unsigned long long red[8];
    const SplitTile t = g.tiles[blockIdx.x];
    const SplitEntry &e = g.ents[t.ent];
    const int op = e.operand;
    const double *__restrict__ src = g.src[op] + e.src_off;
    const int kvb = int(min(int64_t(CKB), e.kpb - int64_t(t.chunk) * CKB)), nq = kvb / 16;
    const int rows = e.rows, K = e.K, nrg = (rows + 7) >> 3, k00 = t.chunk * (CKB / S::ELEM);
    const int total = ((t.rows + 7) >> 3) * nq * 8, inv = (65536 + nq - 1) / nq;
    const int64_t rs2 = e.rs2, ks2 = e.ks2;
    char *dst0 = g.dst[op] + e.dst_off + int64_t(t.chunk) * nrg * (8 * S::NC * CKB);
    // row and 16-byte column of core matrix row i
    auto place = [&](int i, int &row, int &core) {
        const int u = i >> 3, rg = (u * inv) >> 16;  // u / nq, u < 2^14
        core = u - rg * nq;
        row = t.row0 + rg * 8 + (i & 7);
    };
    auto load = [&](int i, double (&d)[EV]) {
        int row, core;
        place(i, row, core);
        const int k = k00 + core * EV;
        const int nk = i < total && row < rows ? K - k : 0;  // elements of this core matrix row within the block
        if (FLAT) {
            const double *__restrict__ p = src + int64_t(row) * rs2 + int64_t(k) * ks2;
#pragma unroll
            for (int v = 0; v < EV; ++v) d[v] = v < nk ? p[v * ks2] : 0.0;
        } else if (e.folded) {
            const int rq = row / e.rd2, kq = k / e.kd2;
            const double *__restrict__ p = src + int64_t(rq) * e.rs1 + int64_t(row - rq * e.rd2) * rs2;
            int k2 = k - kq * e.kd2;
            int64_t off = int64_t(kq) * e.ks1 + int64_t(k2) * ks2;
#pragma unroll
            for (int v = 0; v < EV; ++v) {
                d[v] = v < nk ? p[off] : 0.0;
                off += ks2;
                if (++k2 == e.kd2) {
                    k2 = 0;
                    off += e.ks1 - int64_t(e.kd2) * ks2;
                }
            }
        } else {
            // legs that do not fold: the row-major index over all of them
#pragma unroll
            for (int v = 0; v < EV; ++v) {
                d[v] = 0.0;
                if (v >= nk) continue;
                int64_t rem = int64_t(row) * K + (k + v), so = 0;
#pragma unroll 1
                for (int l = e.rank - 1; l >= 0; --l) {
                    const int64_t q = rem / e.dims[l];
                    so += (rem - q * e.dims[l]) * e.stride[l];
                    rem = q;
                }
                d[v] = src[so];
            }
        }
    };
    // the first elements are on their way while the maximum is formed
    double d0[EV], d1[EV];
    load(threadIdx.x, d0);
    load(threadIdx.x + 256, d1);
    const unsigned long long am = amax_of(g.amax_parts[op], g.parts[op], red);
    if (blockIdx.x == 0) {
        // the GEMM's epilogue reads both maxima
        const unsigned long long other = amax_of(g.amax_parts[1 - op], g.parts[1 - op], red);
        if (threadIdx.x == 0) {
            g.amax[op] = am;
            g.amax[1 - op] = other;
        }
    }
    const int shift = amax_shift(am);
    const bool fast = f64_fast(am, shift);
    const uint32_t rebase = f64_rebase(shift);
    auto store = [&](int i, const double (&d)[EV]) {
        if (i >= total) return;
        int row, core;
        place(i, row, core);
        float x[EV];
        if (fast) {
#pragma unroll
            for (int v = 0; v < EV; ++v) x[v] = f64_to_f32_fast(d[v], rebase);
        } else {
#pragma unroll
            for (int v = 0; v < EV; ++v) x[v] = f64_to_f32_int(d[v], shift);
        }
        uint4 out[S::NC];
        S::split(x, out);
        char *dst = dst0 + int64_t(row >> 3) * (8 * S::NC * kvb) + core * 128 + (row & 7) * 16;
#pragma unroll
        for (int c = 0; c < S::NC; ++c) *reinterpret_cast<uint4 *>(dst + c * 8 * kvb) = out[c];
    };
    store(threadIdx.x, d0);
    store(threadIdx.x + 256, d1);
    for (int i = threadIdx.x + 512; i < total; i += 512) {
        load(i, d0);
        load(i + 256, d1);
        store(i, d0);
        store(i + 256, d1);
    }
}

// What a stage holds, for the MMA thread: up to CKB / 32 <= 4 units of k-steps (3 bits each from
// bit 0), flags, and the tile's N in units of 16.
constexpr uint32_t ST_FIRST = 1u << 12, ST_LAST = 1u << 13, ST_END = 1u << 14;
constexpr int ST_N16 = 16;

// Descriptors of up to 32 tiles of a CTA's list, one per lane.
struct TileRegs {
    int m0, n0, cls, M, N, p0, p1;
    int64_t c_off, add_off;
    __device__ __forceinline__ void fetch(const TcArgs &g, int tile) {
        cls = -1;
        if (tile >= g.ntiles) return;
        const GemmTile t = g.tiles[tile];
        const GemmOut o = g.outs[t.out];
        m0 = t.m0;
        n0 = t.n0;
        cls = t.cls;
        M = o.M;
        N = o.N;
        p0 = o.p0;
        p1 = o.p1;
        c_off = o.c_off;
        add_off = o.add_off;
    }
    __device__ __forceinline__ TileRegs of_lane(int l) const {
        TileRegs r;
        r.m0 = __shfl_sync(0xffffffffu, m0, l);
        r.n0 = __shfl_sync(0xffffffffu, n0, l);
        r.cls = __shfl_sync(0xffffffffu, cls, l);
        r.M = __shfl_sync(0xffffffffu, M, l);
        r.N = __shfl_sync(0xffffffffu, N, l);
        r.p0 = __shfl_sync(0xffffffffu, p0, l);
        r.p1 = __shfl_sync(0xffffffffu, p1, l);
        r.c_off = __shfl_sync(0xffffffffu, c_off, l);
        r.add_off = __shfl_sync(0xffffffffu, add_off, l);
        return r;
    }
};

template <class S, int CKB, int CTAS>
__global__ void __launch_bounds__(TTHREADS, CTAS) k_gemm_tc(TcArgs g, int *err) {
    constexpr int NC = S::NC, NSTAGE = S::NSTAGE, STAGE = stage_bytes(NC, CKB), COPY_BYTES = 128 * CKB;
    constexpr int KS = 32 / S::ELEM, CKU = CKB / 32;  // elements of a k-step, k-steps of a stage
    extern __shared__ __align__(128) char smem[];
    __shared__ uint64_t full[NSTAGE], empty[NSTAGE], acc_full[2], acc_empty[2], drained;
    __shared__ uint32_t stage_word[NSTAGE];
    __shared__ uint32_t tmem_base_sh;
    __shared__ unsigned long long epi_top[4];  // per epilogue warp: largest result
    __shared__ int n_issued, n_consumed;  // stages sent out by the producer, taken by the MMA thread
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // round r of the longest-first tile list, in boustrophedon order across the CTAs, so
    // that every CTA's tiles add up to about the same work
    auto snake_tile = [&](int r) {
        const int64_t G = gridDim.x, b = blockIdx.x;
        const int64_t t = int64_t(r) * G + ((r & 1) ? (G - 1 - b) : b);
        return int(min(t, int64_t(INT32_MAX)));
    };
    const int rounds = (g.ntiles + int(gridDim.x) - 1) / int(gridDim.x);

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_sh)),
                     "r"(2 * TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&acc_full[b], 1);
            mbar_init(&acc_empty[b], 4);  // one arrival per epilogue warp
        }
        mbar_init(&drained, 1);
        asm volatile("fence.mbarrier_init.release.cluster;");
        n_issued = 0;
        n_consumed = 0;
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = tmem_base_sh;

    if (warp == 0) {
        int slot = 0, issued = 0;
        uint32_t phase = 0;  // parity of the ring's current lap
        bool stop = false;
        // lane 0 copies A, lane 1 B
        const bool copies = lane < 2, is_a = lane == 0;
        const char *const base = is_a ? g.A : g.B;
        char *const stage0 = smem + (is_a ? 0 : NC * COPY_BYTES);
        auto wait_slot = [&]() {
            const bool ok = issued < NSTAGE || mbar_wait(&empty[slot], phase ^ 1);
            if (__all_sync(0xffffffffu, ok)) return true;
            if (lane == 0) atomicExch(err, S::ERR);
            stop = true;
            return false;
        };
        auto next_slot = [&]() {
            ++issued;
            if (++slot == NSTAGE) {
                slot = 0;
                phase ^= 1;
            }
        };
        TileRegs mine;
        mine.cls = -1;
        for (int r = 0; r < rounds && !stop; ++r) {
            if ((r & 31) == 0) mine.fetch(g, r + lane < rounds ? snake_tile(r + lane) : INT32_MAX);
            const TileRegs t = mine.of_lane(r & 31);
            if (t.cls != 0) continue;  // past the list, or a tile whose pairs all have K = 0
            const int rga = min(TBM / 8, (t.M - t.m0 + 7) / 8), rgb = min(g.tn / 8, (t.N - t.n0 + 7) / 8);
            const uint32_t row_bytes = uint32_t(NC * 8) * uint32_t(rga + rgb);  // per byte of K
            const uint32_t my_rows = uint32_t(is_a ? rga : rgb) * uint32_t(8 * NC);
            const int64_t my_chunk = int64_t(((is_a ? t.M : t.N) + 7) / 8) * (8 * NC * CKB);
            const int64_t my_first = int64_t(is_a ? t.m0 : t.n0) * NC;
            uint32_t word = (uint32_t(rgb + 1) / 2 << ST_N16) | ST_FIRST;
            int width = 0, nu = 0;  // of the open stage: narrow units wait in it for company
            bool ended = false;     // the tile's last stage has gone out
            const int np = t.p1 - t.p0;
            auto close_stage = [&](uint32_t last) {
                if (lane == 0) {
                    stage_word[slot] = word | last;
                    mbar_arrive(&full[slot]);
                }
                next_slot();
                word &= 0xFu << ST_N16;
                width = nu = 0;
            };
            // the pair of each lane (a batch of 32): offset for this lane's operand and its k-steps
            for (int pb = 0; pb < np && !stop; pb += 32) {
                int64_t a_off = 0, b_off = 0;
                int ksteps = 0;
                if (pb + lane < np) {
                    const GemmPair pr = g.pairs[t.p0 + pb + lane];
                    a_off = pr.a_off;
                    b_off = pr.b_off;
                    ksteps = pr.K / KS + (pr.K % KS != 0);
                }
                for (uint32_t live = __ballot_sync(0xffffffffu, ksteps > 0); live && !stop; live &= live - 1) {
                    const int p = __ffs(int(live)) - 1;
                    const int kp = __shfl_sync(0xffffffffu, ksteps, p);
                    const int64_t ao = __shfl_sync(0xffffffffu, a_off, p), bo = __shfl_sync(0xffffffffu, b_off, p);
                    const char *src = base + (is_a ? ao : bo);
                    int k = 0;
                    if (kp >= CKU) {
                        if (width && !stop) close_stage(0);
                        const bool ends = (live & (live - 1)) == 0 && pb + 32 >= np && kp % CKU == 0;
                        for (; k + CKU <= kp; k += CKU) {
                            if (!wait_slot()) break;
                            if (lane == 0) {
                                stage_word[slot] = word | uint32_t(CKU) | (ends && k + CKU == kp ? ST_LAST : 0u);
                                mbar_arrive_expect_tx(&full[slot], row_bytes * CKB);
                            }
                            __syncwarp();
                            if (copies) bulk_g2s(stage0 + slot * STAGE, src + my_first * CKB, my_rows * CKB, &full[slot]);
                            src += my_chunk;
                            next_slot();
                            word &= 0xFu << ST_N16;
                        }
                        if (stop) break;
                        ended = ends;
                    }
                    const int ku = kp - k, kv = ku * 32;
                    if (ku > 0) {
                        if (width + kv > CKB) close_stage(0);
                        if (width == 0 && !wait_slot()) break;
                        if (lane == 0) mbar_expect_tx_only(&full[slot], row_bytes * uint32_t(kv));
                        __syncwarp();
                        if (copies)
                            bulk_g2s(stage0 + slot * STAGE + width * (128 * NC), src + my_first * kv, my_rows * uint32_t(kv),
                                     &full[slot]);
                        word |= uint32_t(ku) << (3 * nu++);
                        width += kv;
                    }
                }
            }
            __syncwarp();
            if (!stop && !ended && (width || wait_slot())) close_stage(ST_LAST);
        }
        if (!stop && wait_slot()) {
            if (lane == 0) {
                stage_word[slot] = ST_END;
                mbar_arrive(&full[slot]);
            }
            next_slot();
        }
        if (lane == 0) n_issued = issued;
    } else if (warp == 1 && lane == 0) {
        int slot = 0, taken = 0, i = 0;
        uint32_t phase = 0, acc = 0, d = tmem;
        // the descriptors' fixed part; a stage and a k-step only move their start address
        const uint64_t first = make_desc(smem_u32(smem), 0);
        for (;;) {
            if (!mbar_wait(&full[slot], phase)) {
                atomicExch(err, S::ERR + 1);
                break;
            }
            const uint32_t word = *reinterpret_cast<volatile uint32_t *>(&stage_word[slot]);
            if (word & ST_END) {
                ++taken;
                break;
            }
            if (word & ST_FIRST) {
                if (i >= 2 && !mbar_wait(&acc_empty[i & 1], ((i / 2) - 1) & 1)) {
                    atomicExch(err, S::ERR + 1);
                    break;
                }
                d = tmem + uint32_t((i & 1) * TMEM_COLS);
                acc = 0;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t idesc = S::idesc(int((word >> ST_N16) & 15u));
            uint64_t at = first + uint64_t(slot * (STAGE / 16));
            // n k-steps of 32 bytes: a copy of 8 rows takes n * 256 bytes
            auto k_steps = [&](uint64_t from, int n) {
                const uint64_t rows8 = uint64_t(n * (256 / 16));
                from += (rows8 * NC) << 32;
                uint64_t a[NC], b[NC];
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    a[c] = from + c * rows8;
                    b[c] = from + uint64_t(NC * (COPY_BYTES / 16)) + c * rows8;
                }
#pragma unroll
                for (int j = 0; j < CKB / 32; ++j) {
                    if (j >= n) break;
                    S::step(d, a, b, idesc, acc);
                    acc = 1;
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        a[c] += 2 * LBO / 16;
                        b[c] += 2 * LBO / 16;
                    }
                }
            };
            if ((word & 7u) == CKB / 32) {
                k_steps(at, CKB / 32);
            } else {
                for (uint32_t w = word & 0xFFFu; w; w >>= 3) {
                    const uint32_t n = w & 7u;
                    k_steps(at, int(n));
                    at += uint64_t(n * 32 * 128 * NC / 16);
                }
            }
            umma_commit(&empty[slot]);
            if (word & ST_LAST) {
                umma_commit(&acc_full[i & 1]);  // this tile's accumulator is final once its MMAs complete
                ++i;
            }
            ++taken;
            if (++slot == NSTAGE) {
                slot = 0;
                phase ^= 1;
            }
        }
        n_consumed = taken;
        umma_commit(&drained);
    } else if (warp >= 2) {
        // epilogue: the four warps read one TMEM lane quarter (32 rows) each
        const int quarter = warp & 3;
        float *patch = reinterpret_cast<float *>(smem + NSTAGE * STAGE) + quarter * 32 * EPI_PITCH;
        const int shift = amax_shift(g.amax[0]) + amax_shift(g.amax[1]);
        uint32_t top = 0;  // largest |accumulator|, as bits
        int i = 0;
        TileRegs mine;
        mine.cls = -1;
        for (int r = 0; r < rounds; ++r) {
            if ((r & 31) == 0) mine.fetch(g, r + lane < rounds ? snake_tile(r + lane) : INT32_MAX);
            const TileRegs t = mine.of_lane(r & 31);
            if (t.cls < 0) continue;
            const bool have_acc = t.cls == 0;
            const int b = i & 1;
            if (have_acc) {
                int ok = 1;
                if (lane == 0) {
                    ok = mbar_wait(&acc_full[b], (i / 2) & 1) ? 1 : 0;
                    if (!ok) {
                        // a tile of a long K takes longer than one bounded wait (2^23 k-steps, 1.3 s): as many more as
                        // its k-steps can take
                        int64_t steps = 0;
                        for (int p = t.p0; p < t.p1; ++p) steps += (int64_t(g.pairs[p].K) * S::ELEM + 31) / 32;
                        for (int64_t more = steps >> 20; more > 0 && !ok; --more) ok = mbar_wait(&acc_full[b], (i / 2) & 1) ? 1 : 0;
                    }
                }
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {
                    if (lane == 0) atomicExch(err, S::ERR + 1);
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;");
            }
            const bool plain = g.alpha == 1.0 && t.add_off < 0;
            const int row0 = t.m0 + quarter * 32, nr = min(32, t.M - row0), nv = min(g.tn, t.N - t.n0);
            double *const C = g.C + t.c_off + int64_t(row0) * t.N + t.n0;
            const double *const Cadd = t.add_off >= 0 ? g.Cadd + t.add_off + int64_t(row0) * t.N + t.n0 : nullptr;
#pragma unroll 1
            for (int col0 = 0; col0 < nv; col0 += EPI_COLS) {
                if (have_acc) {
                    uint32_t v[EPI_COLS];
                    tmem_load16(v, tmem + (uint32_t(quarter * 32) << 16) + uint32_t(b * TMEM_COLS + col0));
                    __syncwarp();
#pragma unroll
                    for (int j = 0; j < EPI_COLS; ++j) patch[lane * EPI_PITCH + j] = __uint_as_float(v[j]);
                    __syncwarp();
                }
                // The patch's elements in row-major order, 4 x 32 at a time: (x inv) >> 16 is x / w
                // for x < 512, w <= 16.  GB300's FP64 pipe is narrow: the plain case (alpha = 1, no
                // add term) converts with integer operations only; FP64 arithmetic only for
                // tensorgdot's epilogue.
                const int w = min(EPI_COLS, nv - col0), n = nr * w, inv = (65536 + w - 1) / w;
#pragma unroll 1
                for (int x0 = lane; x0 < n; x0 += 128) {
                    float f[4];
                    int64_t at[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int x = min(x0 + 32 * u, n - 1), row = (x * inv) >> 16, col = x - row * w;
                        f[u] = have_acc ? patch[row * EPI_PITCH + col] : 0.0f;
                        at[u] = int64_t(row) * t.N + (col0 + col);
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        if (x0 + 32 * u >= n) break;
                        top = max(top, __float_as_uint(f[u]) & 0x7FFFFFFFu);
                        double val = have_acc ? f32_to_f64_int(f[u], shift) : 0.0;
                        if (!plain) {
                            val *= g.alpha;
                            if (Cadd) val += g.beta * Cadd[at[u]];
                        }
                        C[at[u]] = val;
                    }
                }
            }
            if (have_acc) {
                asm volatile("tcgen05.fence::before_thread_sync;");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[b]);
                ++i;
            }
        }
        // scaling back is monotonic: the largest accumulator is the largest result
        top = __reduce_max_sync(0xffffffffu, top);
        if (lane == 0) epi_top[quarter] = static_cast<unsigned long long>(__double_as_longlong(f32_to_f64_int(__uint_as_float(top), shift)));
    }
    __syncthreads();
    if (tid == 0 && g.amax_out) g.amax_out[blockIdx.x] = max(max(epi_top[0], epi_top[1]), max(epi_top[2], epi_top[3]));
    if (tid == 0) {
        // copies issued but never consumed (only after a timeout) must land before exit, and
        // every MMA must have completed before TMEM is freed
        for (int c = n_consumed; c < n_issued; ++c)
            if (!mbar_wait(&full[c % NSTAGE], (c / NSTAGE) & 1)) atomicExch(err, S::ERR + 1);
        if (!mbar_wait(&drained, 0)) atomicExch(err, S::ERR + 1);
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TMEM_COLS));
    }
}

// the calling thread's error word (one per stream context, so concurrent solves
// on different threads see only their own kernels' status)
int *err_word() {
    Ctx &c = ctx();
    if (!c.tc_err) {
        cuda_check(cudaMalloc(&c.tc_err, sizeof(int)), "cudaMalloc(error word)");
        cuda_check(cudaMemset(c.tc_err, 0, sizeof(int)), "cudaMemset(error word)");
    }
    return c.tc_err;
}

template <class S, int CKB, int CTAS>
void launch_ring(const TcArgs &a) {
    static std::atomic<uint64_t> attr{0};
    constexpr int smem = smem_bytes(S::NC, S::NSTAGE, CKB);
    once_per_device(attr, [] {
        cuda_check(cudaFuncSetAttribute(k_gemm_tc<S, CKB, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem),
                   "tcgen05 GEMM smem attribute");
    });
    // CTAS persistent CTAs an SM; one CTA per tile with the persistent grid switched off
    k_gemm_tc<S, CKB, CTAS><<<gemm_tc_grid(a.ntiles), TTHREADS, smem, ctx().stream>>>(a, err_word());
}

template <class S>
void launch_gemm(const TcArgs &a) {
    if (split_chunk_bytes(a.ntiles) == 128)
        launch_ring<S, 128, 1>(a);
    else
        launch_ring<S, 64, CTAS_PER_SM>(a);
}

}  // namespace

int gemm_tc_grid(int ntiles) { return persistent_gemm() ? std::min(ntiles, CTAS_PER_SM * device_sm_count()) : ntiles; }
int gemm_tile_m() { return TBM; }
int gemm_tile_n(int64_t tiles) { return tiles <= device_sm_count() ? TBN / 2 : TBN; }
int split_copies(int mode) { return mode == GEMM_BF16X3 ? Bf16x3::NC : Tf32x3::NC; }
int split_elem_bytes(int mode) { return mode == GEMM_BF16X3 ? Bf16x3::ELEM : Tf32x3::ELEM; }
// With no more tiles than SMs a CTA has its SM to itself and takes stages of twice the K: half as many
// waits and commits in the chain of a tile.  1 x 1 results over K = 2^20 with 64 bytes and twice the stages 30.0 ms
// (TF32X3), 20.0 with 128.
int split_chunk_bytes(int64_t tiles) { return tiles <= device_sm_count() ? 128 : 64; }

void launch_amax(const AmaxArgs &a) {
    const int n = a.parts[0] + a.parts[1];
    if (n <= 0) return;
    k_amax<<<n, AMAX_THREADS, 0, ctx().stream>>>(a);
    count_launch();
    cuda_check(cudaGetLastError(), "amax kernel launch");
}

template <class S, int CKB>
static void split_with(const SplitArgs &a, unsigned grid, bool flat) {
    if (flat)
        k_split<S, CKB, true><<<grid, 256, 0, ctx().stream>>>(a);
    else
        k_split<S, CKB, false><<<grid, 256, 0, ctx().stream>>>(a);
}
void launch_split(const SplitArgs &a, int64_t ntiles, int mode, int chunk, bool flat) {
    if (ntiles <= 0) return;
    const unsigned grid = unsigned(ntiles);
    if (mode == GEMM_BF16X3)
        chunk == 128 ? split_with<Bf16x3, 128>(a, grid, flat) : split_with<Bf16x3, 64>(a, grid, flat);
    else
        chunk == 128 ? split_with<Tf32x3, 128>(a, grid, flat) : split_with<Tf32x3, 64>(a, grid, flat);
    count_launch();
    cuda_check(cudaGetLastError(), "split kernel launch");
}

void launch_gemm_tc(const TcArgs &a, int mode) {
    if (mode != GEMM_TF32X3 && mode != GEMM_BF16X3) fail(ERR_INVALID_ARGUMENT, "unknown tensor-core GEMM mode");
    if (a.ntiles <= 0) return;
    if (mode == GEMM_BF16X3)
        launch_gemm<Bf16x3>(a);
    else
        launch_gemm<Tf32x3>(a);
    count_launch();
    ctx().tc_used = true;
    cuda_check(cudaGetLastError(), "tcgen05 GEMM launch");
}

// Non-zero when a tensor-core kernel hit a bounded wait (read and cleared; synchronises).
int tc_error_check() {
    Ctx &c = ctx();
    if (!c.tc_used) return 0;
    c.tc_used = false;
    int h = 0;
    cuda_check(cudaMemcpyAsync(&h, err_word(), sizeof(int), cudaMemcpyDeviceToHost, c.stream), "read error word");
    cuda_check(cudaStreamSynchronize(c.stream), "cudaStreamSynchronize");
    if (h) cuda_check(cudaMemsetAsync(err_word(), 0, sizeof(int), c.stream), "clear error word");
    return h;
}

}  // namespace qtt
