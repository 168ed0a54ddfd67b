// Launch wrappers between the host layer and the CUDA kernels.  All tables are
// device pointers prepared by the host planner (uploaded through the staging
// ring); all launches go to the current context stream.
#pragma once
#include <atomic>
#include <cstdint>
#include <memory>
#include <vector>

#include <cuda_runtime.h>

namespace qtt {
struct DevBuf;  // qtt_core.h

// Work over many variable-length segments is cut into chunks of at most
// CHUNK elements that never straddle a segment; one CTA handles one chunk.
constexpr int CHUNK = 2048;
struct Chunk {
    int32_t seg;
    int32_t len;
    int64_t start;  // element offset inside the segment
};

// ------------------------------------------------------------ permute / copy
// Segment = one block: dst[dst_off + e] = src[src_off + sum_d idx_d(e) * stride[d]]
// where idx(e) is the row-major multi-index of e over dims[0..rank).
struct PermEntry {
    int64_t src_off, dst_off;
    int32_t rank, pad;
    int64_t dims[8];
    int64_t stride[8];
};
void launch_permute(const void *src, void *dst, const PermEntry *entries, const Chunk *chunks, int64_t nchunks,
                    int elem_bytes);

// ------------------------------------------------------------ grouped GEMM
// Output block o: C[o] (M x N row-major at c_off) = alpha * sum_{p in [p0,p1)} A_p B_p
//                                                   + beta * Cadd (at add_off, when add_off >= 0).
struct GemmPair {
    int64_t a_off, b_off;
    int32_t K;
    int32_t pad;
};
struct GemmOut {
    int64_t c_off, add_off;
    int32_t M, N;
    int32_t p0, p1;
};
struct GemmTile {
    int32_t out, m0, n0, cls;  // cls: tile class of the FP64 kernel (F64_*)
};
// FP64 pair: the operands in place, rows, columns and K each folded to two strides:
//   A(m, k) = A[a_off + (m / am2) as1 + (m % am2) as2 + (k / k2) ak1 + (k % k2) ak2],
//   B(k, n) = B[b_off + (n / bn2) bs1 + (n % bn2) bs2 + (k / k2) bk1 + (k % k2) bk2],  K = k1 k2.
struct __align__(16) F64Pair {
    int64_t a_off, b_off;
    int32_t k1, k2, ak1, ak2, bk1, bk2;
    int32_t am2, as1, as2, bn2, bs1, bs2;
};
static_assert(sizeof(F64Pair) == 64, "the FP64 GEMM copies pair descriptors in 16-byte pieces");
struct F64Args {
    const double *A;
    const double *B;
    double *C;
    const double *Cadd;
    const F64Pair *pairs;
    const GemmOut *outs;
    const GemmTile *tiles;
    int32_t ntiles;
    int32_t b_strided;  // B's columns are not contiguous: square warps (f64_square)
    double alpha, beta;
};
enum : int32_t { F64_SQUARE = 0, F64_SMALL = 1, F64_TALL = 2, F64_WIDE = 3 };
constexpr int F64_STRIP = 8;  // rows or columns of the short side of a strip
// The tile class of an M x N output block (K: the longest contracted length of its pairs)
// and its tile extents; fine: 16 x 16 instead of 32 x 32 tiles (too few of the latter to
// occupy the SMs evenly: gemm_f64_fine, of the number of 32 x 32 tiles and the mean contracted length).
bool gemm_f64_fine(int64_t square_tiles, double mean_k);
int gemm_f64_class(int64_t M, int64_t N, int64_t K, int *tm, int *tn, bool fine);
void launch_gemm_f64(const F64Args &a);

// Split-precision tensor-core variant (tcgen05).  Both operands are first converted, block
// by block, into "matrix form" split arrays (gemm_tc.cu): `copies` arrays per operand
// (hi / lo TF32, or hi / mid / lo BF16), each rows x K in chunks of split_chunk_bytes() of
// K per row, rows padded to 8 and K to 32 bytes.  Offsets in them are in bytes.
// Every element is scaled by the exact power of two 2^-ilogb(max |x| of the operand) before
// the split, so operands of any magnitude use the FP32 range, and the GEMM epilogue undoes
// the two scales exactly.
struct AmaxArgs {
    const double *x[2];
    int64_t n[2];
    int32_t parts[2];          // CTAs of each operand
    unsigned long long *out;   // one maximum per CTA, operand 0's first
};
void launch_amax(const AmaxArgs &a);
struct SplitEntry {
    int64_t src_off, dst_off;  // source elements; bytes within the operand's split form
    int64_t kpb;               // padded K in bytes
    int32_t operand, rows, K, pad;
    // folded: element (row, k) is at (row / rd2) rs1 + (row % rd2) rs2 + (k / kd2) ks1 + (k % kd2) ks2;
    // otherwise at the row-major index row K + k over dims, with these strides
    int32_t folded, rd2, kd2, rank;
    int64_t rs1, rs2, ks1, ks2;
    int64_t dims[8];
    int64_t stride[8];
};
// One CTA: `rows` rows from row0 (a multiple of 8) of one chunk of K.
struct SplitTile {
    int32_t ent, row0, rows, chunk;
};
struct SplitArgs {
    const double *src[2];
    char *dst[2];
    const SplitEntry *ents;
    const SplitTile *tiles;
    const unsigned long long *amax_parts[2];  // per operand: maxima of its pieces (k_amax's, or a GEMM's amax_out)
    int32_t parts[2];
    unsigned long long *amax;  // receives the two operands' maxima
};
// flat: every entry is folded with rd2 >= rows and kd2 >= K (one stride each)
// chunk: split_chunk_bytes of the GEMM's tiles
void launch_split(const SplitArgs &a, int64_t ntiles, int mode, int chunk, bool flat);
int split_copies(int mode);
int split_elem_bytes(int mode);
int split_chunk_bytes(int64_t tiles);  // bytes of K per row and chunk, for a GEMM of so many tiles
// A pair's a_off / b_off: byte offsets of its blocks in split form; A rows = M,
// B rows = N.  A tile whose pairs all have K = 0 has cls 1, the others 0.
struct TcArgs {
    const char *A, *B;
    const unsigned long long *amax;
    double *C;
    const double *Cadd;
    const GemmPair *pairs;
    const GemmOut *outs;
    const GemmTile *tiles;
    int32_t ntiles;
    int32_t tn;  // columns of a tile: gemm_tile_n
    unsigned long long *amax_out = nullptr;  // not null: one maximum of |C| per CTA (alpha = 1, no add term)
    double alpha, beta;
};
void launch_gemm_tc(const TcArgs &a, int mode);
int gemm_tc_grid(int ntiles);  // its CTAs
int gemm_tile_m();
// Tile columns for a launch of `tiles` tiles of 128 columns: 128, or 64 where those would not
// fill the SMs.
int gemm_tile_n(int64_t tiles);

// ------------------------------------------------------------ elementwise
// A coefficient: mult * (dev ? f(*dev) : 1) with f(x) = x, or f(x) = 1/x when
// invert is set and |x| >= guard (f(x) = 1 below the guard).
struct Coef {
    double mult;
    const double *dev;
    int32_t invert;
    int32_t pad;
    double guard;
};
inline Coef coef_host(double v) { return Coef{v, nullptr, 0, 0, 0.0}; }
// Segment: out[out_off + i] = ca * a[a_off + i] + cb * b[b_off + i]; an offset of -1 reads 0.
struct AxpbySeg {
    int64_t a_off, b_off, out_off;
};
void launch_axpby(const double *a, const double *b, double *out, const AxpbySeg *segs, const Chunk *chunks,
                  int64_t nchunks, Coef ca, Coef cb);
// Segment: sum_i a[a_off + i] * b[b_off + i]; partial sums per chunk then a fixed-order
// reduction into *out (device), so the result is deterministic.
struct DotSeg {
    int64_t a_off, b_off;
};
void launch_dot(const double *a, const double *b, const DotSeg *segs, const Chunk *chunks, int64_t nchunks,
                double *partials, double *out);
// Segment: out[out_off + e] = u[u_off + e] * d[d_off + (e % L)]
struct LastLegSeg {
    int64_t u_off, d_off, out_off, L;
};
void launch_mul_lastleg(const double *u, const double *d, double *out, const LastLegSeg *segs, const Chunk *chunks,
                        int64_t nchunks);
// x[0..n) *= 1/sqrt(sum x^2)   (d /= sqrt(sum(d.pow(2))), sources/dmrg.cpp:188)
void launch_normalize(double *x, int64_t n, double *scratch);
void launch_convert(const void *src, void *dst, int64_t n, int src_f64, int dst_f64);

// ------------------------------------------------------------ sector decompositions
// Sector s: m x n matrix A; the work matrix W (p x q, column-major, p >= q) is A when
// m >= n, A^T otherwise.  Offsets are element offsets into the work, rotation,
// left-vector, right-vector and value buffers.
struct SectorDesc {
    int64_t w_off, rot_off, u_off, v_off, s_off;
    int32_t m, n, p, q;
    int32_t trans;  // 1 when W = A^T
    int32_t mode;   // 0: svd, 1: eigh (symmetric input, shifted to positive definite)
    int32_t warm;   // 1: rot holds an orthogonal start V0 and work holds W V0 (warm start)
    int32_t pad;
    double shift;   // eigh: diagonal shift added before the sweeps
};
// Warm start of one sector SVD: work[w_off ..] (p x q, column-major) <- W V0 with V0 the
// q x q orthogonal matrix at v0 (the work type), and rot[rot_off ..] <- V0.  tmp: scratch
// with the work buffer's offsets.  Tiles of 64 x 64 outputs, tile_start = prefix sums.
struct WarmDesc {
    int64_t w_off, rot_off;
    const void *v0;
    int32_t p, q, tile_start, pad;
};
void launch_warm_apply(void *work, void *rot, void *tmp, const WarmDesc *wd, int nwarm, int ntiles, int f32);
// LQ preconditioning (lq.cu): for each listed sector work (p x q, column-major at w_off) <- W Q and
// rot (q x q at rot_off) <- Q, Q orthogonal, W Q lower trapezoidal on its rows by falling norm.
// 2 <= q <= lq_max_q(f32, sectors) <= p.  The other offsets are the launcher's.
struct LqSec {
    int64_t w_off, rot_off, x_off, v_off, o_off;
    int32_t p, q;
};
constexpr size_t LQ_SMEM_MAX = 200 * 1024;
int lq_max_q(int f32, int nsec);
// Tall sectors (p >= 1.5 q) whose largest squared row norm is at most `graded` times the smallest stay as they are, Q the
// identity: their entry in the returned buffer (an int per sector) is 0.
std::shared_ptr<DevBuf> launch_lq(void *work, void *rot, const std::vector<LqSec> &secs, int f32, double graded);
// FP64 refinement of an FP32 sector decomposition (mixed path): from the FP32
// rotations rot32 (at rot_off; rot_size elements in all), vb <- the FP64-orthogonalised rotation
// (two Newton-Schulz steps through va, with g as q x q scratch; exact: wholly in FP64 products), w1 <- w64 vb (at w_off).
// The FP64 Jacobi then runs warm on (w1, vb).
void launch_svd_refine(const float *rot32, int64_t rot_size, const double *w64, double *w1, double *va, double *vb,
                       double *g, const std::vector<SectorDesc> &secs, bool exact);
// out[s_off + j] = squared norm (FP64) of column j of every sector's work matrix (f32:
// FP32 work matrices)
// amax (optional): launch_pack's, by which the norms are scaled back.
void launch_col_norms(const void *W, const SectorDesc *secs, int nsec, int max_q, double *out, int f32,
                      const uint32_t *amax = nullptr);
// Copies dst[dst_off + r] = src[src_off + r], r < len (FP64, or FP32 with f32), one task each: the gather and scatter
// of the kept columns around the restricted FP64 sweeps, and the rotations kept for warm starts.
struct ColCopy {
    int64_t src_off, dst_off;
    int32_t len, pad;
};
void launch_col_copy(const void *src, void *dst, const std::vector<ColCopy> &cols, int f32);
// Vn = Vg R per sector (FP64): Vg (vrows x k at vg_off, column-major), R (k x k at r_off),
// Vn (vrows x k at vn_off).
struct RotProduct {
    int64_t vg_off, r_off, vn_off;
    int32_t vrows, k;
};
void launch_rot_product(const double *vg, const double *r, double *vn, const std::vector<RotProduct> &t);
// Segment = one input block (rows x cols at src_off) placed at rows [r0, r0+rows),
// cols [c0, c0+cols) of sector `sector`.
struct PackEntry {
    int64_t src_off;
    int32_t sector, rows, cols, r0, c0, pad;
};
void launch_zero(double *p, int64_t n);
void check_sector_count(int64_t nsec);  // refuses more sectors than one decomposition takes
// The work / rotation buffers hold float when f32 != 0 (mixed path), else double.
// amax (optional): packing to FP64 takes the largest |x| of each sector there (zero on entry); packing to FP32 scales each
// sector down by the power of two of its own (sector_exponent).
__host__ __device__ inline int sector_exponent(uint32_t high_word) {
    const int e = int(high_word >> 20);
    return e == 0 || e == 0x7FF ? 0 : e - 1023;
}
void launch_pack(const double *src, void *work, const PackEntry *e, const Chunk *chunks, int64_t nchunks,
                 const SectorDesc *sec, int f32, uint32_t *amax = nullptr);
// eigh: symmetrise W from one triangle, then shift the diagonal by the sector's
// Frobenius norm (written back into sec[s].shift) so the matrix is positive definite.
void launch_eigh_prepare(void *work, SectorDesc *sec, int nsec, int upper, int f32);
// Batched one-sided Jacobi over all sectors in one cooperative launch.
// slot_start[nsec+1]: prefix sums of the pairs each sector contributes per step
// ((q + q%2)/2); max_steps_per_sweep = max over sectors of (q + q%2 - 1).
// sweeps_out[s] receives the number of sweeps sector s used; flags holds
// nsec*max_sweeps ints of scratch.
// sum_q: the sectors' total column count (sizes the cooperative grid to the work).
// vwork (optional, jacobi_vwork_bytes): lets the block kernel defer each step's V
// updates to the next step, where CTAs without a block pair run them; without it
// every CTA updates V right after its block pair.
// defl (optional, launch_deflation_thresholds, the work type): per sector, a column
// whose squared norm falls to the threshold or below is set to zero and leaves the
// sweeps (a numerically zero column); null: no deflation.
// exact: FP64 rotation angles from FP64 square roots and divisions, so that
// the basis of equal singular values is that of the plain formulas; otherwise from FP32.
// skip (optional, the work type): per sector, a pair whose squared column norms are both
// below it is not rotated (columns the caller will discard).
// shear_q: FP64 sectors of at least so many columns may rotate by three shears (see rot_apply).
void launch_jacobi(void *work, void *rot, const SectorDesc *sec, const int *slot_start, int nsec,
                   int max_steps_per_sweep, int max_sweeps, int *sweeps_out, int *flags, int f32, int max_p,
                   int64_t sum_q, void *vwork = nullptr, size_t vwork_bytes = 0, const void *defl = nullptr,
                   void *dnorm = nullptr, const void *skip = nullptr, bool exact = false, int shear_q = INT32_MAX);
// thr[s] <- delta^2 ||W_s||_F^2 for every svd sector (0 for eigh), in the work type; norms: the
// squared column norms (launch_col_norms).
void launch_deflation_thresholds(const double *norms, const SectorDesc *sec, int nsec, double delta, void *thr, int f32);
// dnorm (with defl; the work type, sum of q entries at s_off, zero on entry) receives
// the squared norm of every deflated column.
size_t jacobi_vwork_bytes(int nsec, int64_t sum_q, int max_steps_per_sweep, int max_sweeps, int f32);
// Column norms, sort (descending for svd, ascending eigenvalues for eigh),
// normalisation and completion of null columns; writes U (m x k), V (n x k)
// column-major and s (k) per sector in FP64, k = min(m, n).  max_q: largest q;
// scratch: FP64 buffer with the work buffer's element offsets.  complete_cap >= 0
// completes only the first complete_cap null columns of each sector (in value
// order): the caller truncates the others away.  perm_out (sum of q ints at s_off) with
// complete_cap == 0: the factor writes run on many CTAs per sector (max_elems: the
// largest q * (p + q) over the sectors).  norms (optional): work's squared column norms, which one
// CTA per sector otherwise forms.
void launch_finish(const void *work, const void *rot, double *U, double *V, double *s, const SectorDesc *sec,
                   int nsec, int max_q, double *scratch, int f32, int complete_cap = -1, const void *dnorm = nullptr,
                   int *dpos = nullptr, int *perm_out = nullptr, int64_t max_elems = 0,
                   const double *norms = nullptr);
// The same two launches on an explicit stream (no library context involved).
// tune == false never times block widths (no host synchronisation): the width the
// autotuner settled on for the class is used if there is one, else the default.
void launch_jacobi_on(cudaStream_t stream, void *work, void *rot, const SectorDesc *sec, const int *slot_start,
                      int nsec, int max_steps_per_sweep, int max_sweeps, int *sweeps_out, int *flags, int f32,
                      int max_p, int64_t sum_q, void *vwork = nullptr, size_t vwork_bytes = 0,
                      const void *defl = nullptr, void *dnorm = nullptr, bool tune = true,
                      const void *skip = nullptr, bool exact = false, int shear_q = INT32_MAX);
void launch_finish_on(cudaStream_t stream, const void *work, const void *rot, double *U, double *V, double *s,
                      const SectorDesc *sec, int nsec, int max_q, double *scratch, int f32, int complete_cap = -1,
                      const void *dnorm = nullptr, int *dpos = nullptr, int *perm_out = nullptr,
                      int64_t max_elems = 0, const double *norms = nullptr);
// Segment = one output block (rows x k, row-major) from a sector factor's rows, a block or a run of values:
// dst[i k + j] = src[i rs + j cs].
struct ScatterEntry {
    const double *src;  // element (row, column) of the block: src[row rs + column cs]
    double *dst;        // row-major, k columns
    int64_t rs, cs;
    int32_t k, pad;
};
void launch_scatter(const ScatterEntry *e, const Chunk *chunks, int64_t nchunks);

// ------------------------------------------------------------ 2x2 Ritz step on device
// s[0]=a0, s[1]=b, s[2]=a1  ->  s[3]=E, s[4]=o, s[5]=n, s[6]=nan flag
// (eig2x2Mat_impl, sources/dmrg.cpp:544-572)
void launch_eig2x2(double *s);
void launch_sqrt(double *x);

}  // namespace qtt
