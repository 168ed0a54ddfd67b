// Block-sparse contraction: the planner and the grouped-GEMM dispatch.
//
// btensor::tensordot (sources/btensor.cpp:1971-2119) permutes every block of
// both operands into matrix form (permute_bl :1843-1894), merge-joins the two
// sorted block lists on the contracted block-index suffix and, per output block,
// runs torch::mm on the first matching pair and addmm_ on the others.  Here the
// merge-join produces the same output block list (bit-exact, same order) plus a
// pair table; the block products of the whole contraction then run as one
// grouped GEMM launch.  Operands whose natural row-major layout already is the
// (free x contracted) or (contracted x free) matrix are read in place (plain or
// transposed access); only a genuinely scattered leg order is packed first.
#include <chrono>
#include <numeric>

#include "contract.h"
#include "kernels.h"
#include "ops_util.h"
#include "qtt_core.h"

namespace qtt {

namespace {
std::vector<int64_t> norm_dims(const std::vector<int64_t> &d, int r) {
    std::vector<int64_t> o(d.size());
    for (size_t i = 0; i < d.size(); ++i) {
        int64_t x = d[i] < 0 ? d[i] + r : d[i];
        if (x < 0 || x >= r) fail(ERR_CHECK, "dimension out of range");
        o[i] = x;
    }
    std::vector<int64_t> s = o;
    std::sort(s.begin(), s.end());
    if (std::adjacent_find(s.begin(), s.end()) != s.end()) fail(ERR_CHECK, "repeated dimension in contraction");
    return o;
}

struct Keyed {
    std::vector<int64_t> key;  // all keys, nblocks x rank
    std::vector<int64_t> id;   // original block of each sorted entry
    int r;
    const int64_t *k(size_t i) const { return key.data() + i * r; }
};

Keyed permuted_sorted(const BT &t, const std::vector<int64_t> &perm) {
    Keyed K;
    K.r = t.rank;
    const int64_t nb = t.nblocks();
    std::vector<int64_t> raw(nb * K.r);
    for (int64_t b = 0; b < nb; ++b)
        for (int i = 0; i < K.r; ++i) raw[b * K.r + i] = t.idx(b)[perm[i]];
    std::vector<int64_t> ord(nb);
    std::iota(ord.begin(), ord.end(), 0);
    std::stable_sort(ord.begin(), ord.end(),
                     [&](int64_t a, int64_t b) { return idx_less(raw.data() + a * K.r, raw.data() + b * K.r, K.r); });
    K.key.resize(nb * K.r);
    for (int64_t k = 0; k < nb; ++k) std::copy(raw.begin() + ord[k] * K.r, raw.begin() + (ord[k] + 1) * K.r, K.key.begin() + k * K.r);
    K.id = ord;
    return K;
}

// runs of equal prefix (length nf); with no contracted leg every block is its own run
std::vector<std::pair<size_t, size_t>> runs(const Keyed &K, int nf, bool singletons) {
    std::vector<std::pair<size_t, size_t>> out;
    size_t n = K.id.size(), i = 0;
    while (i < n) {
        size_t j = i + 1;
        if (!singletons)
            while (j < n && std::equal(K.k(j), K.k(j) + nf, K.k(i))) ++j;
        out.push_back({i, j});
        i = j;
    }
    return out;
}

bool is_identity(const std::vector<int64_t> &p) {
    for (size_t i = 0; i < p.size(); ++i)
        if (p[i] != int64_t(i)) return false;
    return true;
}
}  // namespace

namespace {
void host_join(ContractPlan &P, const BT &A, const BT &B, int dl);
bool host_join_packed(ContractPlan &P, const BT &A, const BT &B, int dl);
void set_operand_modes(ContractPlan &P);

bool device_present() {
    static const bool present = [] {
        int n = 0;
        return cudaGetDeviceCount(&n) == cudaSuccess && n > 0;
    }();
    return present;
}

[[noreturn]] void fail_sections(const ContractPlan &P, int i, bool size) {
    const std::string a = std::to_string(P.dA[i]), b = std::to_string(P.dB[i]);
    if (size)
        fail(ERR_CHECK, "contracted section sizes differ between dim " + a + " of the left tensor and dim " + b +
                            " of the right tensor");
    fail(ERR_CHECK, "contracted conserved numbers need to sum to zero, but there is a violation when contracting dim " +
                        a + " of the left tensor with dim " + b + " of the right tensor");
}
}  // namespace

ContractPlan plan_contraction(const BT &A, const BT &B, const std::vector<int64_t> &dA_in,
                              const std::vector<int64_t> &dB_in) {
    const auto t_start = std::chrono::steady_clock::now();
    // compute_tdot_shape / check_product_compat (btensor.cpp:783-883)
    if (dA_in.size() != dB_in.size()) fail(ERR_CHECK, "both dimension lists should have the same length.");
    if (!(A.g == B.g)) fail(ERR_CHECK, "the two tensors have different type of conserved quantities");
    ContractPlan P;
    P.dA = norm_dims(dA_in, A.rank);
    P.dB = norm_dims(dB_in, B.rank);
    const int dl = int(P.dA.size());
    auto adA = A.addrs(), adB = B.addrs();
    // dimension by dimension: the section count, then every section's charges and size
    auto host_check = [&]() {
        for (int i = 0; i < dl; ++i) {
            int64_t a = P.dA[i], b = P.dB[i];
            if (A.sbd[a] != B.sbd[b])
                fail(ERR_CHECK, "contracted dimensions need to match, but first has " + std::to_string(A.sbd[a]) +
                                    " sections along dim " + std::to_string(a) + "  and second has " +
                                    std::to_string(B.sbd[b]) + " sections along dim " + std::to_string(b));
            for (int64_t s = 0; s < A.sbd[a]; ++s) {
                if (!qeq(qadd(A.cv[adA[a] + s], B.cv[adB[b] + s], A.g), Charge{}, A.g)) fail_sections(P, i, false);
                if (A.ssz[adA[a] + s] != B.ssz[adB[b] + s]) fail_sections(P, i, true);
            }
        }
    };
    bool counts_match = true;
    for (int i = 0; i < dl; ++i) counts_match = counts_match && A.sbd[P.dA[i]] == B.sbd[P.dB[i]];
    const int mode = planner_mode();
    const int64_t nbl = A.nblocks() + B.nblocks();
    // the device planner checks the section charges itself; graph capture (no
    // synchronisation allowed) and machines without a device plan on the host
    const bool want_dev = mode != 0 && dl > 0 && counts_match && A.nblocks() > 0 && B.nblocks() > 0 &&
                          (mode == 1 || nbl >= planner_auto_blocks()) && device_present() && !ctx().capturing;
    if (!want_dev) host_check();
    std::vector<char> cA(A.rank, 0), cB(B.rank, 0);
    for (auto d : P.dA) cA[d] = 1;
    for (auto d : P.dB) cB[d] = 1;
    for (int i = 0; i < A.rank; ++i)
        if (!cA[i]) P.freeA.push_back(i);
    for (int i = 0; i < B.rank; ++i)
        if (!cB[i]) P.freeB.push_back(i);
    std::vector<int64_t> p1 = P.freeA, p2 = P.dB, p2p = P.freeB;
    p1.insert(p1.end(), P.dA.begin(), P.dA.end());
    p2.insert(p2.end(), P.freeB.begin(), P.freeB.end());
    p2p.insert(p2p.end(), P.dB.begin(), P.dB.end());
    P.p1 = p1;
    P.p2p = p2p;
    P.p2 = p2;
    // output structure (compute_tdot_cval_sectSize :1908-1935)
    BT &o = P.out;
    o.g = A.g;
    o.rank = int(P.freeA.size() + P.freeB.size());
    if (o.rank > MAXRANK) fail(ERR_CHECK, "contraction result rank exceeds 8");
    o.dt = (A.dt == F64 || B.dt == F64) ? F64 : F32;
    o.sel = qadd(A.sel, B.sel, A.g);
    for (auto d : P.freeA) {
        o.sbd.push_back(A.sbd[d]);
        for (int64_t s = 0; s < A.sbd[d]; ++s) {
            o.ssz.push_back(A.ssz[adA[d] + s]);
            o.cv.push_back(A.cv[adA[d] + s]);
        }
    }
    for (auto d : P.freeB) {
        o.sbd.push_back(B.sbd[d]);
        for (int64_t s = 0; s < B.sbd[d]; ++s) {
            o.ssz.push_back(B.ssz[adB[d] + s]);
            o.cv.push_back(B.cv[adB[d] + s]);
        }
    }
    int on_device = 0;
    if (want_dev) {
        int bad_dim = 0;
        bool bad_size = false;
        on_device = plan_join_device(P, A, B, &bad_dim, &bad_size);
        if (on_device < 0) fail_sections(P, bad_dim, bad_size);
        if (!on_device) {
            planner_account(2, 0.0);
            host_check();
        }
    }
    if (!on_device && !host_join_packed(P, A, B, dl)) host_join(P, A, B, dl);
    o.boff.assign(P.out_p0.size(), 0);
    o.compact_offsets();
    set_operand_modes(P);
    planner_account(on_device ? 1 : 0,
                    std::chrono::duration<double>(std::chrono::steady_clock::now() - t_start).count());
    return P;
}

namespace {
// A block's legs in the order `perm` packed into one integer, the first leg most significant: integer
// order is the lexicographic order of the permuted indices.
struct KeyBlock {
    uint64_t key;
    int32_t id;
};
int leg_bits(const BT &t, int64_t d) {
    int b = 0;
    while ((int64_t(1) << b) < t.sbd[d]) ++b;
    return b;
}
std::vector<KeyBlock> packed_sorted(const BT &t, const std::vector<int64_t> &perm) {
    const int64_t nb = t.nblocks();
    int bits[MAXRANK];
    for (int i = 0; i < t.rank; ++i) bits[i] = leg_bits(t, perm[i]);
    std::vector<KeyBlock> out(nb);
    bool sorted = true;
    for (int64_t b = 0; b < nb; ++b) {
        const int64_t *ix = t.idx(b);
        uint64_t k = 0;
        for (int i = 0; i < t.rank; ++i) k = k << bits[i] | uint64_t(ix[perm[i]]);
        out[b] = KeyBlock{k, int32_t(b)};
        sorted = sorted && (b == 0 || out[b - 1].key < k);
    }
    if (!sorted) std::sort(out.begin(), out.end(), [](const KeyBlock &x, const KeyBlock &y) { return x.key < y.key; });
    return out;
}

// host_join on packed keys: the same output block list and pair order.  False when the keys do not
// fit 63 bits, or the contracted part 32 (nothing done).
bool host_join_packed(ContractPlan &P, const BT &A, const BT &B, int dl) {
    int abits = 0, bbits = 0, sbits = 0;
    for (int i = 0; i < A.rank; ++i) abits += leg_bits(A, i);
    for (int i = 0; i < B.rank; ++i) bbits += leg_bits(B, i);
    for (int i = 0; i < dl; ++i) sbits += leg_bits(A, P.dA[i]);
    if (abits > 63 || bbits > 63 || sbits > 31 || A.nblocks() > INT32_MAX || B.nblocks() > INT32_MAX) return false;
    BT &o = P.out;
    const std::vector<KeyBlock> ka = packed_sorted(A, P.p1), kb = packed_sorted(B, P.p2p);
    const int64_t na = int64_t(ka.size()), nb = int64_t(kb.size());
    const uint64_t smask = (uint64_t(1) << sbits) - 1;
    // runs of B (equal free prefix) and its entries by (contracted suffix, position): positions follow
    // the runs, so the entries of one suffix are in run order
    std::vector<int32_t> run(nb);
    std::vector<uint64_t> by_suffix(nb);
    for (int64_t i = 0; i < nb; ++i) {
        run[i] = i == 0 ? 0 : run[i - 1] + (kb[i].key >> sbits != kb[i - 1].key >> sbits ? 1 : 0);
        by_suffix[i] = (kb[i].key & smask) << 32 | uint64_t(i);
    }
    std::sort(by_suffix.begin(), by_suffix.end());
    // where each suffix starts, for all of them if they are few
    std::vector<int32_t> first;
    if (sbits <= 14) {
        first.assign((size_t(1) << sbits) + 1, 0);
        for (uint64_t e : by_suffix) ++first[(e >> 32) + 1];
        for (size_t k = 1; k < first.size(); ++k) first[k] += first[k - 1];
    }
    struct Match {
        uint64_t order;  // run of B, then position within the run of A (the suffix order)
        int32_t pos;
    };
    std::vector<Match> m;
    for (int64_t i0 = 0; i0 < na;) {
        int64_t i1 = i0 + 1;
        while (i1 < na && ka[i1].key >> sbits == ka[i0].key >> sbits) ++i1;
        m.clear();
        for (int64_t i = i0; i < i1; ++i) {
            const uint64_t s = ka[i].key & smask;
            int64_t at = first.empty() ? std::lower_bound(by_suffix.begin(), by_suffix.end(), s << 32) - by_suffix.begin()
                                       : first[s];
            for (; at < nb && by_suffix[at] >> 32 == s; ++at) {
                const int32_t pos = int32_t(by_suffix[at] & 0xFFFFFFFFu);
                m.push_back(Match{uint64_t(run[pos]) << 32 | uint64_t(i - i0), pos});
            }
        }
        if (i1 - i0 > 1) std::sort(m.begin(), m.end(), [](const Match &x, const Match &y) { return x.order < y.order; });
        const int64_t *ia = A.idx(ka[i0].id);
        for (size_t k = 0; k < m.size();) {
            size_t e = k;
            P.out_p0.push_back(int64_t(P.pair_a.size()));
            for (; e < m.size() && m[e].order >> 32 == m[k].order >> 32; ++e) {
                P.pair_a.push_back(ka[i0 + int64_t(m[e].order & 0xFFFFFFFFu)].id);
                P.pair_b.push_back(kb[m[e].pos].id);
            }
            P.out_p1.push_back(int64_t(P.pair_a.size()));
            const int64_t *ib = B.idx(kb[m[k].pos].id);
            for (auto d : P.freeA) o.bidx.push_back(ia[d]);
            for (auto d : P.freeB) o.bidx.push_back(ib[d]);
            k = e;
        }
        i0 = i1;
    }
    return true;
}

void host_join(ContractPlan &P, const BT &A, const BT &B, int dl) {
    BT &o = P.out;
    // merge-join (btensor.cpp:1998-2114): for every run of A (equal free prefix) and
    // every run of B, in that nested order, the pairs with equal contracted suffix.
    // Only the runs of B that share a suffix with the run of A can produce pairs, so
    // they are found through a sorted (suffix, run) index of B instead of trying
    // every run pair: the same output block list and pair order, in
    // O(n log n + pairs) instead of O(runs_A x runs_B).
    Keyed t1 = permuted_sorted(A, P.p1), t2 = permuted_sorted(B, P.p2p);
    const int nfa = A.rank - dl, nfb = B.rank - dl;
    auto r1 = runs(t1, nfa, dl == 0), r2 = runs(t2, nfb, dl == 0);
    auto join = [&](const std::pair<size_t, size_t> &ra, const std::pair<size_t, size_t> &rb) {
        size_t ia = ra.first, ib = rb.first;
        size_t first_pair = P.pair_a.size();
        while (ia < ra.second && ib < rb.second) {
            const int64_t *sa = t1.k(ia) + nfa, *sb = t2.k(ib) + nfb;
            if (idx_less(sa, sb, dl))
                ++ia;
            else if (idx_less(sb, sa, dl))
                ++ib;
            else {
                P.pair_a.push_back(t1.id[ia]);
                P.pair_b.push_back(t2.id[ib]);
                ++ia;
                ++ib;
            }
        }
        if (P.pair_a.size() > first_pair) {
            o.bidx.insert(o.bidx.end(), t1.k(ra.first), t1.k(ra.first) + nfa);
            o.bidx.insert(o.bidx.end(), t2.k(rb.first), t2.k(rb.first) + nfb);
            P.out_p0.push_back(int64_t(first_pair));
            P.out_p1.push_back(int64_t(P.pair_a.size()));
        }
    };
    if (dl == 0) {
        for (auto &ra : r1)
            for (auto &rb : r2) join(ra, rb);
    } else {
        // (suffix, run of B) for every block of B, sorted by suffix then run
        std::vector<std::pair<size_t, int32_t>> sidx;  // (entry of t2, run)
        sidx.reserve(t2.id.size());
        for (size_t r = 0; r < r2.size(); ++r)
            for (size_t i = r2[r].first; i < r2[r].second; ++i) sidx.push_back({i, int32_t(r)});
        auto suf2 = [&](size_t i) { return t2.k(i) + nfb; };
        std::sort(sidx.begin(), sidx.end(), [&](const auto &x, const auto &y) {
            if (idx_less(suf2(x.first), suf2(y.first), dl)) return true;
            if (idx_less(suf2(y.first), suf2(x.first), dl)) return false;
            return x.second < y.second;
        });
        std::vector<int32_t> cand;
        for (auto &ra : r1) {
            cand.clear();
            for (size_t ia = ra.first; ia < ra.second; ++ia) {
                const int64_t *s = t1.k(ia) + nfa;
                auto lo = std::lower_bound(sidx.begin(), sidx.end(), s,
                                           [&](const auto &x, const int64_t *key) { return idx_less(suf2(x.first), key, dl); });
                for (auto it = lo; it != sidx.end() && !idx_less(s, suf2(it->first), dl); ++it) cand.push_back(it->second);
            }
            std::sort(cand.begin(), cand.end());
            cand.erase(std::unique(cand.begin(), cand.end()), cand.end());
            for (int32_t rb : cand) join(ra, r2[rb]);
        }
    }
}

void set_operand_modes(ContractPlan &P) {
    // operand layouts
    const std::vector<int64_t> &p1 = P.p1, &p2 = P.p2;
    P.a_mode = is_identity(p1) ? 0 : -1;
    if (P.a_mode < 0) {
        // rotation: contracted legs leading in dims order, free legs trailing in order
        std::vector<int64_t> rot = P.dA;
        rot.insert(rot.end(), P.freeA.begin(), P.freeA.end());
        P.a_mode = is_identity(rot) ? 1 : 2;
    }
    P.b_mode = is_identity(p2) ? 0 : -1;
    if (P.b_mode < 0) {
        std::vector<int64_t> rot = P.freeB;
        rot.insert(rot.end(), P.dB.begin(), P.dB.end());
        P.b_mode = is_identity(rot) ? 1 : 2;
    }
}
}  // namespace

namespace {
// permuted copy of every block of t with permutation perm (compact, block-list order)
BufPtr pack_operand(const BT &t, const std::vector<int64_t> &perm, std::vector<int64_t> &offs) {
    const int r = t.rank;
    const int64_t nb = t.nblocks();
    offs.assign(nb, 0);
    std::vector<PermEntry> ents(nb);
    std::vector<int64_t> lens(nb);
    int64_t o = 0;
    for (int64_t b = 0; b < nb; ++b) {
        int64_t shp[MAXRANK], str[MAXRANK];
        t.block_shape(b, shp);
        int64_t s = 1;
        for (int d = r - 1; d >= 0; --d) {
            str[d] = s;
            s *= shp[d];
        }
        PermEntry &e = ents[b];
        std::memset(&e, 0, sizeof(e));
        e.src_off = t.boff[b];
        e.dst_off = o;
        e.rank = r;
        for (int i = 0; i < r; ++i) {
            e.dims[i] = shp[perm[i]];
            e.stride[i] = str[perm[i]];
        }
        offs[b] = o;
        lens[b] = t.block_numel(b);
        o += lens[b];
    }
    auto buf = dev_alloc(size_t(std::max<int64_t>(o, 1)) * 8);
    auto chunks = make_chunks(lens);
    StatScope sc(ST_PERMUTE, 2.0 * 8.0 * double(o));
    launch_permute(t.data(), buf->p, upload_vec(ents), upload_vec(chunks), int64_t(chunks.size()), 8);
    return buf;
}

int64_t prod_sizes(const BT &t, int64_t b, const std::vector<int64_t> &dims) {
    int64_t shp[MAXRANK];
    t.block_shape(b, shp);
    int64_t p = 1;
    for (auto d : dims) p *= shp[d];
    return p;
}
// the product of the sizes of legs `dims`, for every block
std::vector<int64_t> sizes_of(const BT &t, const std::vector<int64_t> &dims) {
    const auto ad = t.addrs();
    std::vector<int64_t> out(t.nblocks());
    for (int64_t b = 0; b < t.nblocks(); ++b) {
        const int64_t *ix = t.idx(b);
        int64_t p = 1;
        for (auto d : dims) p *= t.ssz[ad[d] + ix[d]];
        out[b] = p;
    }
    return out;
}
}  // namespace

namespace {
// Legs of one block with their strides in that block, folded: legs of size 1 dropped and
// neighbours merged wherever the outer stride is the inner extent times the inner stride
// (of both operands, for the contracted legs).  At most two groups (outer, inner) remain,
// or the block does not fold.
struct Fold {
    int64_t d1 = 1, d2 = 1;          // extents, outer and inner
    int64_t x1 = 0, x2 = 0;          // strides of the first operand
    int64_t y1 = 0, y2 = 0;          // strides of the second (contracted legs)
};
struct FoldLeg {
    int64_t d, x, y;
};
bool fold_legs(const FoldLeg *legs, int n, Fold &f) {
    FoldLeg g[MAXRANK];
    int k = 0;
    for (int i = 0; i < n; ++i) {
        const FoldLeg &l = legs[i];
        if (l.d == 1) continue;
        if (k && g[k - 1].x == l.d * l.x && g[k - 1].y == l.d * l.y)
            g[k - 1] = FoldLeg{g[k - 1].d * l.d, l.x, l.y};
        else
            g[k++] = l;
    }
    if (k > 2) return false;
    f = Fold();
    if (k == 2) {
        f.d1 = g[0].d;
        f.x1 = g[0].x;
        f.y1 = g[0].y;
    }
    if (k) {
        f.d2 = g[k - 1].d;
        f.x2 = g[k - 1].x;
        f.y2 = g[k - 1].y;
    }
    return true;
}

struct Strided {
    int64_t d[MAXRANK], s[MAXRANK];
};
Strided block_strides(const BT &t, int64_t b) {
    Strided r;
    t.block_shape(b, r.d);
    int64_t s = 1;
    for (int i = t.rank - 1; i >= 0; --i) {
        r.s[i] = s;
        s *= r.d[i];
    }
    return r;
}

// Pair descriptors that read both operands where they lie; false when a block's legs do
// not fold to two strides or a stride exceeds 32 bits (the caller packs the operands).
bool f64_pairs_in_place(const ContractPlan &P, const BT &A, const BT &B, std::vector<F64Pair> &out) {
    auto fits = [](int64_t v) { return v <= INT32_MAX; };
    // per block: the folded free legs, and the contracted legs of more than one element (the same
    // ones in both blocks of a pair)
    struct Side {
        int32_t d2, s1, s2, n;
        int64_t d[2], s[2];
    };
    bool narrow = true;  // no block has more than two such legs
    auto side = [&](const BT &t, const std::vector<int64_t> &free, const std::vector<int64_t> &legs, std::vector<Side> &v) {
        v.resize(t.nblocks());
        for (int64_t b = 0; b < t.nblocks(); ++b) {
            const Strided st = block_strides(t, b);
            FoldLeg l[MAXRANK];
            int n = 0;
            for (auto d : free)
                if (st.d[d] != 1) l[n++] = FoldLeg{st.d[d], st.s[d], 0};
            Fold f;
            if (!fold_legs(l, n, f) || !fits(f.d2) || !fits(f.x1) || !fits(f.x2)) return false;
            Side &x = v[b];
            x.d2 = int32_t(std::max<int64_t>(f.d2, 1));
            x.s1 = int32_t(f.x1);
            x.s2 = int32_t(f.x2);
            x.n = 0;
            for (auto d : legs)
                if (st.d[d] != 1) {
                    if (x.n < 2) {
                        x.d[x.n] = st.d[d];
                        x.s[x.n] = st.s[d];
                    }
                    ++x.n;
                }
            narrow = narrow && x.n <= 2;
        }
        return true;
    };
    std::vector<Side> va, vb;
    if (!side(A, P.freeA, P.dA, va) || !side(B, P.freeB, P.dB, vb)) return false;
    out.resize(P.pair_a.size());
    for (size_t k = 0; k < out.size(); ++k) {
        const int64_t ia = P.pair_a[k], ib = P.pair_b[k];
        const Side &x = va[ia], &y = vb[ib];
        Fold c;
        if (x.n == 1) {
            c.d2 = x.d[0];
            c.x2 = x.s[0];
            c.y2 = y.s[0];
        } else if (x.n > 1) {
            FoldLeg l[MAXRANK];
            int n = 0;
            if (narrow) {
                for (; n < 2; ++n) l[n] = FoldLeg{x.d[n], x.s[n], y.s[n]};
            } else {
                const Strided sa = block_strides(A, ia), sb = block_strides(B, ib);
                for (size_t i = 0; i < P.dA.size(); ++i)
                    l[n++] = FoldLeg{sa.d[P.dA[i]], sa.s[P.dA[i]], sb.s[P.dB[i]]};
            }
            if (!fold_legs(l, n, c)) return false;
        }
        if (!fits(c.d1) || !fits(c.d2) || !fits(c.x1) || !fits(c.x2) || !fits(c.y1) || !fits(c.y2)) return false;
        out[k] = F64Pair{A.boff[ia],     B.boff[ib],     int32_t(c.d1),  int32_t(c.d2),  int32_t(c.x1), int32_t(c.x2),
                         int32_t(c.y1),  int32_t(c.y2),  x.d2,           x.s1,           x.s2,          y.d2,
                         y.s1,           y.s2};
    }
    return true;
}

// The blocks of one operand (legs permuted by perm; the first nrow legs form the rows, the
// rest K) as entries and tiles of the split kernel: offs receives the blocks' byte offsets
// in the operand's split form, the return value is its size (a multiple of 128 bytes).
int64_t split_tables(const BT &t, const std::vector<int64_t> &perm, int nrow, int operand, int mode, int64_t ck,
                     std::vector<SplitEntry> &ents, std::vector<SplitTile> &tiles, std::vector<int64_t> &offs) {
    const int64_t nb = t.nblocks(), es = split_elem_bytes(mode);
    offs.assign(nb, 0);
    int64_t o = 0;
    for (int64_t b = 0; b < nb; ++b) {
        const Strided st = block_strides(t, b);
        SplitEntry e{};
        FoldLeg rl[MAXRANK], kl[MAXRANK];
        int64_t rows = 1, K = 1;
        for (int i = 0; i < t.rank; ++i) {
            e.dims[i] = st.d[perm[i]];
            e.stride[i] = st.s[perm[i]];
            (i < nrow ? rl[i] : kl[i - nrow]) = FoldLeg{e.dims[i], e.stride[i], 0};
            (i < nrow ? rows : K) *= e.dims[i];
        }
        if (K > INT32_MAX - 64) fail(ERR_INVALID_ARGUMENT, "contracted dimension too large");
        if (rows > INT32_MAX - 64) fail(ERR_INVALID_ARGUMENT, "block too large");
        Fold fr, fk;
        e.folded = fold_legs(rl, nrow, fr) && fold_legs(kl, t.rank - nrow, fk) ? 1 : 0;
        if (e.folded) {
            e.rd2 = int32_t(std::max<int64_t>(fr.d2, 1));
            e.rs1 = fr.x1;
            e.rs2 = fr.x2;
            e.kd2 = int32_t(std::max<int64_t>(fk.d2, 1));
            e.ks1 = fk.x1;
            e.ks2 = fk.x2;
        }
        e.src_off = t.boff[b];
        e.dst_off = o;
        e.operand = operand;
        e.rank = t.rank;
        e.rows = int32_t(rows);
        e.K = int32_t(K);
        e.kpb = (K * es + 31) & ~int64_t(31);
        offs[b] = o;
        o += ((rows + 7) / 8) * 8 * e.kpb * split_copies(mode);
        // 8192 elements a tile or so: few tiles to list, enough of them to spread
        for (int64_t k0 = 0; k0 < e.kpb; k0 += ck) {
            const int64_t kv = std::min<int64_t>(ck, e.kpb - k0);
            const int64_t step = 64 * std::max<int64_t>(1, 128 * es / kv / 2);
            for (int64_t r0 = 0; r0 < rows; r0 += step)
                tiles.push_back(SplitTile{int32_t(ents.size()), int32_t(r0), int32_t(std::min(step, rows - r0)), int32_t(k0 / ck)});
        }
        ents.push_back(e);
    }
    return std::max<int64_t>(o, 128);
}

// Output blocks by falling total K (ties in block order): their tiles in this order leave the
// cheap ones for the tail of the grid.
std::vector<int32_t> longest_first(const std::vector<GemmOut> &outs, const std::vector<int64_t> &Ks) {
    constexpr uint64_t top = UINT32_MAX;
    std::vector<uint64_t> keys(outs.size());
    for (size_t o = 0; o < outs.size(); ++o) {
        uint64_t total = 0;
        for (int32_t p = outs[o].p0; p < outs[o].p1; ++p) total += uint64_t(Ks[p]);
        keys[o] = (top - std::min(total, top)) << 32 | uint64_t(o);
    }
    std::sort(keys.begin(), keys.end());
    std::vector<int32_t> order(outs.size());
    for (size_t o = 0; o < outs.size(); ++o) order[o] = int32_t(keys[o] & top);
    return order;
}

void contract_f64(const ContractPlan &P, const BT &A, const BT &B, BT &out, const BT *add, double beta, double alpha,
                  const std::vector<GemmOut> &outs, const std::vector<int64_t> &Ks, double flops) {
    std::vector<F64Pair> pairs;
    BufPtr pa, pb;
    const double *Ap = static_cast<const double *>(A.data());
    const double *Bp = static_cast<const double *>(B.data());
    if (!f64_pairs_in_place(P, A, B, pairs)) {
        // matrix form: an operand that is neither (free x contracted) nor its transpose is packed
        std::vector<int64_t> offa, offb;
        const std::vector<int64_t> *oa = &A.boff, *ob = &B.boff;
        if (P.a_mode == 2) {
            pa = pack_operand(A, P.p1, offa);
            Ap = static_cast<const double *>(pa->p);
            oa = &offa;
        }
        if (P.b_mode == 2) {
            pb = pack_operand(B, P.p2, offb);
            Bp = static_cast<const double *>(pb->p);
            ob = &offb;
        }
        pairs.resize(P.pair_a.size());
        for (size_t k = 0; k < pairs.size(); ++k) {
            const int64_t ia = P.pair_a[k], ib = P.pair_b[k];
            const int64_t M = prod_sizes(A, ia, P.freeA), N = prod_sizes(B, ib, P.freeB), K = prod_sizes(A, ia, P.dA);
            if (M > INT32_MAX || N > INT32_MAX || K > INT32_MAX) fail(ERR_INVALID_ARGUMENT, "block too large");
            F64Pair &p = pairs[k];
            std::memset(&p, 0, sizeof(p));
            p.a_off = (*oa)[ia];
            p.b_off = (*ob)[ib];
            p.k1 = 1;
            p.k2 = int32_t(K);
            p.am2 = int32_t(std::max<int64_t>(M, 1));
            p.bn2 = int32_t(std::max<int64_t>(N, 1));
            p.as2 = int32_t(P.a_mode == 1 ? 1 : K);
            p.ak2 = int32_t(P.a_mode == 1 ? M : 1);
            p.bs2 = int32_t(P.b_mode == 1 ? K : 1);
            p.bk2 = int32_t(P.b_mode == 1 ? 1 : N);
        }
    }
    int64_t squares = 0;
    double area = 0;
    for (const GemmOut &o : outs) {
        squares += ((int64_t(o.M) + 31) / 32) * ((int64_t(o.N) + 31) / 32);
        area += double(o.M) * double(o.N);
    }
    const bool fine = gemm_f64_fine(squares, flops / (2.0 * std::max(area, 1.0)));
    std::vector<GemmTile> tiles;
    for (int32_t o : longest_first(outs, Ks)) {
        int64_t kmax = 0;
        for (int32_t p = outs[o].p0; p < outs[o].p1; ++p) kmax = std::max(kmax, Ks[p]);
        int tm, tn;
        const int cls = gemm_f64_class(outs[o].M, outs[o].N, kmax, &tm, &tn, fine);
        for (int64_t m0 = 0; m0 < outs[o].M; m0 += tm)
            for (int64_t n0 = 0; n0 < outs[o].N; n0 += tn)
                tiles.push_back(GemmTile{o, int32_t(m0), int32_t(n0), cls});
    }
    F64Args g;
    g.A = Ap;
    g.B = Bp;
    g.C = static_cast<double *>(out.data());
    g.Cadd = add ? static_cast<const double *>(add->data()) : nullptr;
    const BufPtr tables = upload_many({table(pairs, g.pairs), table(outs, g.outs), table(tiles, g.tiles)});
    g.ntiles = int32_t(tiles.size());
    g.b_strided = !pb && !P.freeB.empty() && P.freeB.back() != B.rank - 1 ? 1 : 0;
    g.alpha = alpha;
    g.beta = beta;
    StatScope sc(ST_GEMM, flops);
    launch_gemm_f64(g);
}
}  // namespace

void run_contraction(const ContractPlan &P, const BT &A, const BT &B, BT &out, const BT *add, double beta,
                     double alpha, const std::vector<int64_t> *add_block, const Maxima *a_max, Maxima *c_max) {
    require_f64(A);
    require_f64(B);
    const int64_t nout = int64_t(P.out_p0.size());
    if (nout == 0) return;
    const int mode = gemm_mode();
    const std::vector<int64_t> rows = sizes_of(A, P.freeA), cols = sizes_of(B, P.freeB), depth = sizes_of(A, P.dA);
    std::vector<int64_t> Ks(P.pair_a.size());
    for (size_t k = 0; k < Ks.size(); ++k) Ks[k] = depth[P.pair_a[k]];
    std::vector<GemmOut> outs(nout);
    double flops = 0;
    for (int64_t o = 0; o < nout; ++o) {
        int64_t ia = P.pair_a[P.out_p0[o]], ib = P.pair_b[P.out_p0[o]];
        const int64_t M = rows[ia], N = cols[ib];
        if (M > INT32_MAX || N > INT32_MAX) fail(ERR_INVALID_ARGUMENT, "block too large");
        outs[o].c_off = out.boff[o];
        outs[o].add_off = (add && add_block && (*add_block)[o] >= 0) ? add->boff[(*add_block)[o]] : -1;
        outs[o].M = int32_t(M);
        outs[o].N = int32_t(N);
        outs[o].p0 = int32_t(P.out_p0[o]);
        outs[o].p1 = int32_t(P.out_p1[o]);
        double ksum = 0;
        for (int64_t p = P.out_p0[o]; p < P.out_p1[o]; ++p) ksum += double(Ks[p]);
        flops += 2.0 * double(M) * double(N) * ksum;
    }
    if (mode == GEMM_F64) {
        contract_f64(P, A, B, out, add, beta, alpha, outs, Ks, flops);
        return;
    }
    const int TM = gemm_tile_m();
    auto tiles_of = [&](int tn) {
        int64_t n = 0;
        for (const GemmOut &o : outs) n += ((int64_t(o.M) + TM - 1) / TM) * ((int64_t(o.N) + tn - 1) / tn);
        return n;
    };
    const int TN = gemm_tile_n(tiles_of(128));
    const int chunk = split_chunk_bytes(tiles_of(TN));
    std::vector<SplitEntry> ents;
    std::vector<SplitTile> stiles;
    std::vector<int64_t> offa, offb;
    const int64_t asz = split_tables(A, P.p1, int(P.freeA.size()), 0, mode, chunk, ents, stiles, offa);
    const int64_t bsz = split_tables(B, P.p2p, int(P.freeB.size()), 1, mode, chunk, ents, stiles, offb);
    // one buffer: the two maxima, their per-CTA parts, then the split arrays.  The maxima of an operand that a
    // GEMM has just written come from its epilogue: reading the operand again for them is 8 of the 24 bytes an
    // element that the split moves otherwise.
    AmaxArgs am;
    am.x[0] = static_cast<const double *>(A.data());
    am.x[1] = static_cast<const double *>(B.data());
    am.n[0] = A.nnz;
    am.n[1] = B.nnz;
    for (int i = 0; i < 2; ++i)
        am.parts[i] = int32_t(std::min<int64_t>((am.n[i] + 4095) / 4096, 2 * device_sm_count()));
    const bool known = a_max && a_max->parts > 0;
    if (known) am.parts[0] = 0;
    const int64_t head = (int64_t(2 + am.parts[0] + am.parts[1]) * 8 + 255) & ~int64_t(255);
    BufPtr split = dev_alloc(size_t(head + asz + bsz));
    auto *amax = static_cast<unsigned long long *>(split->p);
    am.out = amax + 2;
    SplitArgs sa;
    for (int i = 0; i < 2; ++i) {
        sa.src[i] = am.x[i];
        sa.parts[i] = am.parts[i];
        sa.amax_parts[i] = am.out + (i ? am.parts[0] : 0);
    }
    if (known) {
        sa.parts[0] = a_max->parts;
        sa.amax_parts[0] = static_cast<const unsigned long long *>(a_max->buf->p);
    }
    sa.dst[0] = static_cast<char *>(split->p) + head;
    sa.dst[1] = sa.dst[0] + asz;
    sa.amax = amax;
    std::vector<GemmPair> pairs(P.pair_a.size());
    for (size_t k = 0; k < pairs.size(); ++k) {
        pairs[k].a_off = offa[P.pair_a[k]];
        pairs[k].b_off = offb[P.pair_b[k]];
        pairs[k].K = int32_t(Ks[k]);
        pairs[k].pad = 0;
    }
    std::vector<GemmTile> tiles;
    for (int32_t o : longest_first(outs, Ks)) {
        bool empty = true;
        for (int32_t p = outs[o].p0; p < outs[o].p1; ++p) empty = empty && Ks[p] == 0;
        for (int64_t m0 = 0; m0 < outs[o].M; m0 += TM)
            for (int64_t n0 = 0; n0 < outs[o].N; n0 += TN)
                tiles.push_back(GemmTile{o, int32_t(m0), int32_t(n0), empty ? 1 : 0});
    }
    TcArgs g;
    g.A = sa.dst[0];
    g.B = sa.dst[1];
    g.amax = amax;
    g.tn = TN;
    g.C = static_cast<double *>(out.data());
    g.Cadd = add ? static_cast<const double *>(add->data()) : nullptr;
    g.ntiles = int32_t(tiles.size());
    g.alpha = alpha;
    g.beta = beta;
    if (c_max && !add && alpha == 1.0) {
        const int grid = gemm_tc_grid(g.ntiles);
        if (grid <= 2 * device_sm_count()) {
            c_max->buf = dev_alloc(size_t(grid) * 8);
            c_max->parts = grid;
            g.amax_out = static_cast<unsigned long long *>(c_max->buf->p);
        }
    }
    BufPtr tables;
    {
        StatScope sc(ST_PACK, (mode == GEMM_BF16X3 ? 14.0 : 16.0) * double(A.nnz + B.nnz));
        launch_amax(am);
        tables = upload_many({table(ents, sa.ents), table(stiles, sa.tiles), table(pairs, g.pairs), table(outs, g.outs),
                              table(tiles, g.tiles)});
        bool flat = true;
        for (const SplitEntry &e : ents) flat = flat && e.folded && e.rd2 >= e.rows && e.kd2 >= e.K;
        launch_split(sa, int64_t(stiles.size()), mode, chunk, flat);
    }
    StatScope sc(ST_GEMM, flops);
    launch_gemm_tc(g, mode);
}

BT tensordot(const BT &a, const BT &b, const std::vector<int64_t> &da, const std::vector<int64_t> &db, const Maxima *a_max,
             Maxima *c_max) {
    ContractPlan P = plan_contraction(a, b, da, db);
    BT out = P.out;
    if (!a.has_data || !b.has_data) {
        if (a.has_data != b.has_data && a.nblocks() && b.nblocks()) fail(ERR_NO_DATA, "mixing structure-only and data btensors");
        return out;
    }
    out.alloc_data();
    run_contraction(P, a, b, out, nullptr, 0.0, 1.0, nullptr, a_max, c_max);
    return out;
}

// beta*add + alpha*tensordot(a, b): blocks of the product that also exist in add
// take the add term in the GEMM epilogue; blocks only in add are scaled copies.
BT tensorgdot(const BT &add, const BT &a, const BT &b, const std::vector<int64_t> &da, const std::vector<int64_t> &db,
              double beta, double alpha) {
    ContractPlan P = plan_contraction(a, b, da, db);
    if (!same_shape(P.out, add)) fail(ERR_INVALID_ARGUMENT, "the add tensor's shape differs from the contraction's output");
    // union of add's blocks and the product's blocks
    BT prod = P.out;
    auto u = union_plan(add, prod);
    BT out = add.shape_only();
    out.bidx = u.idx;
    out.boff.assign(u.a.size(), 0);
    out.compact_offsets();
    if (!a.has_data || !b.has_data || (!add.has_data && add.nblocks())) return out;
    require_f64(add);
    out.alloc_data();
    // product blocks write at the union positions
    std::vector<int64_t> prod_pos(prod.nblocks(), -1), add_of_prod(prod.nblocks(), -1);
    std::vector<AxpbySeg> segs;
    std::vector<int64_t> lens;
    for (size_t k = 0; k < u.a.size(); ++k) {
        if (u.b[k] >= 0) {
            prod_pos[u.b[k]] = int64_t(k);
            add_of_prod[u.b[k]] = u.a[k];
        } else {
            segs.push_back(AxpbySeg{add.boff[u.a[k]], -1, out.boff[k]});
            lens.push_back(out.block_numel(int64_t(k)));
        }
    }
    BT target = prod;  // product structure with offsets into out's buffer
    for (int64_t o = 0; o < prod.nblocks(); ++o) target.boff[o] = out.boff[prod_pos[o]];
    target.buf = out.buf;
    target.has_data = true;
    run_contraction(P, a, b, target, &add, beta, alpha, &add_of_prod);
    if (!segs.empty()) {
        auto chunks = make_chunks(lens);
        launch_axpby(static_cast<const double *>(add.data()), nullptr, static_cast<double *>(out.data()),
                     upload_vec(segs), upload_vec(chunks), int64_t(chunks.size()), coef_host(beta), coef_host(0.0));
    }
    return out;
}

}  // namespace qtt
