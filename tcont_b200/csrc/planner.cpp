// planner.cpp -- see planner.hpp.
#include "planner.hpp"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <sstream>

namespace tcontb {
namespace {

int find_char(const std::string& s, char c)
{
    const size_t p = s.find(c);
    return p == std::string::npos ? -1 : static_cast<int>(p);
}

bool has_duplicates(const std::string& s)
{
    for (size_t i = 0; i < s.size(); ++i)
        for (size_t j = i + 1; j < s.size(); ++j)
            if (s[i] == s[j]) return true;
    return false;
}

int index_of(const std::vector<int>& v, int x)
{
    for (size_t i = 0; i < v.size(); ++i)
        if (v[i] == x) return static_cast<int>(i);
    return -1;
}

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

// Builds the kernel-facing problem from mode strings of C, left and right.
// Returns 0 / 1 (invalid) / 3 (unsupported).
// `parC` / `parL` / `parR`: for a sub-tensor view, the extents of the tensor's modes in the parent it is a view of
// (by position; empty = the tensor is dense).
int build_problem(const std::string& mC, const std::string& mL, const std::string& mR, const std::string& ext_mode,
                  const std::vector<int64_t>& ext_val, int scalar_type, Problem* out, std::string* err,
                  const std::vector<int64_t>& parC = {}, const std::vector<int64_t>& parL = {}, const std::vector<int64_t>& parR = {})
{
    Problem p;
    p.scalar_type = scalar_type;
    auto extent_of = [&](char c) -> int64_t {
        const int i = find_char(ext_mode, c);
        return i < 0 ? -1 : ext_val[static_cast<size_t>(i)];
    };
    for (const std::string* s : {&mC, &mL, &mR}) {
        for (char c : *s) {
            const int64_t e = extent_of(c);
            if (e < 0) {
                *err = std::string("Missing extent for mode: ") + c;
                return 1;
            }
            if (e == 0) {
                *err = std::string("Extent of mode '") + c + "' must be positive";
                return 1;
            }
        }
        if (has_duplicates(*s)) {
            *err = "A mode appears twice in one tensor (traces/diagonals are not expressible)";
            return 3;
        }
        // Element counts are products of caller-supplied 64-bit extents: multiply with an overflow check
        // before anything derives strides, table sizes or allocations from them.
        int64_t n = 1;
        for (char c : *s) {
            const int64_t e = extent_of(c);
            if (e >= (int64_t(1) << 31) || __builtin_mul_overflow(n, e, &n) || n >= (int64_t(1) << 40)) {
                *err = "Tensor too large: extents must stay below 2^31 and a tensor below 2^40 elements";
                return 3;
            }
        }
    }
    // C's stride-1 mode decides which caller operand plays role A.
    p.swapped = !mC.empty() && find_char(mL, mC[0]) < 0 && find_char(mR, mC[0]) >= 0;
    const std::string& mA = p.swapped ? mR : mL;
    const std::string& mB = p.swapped ? mL : mR;

    std::string all;
    for (char c : mC + mA + mB)
        if (find_char(all, c) < 0) all.push_back(c);
    for (char c : all) {
        const bool inC = find_char(mC, c) >= 0, inA = find_char(mA, c) >= 0, inB = find_char(mB, c) >= 0;
        Mode m;
        m.names = std::string(1, c);
        m.extent = extent_of(c);
        if (inC && inA && inB) {
            *err = std::string("Mode '") + c + "' is in C, A and B: batch modes are not supported (the reference rejects them too)";
            return 3;
        }
        if (inC && !inA && !inB) {
            *err = std::string("Mode '") + c + "' of C is in neither input";
            return 3;
        }
        if (!inC && inA != inB) {
            *err = std::string("Mode '") + c + "' is in one input only and not in C (free reductions are not supported)";
            return 3;
        }
        m.group = inC ? (inA ? GROUP_M : GROUP_N) : GROUP_K;
        p.modes.push_back(m);
    }
    auto ids = [&](const std::string& s) {
        std::vector<int> v;
        for (char c : s) v.push_back(find_char(all, c));
        return v;
    };
    p.A = ids(mA);
    p.B = ids(mB);
    p.C = ids(mC);
    // Element strides, mode by mode, before anything is fused: the product of the extents in front of the mode, taken
    // from the parent where the tensor is a view of a larger one.
    const std::vector<int64_t>& parA = p.swapped ? parR : parL;
    const std::vector<int64_t>& parB = p.swapped ? parL : parR;
    auto set_strides = [&](const std::vector<int>& t, const std::vector<int64_t>& parent, int which, int64_t* span) -> bool {
        if (!parent.empty() && parent.size() != t.size()) return false;
        int64_t st = 1;
        for (size_t i = 0; i < t.size(); ++i) {
            Mode& m = p.modes[static_cast<size_t>(t[i])];
            (which == 0 ? m.sA : which == 1 ? m.sB : m.sC) = st;
            const int64_t e = parent.empty() ? m.extent : parent[i];
            if (e < m.extent || e >= (int64_t(1) << 31) || __builtin_mul_overflow(st, e, &st) || st >= (int64_t(1) << 40)) return false;
        }
        *span = st;
        return true;
    };
    int64_t spanA = 1, spanB = 1, spanC = 1;
    if (!set_strides(p.A, parA, 0, &spanA) || !set_strides(p.B, parB, 1, &spanB) || !set_strides(p.C, parC, 2, &spanC)) {
        *err = "Parent extents of a sub-tensor view must be given for every mode, be at least the view's extents and stay below 2^40 elements";
        return 1;
    }
    p.strided = !parC.empty() || !parL.empty() || !parR.empty();
    p.c_strided = !parC.empty();

    // Fuse y into x when y follows x immediately in every tensor that holds them.
    bool fused = true;
    while (fused) {
        fused = false;
        for (size_t x = 0; x < p.modes.size() && !fused; ++x) {
            for (size_t y = 0; y < p.modes.size() && !fused; ++y) {
                if (x == y || p.modes[x].group != p.modes[y].group) continue;
                if (p.modes[x].extent == 0 || p.modes[y].extent == 0) continue;
                bool ok = true;
                int which = 0;
                for (std::vector<int>* t : {&p.A, &p.B, &p.C}) {
                    const int ix = index_of(*t, static_cast<int>(x)), iy = index_of(*t, static_cast<int>(y));
                    if ((ix < 0) != (iy < 0)) ok = false;
                    else if (ix >= 0 && iy != ix + 1) ok = false;
                    else if (ix >= 0) {   // and y must follow x in memory too (a view may have gaps between them)
                        const Mode &mx = p.modes[x], &my = p.modes[y];
                        const int64_t sx = which == 0 ? mx.sA : which == 1 ? mx.sB : mx.sC, sy = which == 0 ? my.sA : which == 1 ? my.sB : my.sC;
                        if (sy != sx * mx.extent) ok = false;
                    }
                    ++which;
                }
                if (!ok) continue;
                p.modes[x].names += p.modes[y].names;
                p.modes[x].extent *= p.modes[y].extent;
                p.modes[y].extent = 0;  // tombstone
                for (std::vector<int>* t : {&p.A, &p.B, &p.C}) {
                    const int iy = index_of(*t, static_cast<int>(y));
                    if (iy >= 0) t->erase(t->begin() + iy);
                }
                fused = true;
            }
        }
    }
    // element counts of the views (what is read, written and computed); spans are what the strides cover
    auto count_of = [&](const std::vector<int>& t) {
        int64_t n = 1;
        for (int id : t) n *= p.modes[static_cast<size_t>(id)].extent;
        return n;
    };
    p.sizeA = count_of(p.A);
    p.sizeB = count_of(p.B);
    p.sizeC = count_of(p.C);
    p.spanA = spanA;
    p.spanB = spanB;
    p.spanC = spanC;

    for (int id : p.C) {
        if (p.modes[static_cast<size_t>(id)].group == GROUP_M) p.M.push_back(id);
        else p.N.push_back(id);
    }
    // K order: follow the operand whose stride-1 mode is contracted, so that operand's loads
    // run along memory; A decides when both or neither are.
    const bool a_kfirst = !p.A.empty() && p.modes[static_cast<size_t>(p.A[0])].group == GROUP_K;
    const bool b_kfirst = !p.B.empty() && p.modes[static_cast<size_t>(p.B[0])].group == GROUP_K;
    const std::vector<int>& korder = (!a_kfirst && b_kfirst) ? p.B : p.A;
    for (int id : korder)
        if (p.modes[static_cast<size_t>(id)].group == GROUP_K) p.K.push_back(id);
    for (int id : p.M) p.Mtot *= p.modes[static_cast<size_t>(id)].extent;
    for (int id : p.N) p.Ntot *= p.modes[static_cast<size_t>(id)].extent;
    for (int id : p.K) p.Ktot *= p.modes[static_cast<size_t>(id)].extent;
    *out = p;
    return 0;
}

// Fills one operand's staging description. `t` = tensor mode list, `rows` = its row modes in C
// order, `tile_rows` = 128 for A, BN for B.
bool stage_operand(const Problem& p, const std::vector<int>& t, const std::vector<int>& rows, bool is_a, int kc_mode,
                   int BK, UmmaOperand* o, std::string* why)
{
    const int elt = p.scalar_type == 1 ? 8 : 4, W = 128 / elt;  // W = elements per 128-byte swizzle row
    o->rank = static_cast<int>(t.size());
    for (int d = 0; d < kMaxTmaRank; ++d) {
        o->ext[d] = 1;
        o->box[d] = 1;
        o->stride[d] = 0;
    }
    const int64_t s = is_a ? p.spanA : p.spanB;  // elements the strides cover (the parent's, for a view)
    for (int d = 0; d < o->rank; ++d) {
        const Mode& m = p.modes[static_cast<size_t>(t[static_cast<size_t>(d)])];
        o->ext[d] = m.extent;
        o->stride[d] = is_a ? m.sA : m.sB;
        if (m.extent >= (int64_t(1) << 31)) {
            *why = "a mode extent does not fit a TMA dimension";
            return false;
        }
        if (d > 0 && (o->stride[d] * elt) % 16 != 0) {
            *why = "a stride is not a multiple of 16 bytes (TMA global strides)";
            return false;
        }
    }
    if (o->rank > 0 && o->stride[0] != 1) {
        *why = "the first mode is not contiguous";
        return false;
    }
    const int64_t pad = (s + 3) / 4 * 4;  // (any multiple of 16 bytes will do)
    for (int d = o->rank; d < kMaxTmaRank; ++d) o->stride[d] = pad;  // padded unit dims
    if (s * elt >= (int64_t(1) << 40)) {
        *why = "tensor too large for TMA strides";
        return false;
    }
    const int first = t[0];
    o->major = p.modes[static_cast<size_t>(first)].group == GROUP_K ? 0 : 1;
    o->kc_dim = index_of(t, kc_mode);
    int slab_mode;
    if (o->major == 1) {
        slab_mode = first;
        o->slab_w = W;
        // FP64: slabs of 8 doubles (64-byte rows, 64-byte swizzle) where 16 would pad the mode by over 8 %
        // (extent 72: 5 x 16 = 80 against 9 x 8)
        const int64_t e = p.modes[static_cast<size_t>(first)].extent;
        if (elt == 8 && double(ceil_div(e, 16) * 16) > 1.08 * double(ceil_div(e, 8) * 8)) o->slab_w = 8;
    } else {
        if (first != kc_mode) {
            *why = "K-major operand whose stride-1 mode is not the chunked K mode";
            return false;
        }
        slab_mode = rows[0];
        o->slab_w = 8;  // refined by the caller once the tile height is known
    }
    o->slab_dim = index_of(t, slab_mode);
    const Mode& sm = p.modes[static_cast<size_t>(slab_mode)];
    o->slab_mode_ext = sm.extent;
    o->row_elem_cstride = sm.sC;
    (void)is_a;
    (void)BK;
    return true;
}

// `lead_mode` >= 0: that row mode becomes digit 0 of the slab index, in front of the chunk digit, so that the
// slabs of a tile are consecutive indices of it (see rows_across_slabs).
void finish_operand(const Problem& p, const std::vector<int>& t, const std::vector<int>& rows, int tile_rows, int BK,
                    const std::vector<int>& kdigits, UmmaOperand* o, int max_slab_rows = 256, int lead_mode = -1)
{
    const int elt = p.scalar_type == 1 ? 8 : 4, W = 128 / elt;
    if (o->major == 0) {
        // K-major: rows per slab = the largest power of two (8..tile height) that pads the slab
        // mode by at most 15 % (TF32, where fewer and larger TMA boxes matter more) or 3 % (FP64,
        // where padded rows cost FP64 tensor time); failing that, the one that pads least.
        const double limit = p.scalar_type == 1 ? 1.03 : 1.15;
        int best = 8;
        double best_waste = 1e30;
        for (int w = 8; w <= tile_rows && w <= max_slab_rows; w *= 2) {
            const double waste = double(ceil_div(o->slab_mode_ext, w) * w) / double(o->slab_mode_ext);
            const bool ok = waste <= limit, best_ok = best_waste <= limit;
            if ((ok && (!best_ok || w > best)) || (!ok && !best_ok && waste < best_waste - 1e-12)) {
                best = w;
                best_waste = waste;
            }
        }
        if (tile_rows / best > 16) best = tile_rows / 16;  // at most 16 slabs per operand tile
        o->slab_w = best;
    }
    o->slabs_per_tile = tile_rows / o->slab_w;
    const int slab_mode = t[static_cast<size_t>(o->slab_dim)];
    o->n_row_digits = 0;
    o->chunk_digit = 0;
    o->total_slabs = 1;
    if (lead_mode >= 0) {
        const Mode& m = p.modes[static_cast<size_t>(lead_mode)];
        o->row_digit_dim[0] = index_of(t, lead_mode);
        o->row_digit_ext[0] = m.extent;
        o->row_digit_cstride[0] = m.sC;
        o->n_row_digits = 1;
        o->chunk_digit = 1;
        o->total_slabs = m.extent;
    }
    {
        const int n = o->n_row_digits++;
        o->row_digit_dim[n] = o->slab_dim;
        o->row_digit_ext[n] = ceil_div(o->slab_mode_ext, o->slab_w);
        o->row_digit_cstride[n] = o->row_elem_cstride * o->slab_w;
        o->total_slabs *= o->row_digit_ext[n];
    }
    for (int id : rows) {
        if (id == slab_mode || id == lead_mode) continue;
        const Mode& m = p.modes[static_cast<size_t>(id)];
        const int n = o->n_row_digits++;
        o->row_digit_dim[n] = index_of(t, id);
        o->row_digit_ext[n] = m.extent;
        o->row_digit_cstride[n] = m.sC;
        o->total_slabs *= m.extent;
    }
    for (int i = 0; i < 3; ++i)
        o->k_digit_dim[i] = i < static_cast<int>(kdigits.size()) ? index_of(t, kdigits[static_cast<size_t>(i)]) : -1;
    if (o->major == 1) {
        o->box[o->slab_dim] = o->slab_w;
        o->box[o->kc_dim] = BK;
        o->slab_bytes = BK * o->slab_w * elt;
    } else {
        o->box[o->kc_dim] = BK;  // = W except for FP64 with a k chunk of 8: 64-byte rows
        o->box[o->slab_dim] = o->slab_w;
        o->slab_bytes = o->slab_w * BK * elt;
    }
    o->slabs_per_op = 1;
    o->k0_scale = BK;
    o->digit0_scale = o->slab_w;
    o->oob_coord = static_cast<int>(ceil_div(o->slab_mode_ext, W) * W);  // (any coordinate past the mode's end)
}

// Merged boxes for an MN-major operand: the slab mode (stride-1, extent a multiple of 32) is
// presented to TMA as two dimensions (32 contiguous elements, extent/32 chunks), ordered
// (lo, chunked K mode, hi, rest...), so that one copy with box {32, BK, g} lands g whole slabs one
// after the other.  Fewer, larger copies: the 4 KB single-slab boxes kept the copy engine busy
// with per-copy overhead (GEMM 8192x8192x4096 on B200: 377 TFLOP/s with 12 copies per stage
// against 615 with 2).  `cta_slabs` = slabs of this operand one CTA stages per K step.
void merge_slabs(UmmaOperand* o, int BK, int cta_slabs)
{
    const int W = o->slab_w;  // 32 floats or 16 doubles
    if (o->major != 1 || o->rank > kMaxTmaRank - 1 || o->slab_dim != 0 || o->slab_mode_ext % W || o->slabs_per_op > 1) return;
    const int64_t chunks = o->slab_mode_ext / W;
    // (with no other row digit a box may run over the last chunk: what lies past it is zero-filled like any slab past the tensor)
    int g = 1;
    while (g * 2 <= cta_slabs && (chunks % (g * 2) == 0 || o->n_row_digits == 1) && cta_slabs % (g * 2) == 0) g *= 2;
    if (g <= 1) return;
    UmmaOperand n = *o;
    int map[kMaxTmaRank];
    for (int d = 0; d < kMaxTmaRank; ++d) map[d] = -1;
    n.ext[0] = W; n.stride[0] = 1;
    n.ext[1] = o->ext[o->kc_dim]; n.stride[1] = o->stride[o->kc_dim];
    n.ext[2] = chunks; n.stride[2] = W;
    map[0] = 2;
    map[o->kc_dim] = 1;
    int next = 3;
    for (int d = 1; d < o->rank; ++d) {
        if (d == o->kc_dim) continue;
        n.ext[next] = o->ext[d];
        n.stride[next] = o->stride[d];
        map[d] = next++;
    }
    const int64_t total = o->stride[kMaxTmaRank - 1];  // padded dims carry the tensor's element count
    for (int d = next; d < kMaxTmaRank; ++d) { n.ext[d] = 1; n.stride[d] = total; }
    n.rank = o->rank + 1;
    for (int d = 0; d < kMaxTmaRank; ++d) n.box[d] = 1;
    n.box[0] = W; n.box[1] = BK; n.box[2] = g;
    n.slab_dim = 2;
    n.kc_dim = 1;
    for (int i = 0; i < o->n_row_digits; ++i) n.row_digit_dim[i] = map[o->row_digit_dim[i]];
    for (int i = 0; i < 3; ++i) n.k_digit_dim[i] = o->k_digit_dim[i] >= 0 ? map[o->k_digit_dim[i]] : -1;
    n.slabs_per_op = g;
    n.digit0_scale = 1;
    n.oob_coord = static_cast<int>(chunks);
    *o = n;
}

// How much slabs of 16 or 8 doubles pad a stride-1 mode of extent e.
double slab_padding_f64(int64_t e)
{
    return double(std::min(ceil_div(e, 16) * 16, ceil_div(e, 8) * 8)) / double(e);
}

// K-major operand with a k chunk of 64 (two 128-byte rows of k per tile row): the chunked mode is shown to TMA
// as two dimensions (32 contiguous elements, extent / 32 chunks), the chunk dimension last, so that ONE copy
// with box {32, rows, ..., 2} lands the two 32-wide K chunks of the slab one after the other, each a canonical
// K-major tile of `rows` x 128 bytes.  Needs a free tensor-map dimension, an extent that is a multiple of 32
// (a ragged last chunk would read the next row's elements instead of zeros) and one slab per CTA (the rows of
// a chunk must be contiguous in shared memory for the MMA descriptor).
bool chunk_kmajor(UmmaOperand* o, int BK, int cta_slabs)
{
    if (o->major != 0 || BK <= 32) return true;
    if (o->rank >= kMaxTmaRank || o->kc_dim != 0 || o->ext[0] % 32 || cta_slabs != 1) return false;
    const int r = o->rank;
    o->ext[r] = o->ext[0] / 32;
    o->stride[r] = 32;
    o->box[r] = BK / 32;
    o->ext[0] = 32;
    o->box[0] = 32;
    o->rank = r + 1;
    o->k_digit_dim[0] = r;
    o->k0_scale = BK / 32;
    return true;
}

void plan_umma_impl(const Problem& p_in, const CostTable& cost, UmmaSpec* u, int bk_request, bool fuse_rows, bool narrow = false)
{
    u->eligible = false;
    const bool f64 = p_in.scalar_type == 1;
    // Operand-level row fusion (FP64 kernel, whose epilogue takes every row's C offset from a table): when the
    // stride-1 mode of an MN-major operand is so short that whole slabs would pad it by over 8 % (extent 6:
    // a quarter of every 8-row slab empty) and the next row mode in C's order follows it directly in the
    // operand, the two are staged as ONE mode: TMA sees a single dimension of the fused extent, tiles have no
    // empty rows, and the table builder splits a row's position back into the two C modes.
    Problem p = p_in;
    int64_t split_inner[2] = {0, 0}, split_outer_cstride[2] = {0, 0};
    // Float32 does the same: slabs of 32 pad an extent of 72 by a third.  A K-major operand is fused wherever whole
    // 128-row slabs do not fit its first row mode, because one box of 128 rows then replaces up to 16 small ones.
    if (fuse_rows && !std::getenv("TCONT_NO_ROW_FUSION")) {
        for (int which = 0; which < 2; ++which) {
            std::vector<int>& t = which == 0 ? p.A : p.B;
            std::vector<int>& rows = which == 0 ? p.M : p.N;
            if (t.size() < 3 || rows.size() < 2) continue;
            const int at = index_of(t, rows[0]);
            if (at < 0 || at + 1 >= static_cast<int>(t.size()) || t[static_cast<size_t>(at) + 1] != rows[1]) continue;
            if (f64 && at != 0) continue;
            const Mode m0 = p.modes[static_cast<size_t>(rows[0])], m1 = p.modes[static_cast<size_t>(rows[1])];
            if (f64 ? slab_padding_f64(m0.extent) <= 1.08
                    : at == 0 ? double(ceil_div(m0.extent, 32) * 32) <= 1.08 * double(m0.extent)
                              : p.modes[static_cast<size_t>(t[0])].group != GROUP_K || m0.extent % 128 == 0) continue;
            if ((which == 0 ? m1.sA : m1.sB) != (which == 0 ? m0.sA : m0.sB) * m0.extent) continue;  // (a view with a gap between them)
            Mode f;
            f.names = m0.names + m1.names;
            f.extent = m0.extent * m1.extent;
            f.group = m0.group;
            f.sA = m0.sA;
            f.sB = m0.sB;
            f.sC = m0.sC;
            const int id = static_cast<int>(p.modes.size());
            p.modes.push_back(f);
            split_inner[which] = m0.extent;
            split_outer_cstride[which] = m1.sC;
            t[static_cast<size_t>(at)] = id;
            t.erase(t.begin() + at + 1);
            rows[0] = id;
            rows.erase(rows.begin() + 1);
        }
    }
    const int elt = f64 ? 8 : 4, W = 128 / elt;
    u->elt = elt;
    if (const char* k = std::getenv("TCONT_KERNEL")) {
        // Debug switch: TCONT_KERNEL=gather keeps FP64 on the cp.async gather kernel.
        if (f64 && std::strcmp(k, "gather") == 0) { u->why_not = "disabled by TCONT_KERNEL=gather"; return; }
        // Debug switch: TCONT_KERNEL=simt keeps Float32 contractions on the CUDA-core kernel.
        if (std::strcmp(k, "simt") == 0) { u->why_not = "disabled by TCONT_KERNEL=simt"; return; }
    }
    if (p.A.size() < 2 || p.B.size() < 2 || p.A.size() > kMaxTmaRank || p.B.size() > kMaxTmaRank) {
        u->why_not = "operand rank outside 2..5 after fusion";
        return;
    }
    if (p.M.empty() || p.N.empty() || p.K.empty() || p.K.size() > 3) {
        u->why_not = "needs M, N and 1..3 K modes";
        return;
    }
    const bool a_kmajor = p.modes[static_cast<size_t>(p.A[0])].group == GROUP_K;
    const bool b_kmajor = p.modes[static_cast<size_t>(p.B[0])].group == GROUP_K;
    int kc;
    if (a_kmajor && b_kmajor) {
        if (p.A[0] != p.B[0]) { u->why_not = "both operands K-major on different modes"; return; }
        kc = p.A[0];
    } else if (a_kmajor) kc = p.A[0];
    else if (b_kmajor) kc = p.B[0];
    else {
        // Both operands MN-major: any contracted mode may be the one cut into BK-row chunks.  The
        // rows of a TMA box are one stride of that mode apart; far-apart rows (a slow mode) cost
        // DRAM-page and TLB locality, and the B tile is up to twice as tall as the A tile, so weigh
        // log2(stride) by the tile height.  (cfg5 on B200: 446 TFLOP/s with B's fast K mode chunked,
        // 274 with A's.)
        kc = p.K[0];
        double best = 1e300;
        for (int id : p.K) {
            const Mode& m = p.modes[static_cast<size_t>(id)];
            const double cost = 128.0 * std::log2(double(m.sA)) + 256.0 * std::log2(double(m.sB));
            if (cost < best) {
                best = cost;
                kc = id;
            }
        }
        // Tuning switch: TCONT_UMMA_KC=<mode letter> picks the contracted mode that is cut into
        // BK-sized chunks when both operands are MN-major (any K mode is legal then).
        if (const char* want = std::getenv("TCONT_UMMA_KC"))
            for (int id : p.K)
                if (p.modes[static_cast<size_t>(id)].names.find(want[0]) != std::string::npos) kc = id;
    }
    const int64_t kc_ext = p.modes[static_cast<size_t>(kc)].extent;
    u->kc_names = p.modes[static_cast<size_t>(kc)].names;
    int BK = W;  // a K-major operand brings 128 bytes of K per row
    // Both operands MN-major: the k chunk may be narrower than a 128-byte row.  FP64 takes 8 instead of
    // 16 where that spares more than 15 % of zero-filled k (24 = 3 x 8 against 2 x 16).
    // (A K-major FP64 operand then has 64-byte rows under the 64-byte swizzle; the tcgen05 kernel keeps
    // 128-byte rows for K-major operands.)
    if (f64) BK = kc_ext <= 8 || double(ceil_div(kc_ext, 16) * 16) > 1.15 * double(ceil_div(kc_ext, 8) * 8) ? 8 : 16;
    else if (!a_kmajor && !b_kmajor) {
        BK = kc_ext <= 8 ? 8 : kc_ext <= 16 ? 16 : 32;
        // chunks of 24 (three MMAs per stage) where 32 would pad the mode by over 15 % and 24 by nothing: extents 24, 72, 120
        if (kc_ext % 24 == 0 && double(ceil_div(kc_ext, 32) * 32) > 1.15 * double(kc_ext) && !std::getenv("TCONT_UMMA_NO_BK24")) BK = 24;
    }
    // A k chunk of 64 (eight MMAs per stage, stages of 64 KB per CTA of a pair): half the barrier round trips and
    // half the copy instructions per flop.  The producer warp needs 700 to 900 cycles per stage for its
    // wait / announce / copy sequence whatever the stage holds, which is more than the 512 cycles four MMAs take
    // and less than the 1 024 of eight.  Only where it pads the chunked mode by at most a tenth more.
    if (!f64 && bk_request == 64 && BK == 32 && kc_ext >= 64 &&
        double(ceil_div(kc_ext, 64) * 64) <= 1.1 * double(ceil_div(kc_ext, 32) * 32))
        BK = 64;
    u->BK = BK;
    std::vector<int> kdigits{kc};
    for (int id : p.K)
        if (id != kc) kdigits.push_back(id);
    u->n_k_digits = static_cast<int>(kdigits.size());
    u->k_iters = 1;
    for (int i = 0; i < 3; ++i) u->k_digit_ext[i] = 1;
    for (size_t i = 0; i < kdigits.size(); ++i) {
        const int64_t e = p.modes[static_cast<size_t>(kdigits[i])].extent;
        u->k_digit_ext[i] = i == 0 ? ceil_div(e, BK) : e;
        u->k_iters *= u->k_digit_ext[i];
    }
    u->k_computed = double(u->k_iters) * BK;
    if (f64 && BK == 16) {   // the FP64 kernel leaves out the second half of a last chunk of eight k or fewer
        const bool half = kc_ext % 16 >= 1 && kc_ext % 16 <= 8;
        u->full_chunks = u->k_digit_ext[0] - (half ? 1 : 0);
        if (half) u->k_computed *= 1.0 - 0.5 / double(u->k_digit_ext[0]);
    }
    if (!stage_operand(p, p.A, p.M, true, kc, BK, &u->a, &u->why_not)) return;
    if (!stage_operand(p, p.B, p.N, false, kc, BK, &u->b, &u->why_not)) return;

    u->BM = 128;
    finish_operand(p, p.A, p.M, u->BM, BK, kdigits, &u->a);
    // Rows across slabs (FP64 kernel): A is MN-major on a mode that is not C's stride-1 mode (reference cases 3,
    // 4, 6-8: C[a,...] from A[d,...,a]).  Rows that run along A's stride-1 mode alone would be stored element by
    // element, and moving a 200-300 MB A through a transpose first costs more than the contraction.  Instead a
    // tile is 8 slabs of 16 rows: 16 consecutive elements of A's stride-1 mode (one 128-byte TMA row) times 8
    // consecutive indices of C's stride-1 mode, fetched by ONE box that spans both modes, and four
    // lanes store the same row of the eight slabs, 64 bytes of C, two slabs each.  Needs C's stride-1 mode behind the
    // chunked contracted mode in A's memory order (the box then lands slab by slab) and an extent that is a
    // multiple of 8 (a tile never wraps to the next chunk).
    int lead_a = -1;
    if (f64 && u->a.major == 1 && u->a.row_elem_cstride != 1 && split_inner[0] == 0 && !p.M.empty() && !std::getenv("TCONT_NO_ROWS_ACROSS_SLABS")) {
        const int c1 = p.M[0];
        const Mode& m1 = p.modes[static_cast<size_t>(c1)];
        const int dim1 = index_of(p.A, c1);
        if (m1.sC == 1 && dim1 > u->a.kc_dim && dim1 != u->a.slab_dim && m1.extent % 8 == 0) {
            lead_a = c1;
            u->a.slab_w = 16;
            finish_operand(p, p.A, p.M, u->BM, BK, kdigits, &u->a, 256, lead_a);
            u->a.box[dim1] = u->a.slabs_per_tile;   // one copy per stage: 8 slabs = 8 indices of C's stride-1 mode
            u->a.slabs_per_op = u->a.slabs_per_tile;
            u->store_across_slabs = true;
        }
    }
    u->tiles_m = ceil_div(u->a.total_slabs, u->a.slabs_per_tile);
    // N tile: the widest of 256/128/64/32 that is not wider than the (padded) N extent needs and
    // still yields at least one tile per SM; otherwise the narrowest admissible one.
    int bn = 32;
    if (f64) {
        // the FP64 kernel has 128 x 64 and 128 x 32 tiles: the narrow one where it pads N by over 15 % less
        UmmaOperand probe = u->b;
        finish_operand(p, p.B, p.N, 32, BK, kdigits, &probe);
        const int64_t padded = probe.total_slabs * probe.slab_w;
        bn = double(ceil_div(padded, 32) * 32) * 1.15 < double(ceil_div(padded, 64) * 64) ? 32 : 64;
        if (narrow) bn = 32;
    } else {
        UmmaOperand probe = u->b;
        finish_operand(p, p.B, p.N, 32, BK, kdigits, &probe);
        const int64_t padded = probe.total_slabs * probe.slab_w;
        int widest = 32;
        while (widest < 256 && widest < padded) widest *= 2;
        bn = widest;
        for (int cand = widest; cand >= 32; cand /= 2) {
            UmmaOperand tmp = u->b;
            finish_operand(p, p.B, p.N, cand, BK, kdigits, &tmp);
            if (tmp.slabs_per_tile < 1) break;
            bn = cand;
            if (u->tiles_m * ceil_div(tmp.total_slabs, tmp.slabs_per_tile) >= cost.num_sms) break;
        }
    }
    u->BN = bn;
    finish_operand(p, p.B, p.N, u->BN, BK, kdigits, &u->b);
    if (u->b.slabs_per_tile < 1 || u->a.slabs_per_tile + u->b.slabs_per_tile > 32) {
        u->why_not = "too many slabs per stage";
        return;
    }
    u->tiles_n = ceil_div(u->b.total_slabs, u->b.slabs_per_tile);
    if (u->tiles_m * u->tiles_n >= (int64_t(1) << 31) || (u->tiles_m + 1) * u->a.slabs_per_tile >= (int64_t(1) << 31) ||
        (u->tiles_n + 1) * u->b.slabs_per_tile >= (int64_t(1) << 31)) {
        u->why_not = "tile or slab count does not fit 32 bits";
        return;
    }
    // Two-CTA pairs (256-row tiles): each CTA stages its own 128 rows of A and half of the B tile,
    // so B must split into an even number of slabs.  TCONT_UMMA_PAIR=1 selects it.
    {
        UmmaOperand b2 = u->b;
        if (b2.major == 0 && b2.slabs_per_tile % 2) finish_operand(p, p.B, p.N, u->BN, BK, kdigits, &b2, u->BN / 2);
        const int64_t tn2 = ceil_div(b2.total_slabs, b2.slabs_per_tile);
        // (a short K loop is output-bound: pairing buys nothing there and costs the cluster handshakes)
        // Measured on B200 the pair kernel does not beat one CTA per tile (GEMM 8192x8192x4096: 580 vs
        // 605 TFLOP/s; cfg5: 455 vs 526): the MMA of a pair reads half of B from the partner SM and issues
        // more slowly, which eats the saving in copies.  It therefore stays opt-in.
        // With a k chunk of 64 the pair is the point: 64 KB per CTA per stage is what the 64 B/clk an SM takes in
        // from L2 delivers in the 1 024 cycles the stage's eight MMAs need, where one CTA per 128 x 256 tile would
        // need 96 KB.  Taken when there are at least two waves of pairs and four stages of k.
        bool pair = false;
        if (f64) b2 = u->b;
        const bool can_pair = !f64 && u->tiles_m >= 2 && b2.slabs_per_tile % 2 == 0;
        if (BK == 64) pair = can_pair && u->BN == 256 && ceil_div(u->tiles_m, 2) * tn2 >= cost.num_sms && u->k_iters >= 4;
        if (const char* e = std::getenv("TCONT_UMMA_PAIR")) {
            if (e[0] == '0') pair = false;
            else if (e[0] == '1') pair = can_pair;
        }
        if (BK == 64 && !pair) {
            u->why_not = "a k chunk of 64 is only used by CTA pairs";
            return;
        }
        if (pair) {
            u->pair = true;
            u->b = b2;
            u->tiles_n = tn2;
        }
    }
    {
        const double a_bytes = double(u->a.slabs_per_tile) * u->a.slab_bytes;
        const double b_bytes = double(u->b.slabs_per_tile) * u->b.slab_bytes;
        // rows of a box that lie in different 2 MB pages
        const bool a_far = u->a.major == 1 && u->a.stride[u->a.kc_dim] * elt >= (int64_t(2) << 20);
        const bool b_far = u->b.major == 1 && u->b.stride[u->b.kc_dim] * elt >= (int64_t(2) << 20);
        u->far_fraction = ((a_far ? a_bytes : 0.0) + (b_far ? b_bytes : 0.0)) / (a_bytes + b_bytes);
    }
    if (!chunk_kmajor(&u->a, BK, u->a.slabs_per_tile) ||
        !chunk_kmajor(&u->b, BK, u->pair ? u->b.slabs_per_tile / 2 : u->b.slabs_per_tile)) {
        u->why_not = "a K-major operand cannot be staged with a k chunk of 64";
        return;
    }
    if (!std::getenv("TCONT_UMMA_NO_MERGE")) {
        merge_slabs(&u->a, BK, u->a.slabs_per_tile);
        merge_slabs(&u->b, BK, u->pair ? u->b.slabs_per_tile / 2 : u->b.slabs_per_tile);
    }
    const int stage_bytes = u->a.slabs_per_tile * u->a.slab_bytes +
                            (u->pair ? u->b.slabs_per_tile / 2 : u->b.slabs_per_tile) * u->b.slab_bytes;
    // both kernels own an SM; the FP64 one stops at eight 24 KB stages
    const int budget = f64 ? 200 * 1024 : 227 * 1024 - 8 * 1024;
    u->stages = std::max(2, std::min(8, budget / stage_bytes));
    if (f64) {   // one ring of stages per consumer group
        const int groups = u->BN == 32 ? 3 : 2;
        if (groups == 3) u->stages = std::max(3, std::min(12, (227 * 1024 - 7 * 1024) / stage_bytes));
        u->stages -= u->stages % groups;
    }
    // One CTA per tile (k chunks of up to 32: a stage is at most four MMAs, 512 cycles): two producer warps take
    // turns stage by stage, because one warp's wait-announce-copy round trip takes 700 to 900 cycles whatever the
    // stage holds (reference cases 13, 15, 21, 24 in TF32: 1.24 to 1.67 times faster; nothing to gain with one k
    // iteration per tile).  CTA pairs keep one producer and stages of 64 k (two producers on half-size stages were
    // measured slower there: 0.297 against 0.248 ms on the 3-D configuration).  TCONT_UMMA_PRODUCERS=1|2 overrides.
    if (!f64 && !u->pair && u->stages >= 4 && u->k_iters >= 2) u->producers = 2;
    if (const char* e = std::getenv("TCONT_UMMA_PRODUCERS"))
        if (!f64) u->producers = std::atoi(e) == 2 && u->stages >= 4 ? 2 : 1;
    if (u->producers == 2) u->stages &= ~1;
    u->smem_bytes = u->stages * stage_bytes + (f64 ? u->BN == 32 ? 6 : 9 : 8) * 1024 + 1024;
    // Split-K: with few waves of tiles and a long contracted extent, cut the k iterations into ranges
    // computed as separate work units (partials summed by a second kernel).  Of the admissible counts
    // (ranges of at least 4 iterations, workspace of at most 512 MB) the one with the smallest estimate
    // wins: arithmetic over the share of the last wave's SMs that have a unit, plus the partials written
    // and read back.  A wave is one unit per SM for the tcgen05 kernel (per SM pair for CTA pairs) and two for the FP64 kernel, which
    // wants a unit for each of its two consumer groups.
    {
        const int64_t tiles = (u->pair ? ceil_div(u->tiles_m, 2) : u->tiles_m) * u->tiles_n;
        const int64_t wave = f64 ? 2 * cost.num_sms : u->pair ? cost.num_sms / 2 : cost.num_sms;
        const double flops = 2.0 * double(u->tiles_m * u->BM) * double(u->tiles_n * u->BN) * double(u->k_iters * u->BK);
        const double rate = (f64 ? cost.dmma_f64_tflops : cost.umma_tf32_tflops) * 1e6;  // flops per microsecond
        // The tcgen05 kernel's ring advances by one stage per `umma_stage_us` at best, whatever the stage holds (the
        // producer's wait-announce-copy round trip): a work unit takes at least its stages times that, which is what
        // a long k loop on narrow tiles costs, not its flops.
        auto estimate = [&](int64_t s) {
            const int64_t units = tiles * s;
            const int64_t rounds = ceil_div(units, wave);
            const double eff = double(units) / double(rounds * wave);
            double t = flops / (rate * eff);
            if (!f64) t = std::max(t, double(rounds) * double(ceil_div(u->k_iters, s)) * cost.umma_stage_us / u->producers);
            return t + (s > 1 ? cost.launch_us + 2.0 * double(s) * double(p.sizeC) * elt / (cost.hbm_gbs * 1e3) : 0.0);
        };
        int64_t splits = 1;
        // (a C that is a view into a larger tensor has no workspace "laid out like C" to add partial tiles up in)
        if (tiles < 4 * wave && u->k_iters >= 8 && !p.c_strided) {
            double best = estimate(1);
            for (int64_t s = 2; s <= std::min<int64_t>(64, u->k_iters / 4); ++s) {
                if (double(s) * double(p.sizeC) * elt > 512.0 * 1024 * 1024) break;  // workspace
                const double e = estimate(s);
                if (e < 0.97 * best) best = e, splits = s;  // (a split has to pay for its second kernel)
            }
        }
        if (const char* e = std::getenv("TCONT_SPLITK")) {
            splits = p.c_strided ? 1 : std::max<int64_t>(1, std::min<int64_t>(std::atoll(e), u->k_iters));
            while (splits > 1 && double(splits) * double(p.sizeC) * elt > 512.0 * 1024 * 1024) --splits;
        }
        u->k_iters_per_split = ceil_div(u->k_iters, splits);
        u->k_splits = static_cast<int>(ceil_div(u->k_iters, u->k_iters_per_split));
    }
    u->raster_group = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(u->tiles_m,
                      std::llround(std::sqrt(double(cost.num_sms) * u->BN / u->BM)))));
    // Tiles across slabs store 64 bytes at a time.  Where the next mode of C is a row mode, neighbouring tile rows continue them, and C
    // leaves the faster the more of those are in work together: all rows of a column of tiles one after the other, as long as their part
    // of A stays in L2 (48 x 32 x 64 x 32 x 32 by 8: 6 rows 192 us, 24 175, 200 138, all 384 130; by 16, 48 in the place of the last 32: 347, 342, 297, 281).
    if (u->store_across_slabs && p.C.size() > 1 && p.modes[static_cast<size_t>(p.C[1])].group == GROUP_M)
        u->raster_group = static_cast<int>(std::min<int64_t>(u->tiles_m, std::max<int64_t>(u->raster_group, (int64_t(16) << 20) / (u->BM * elt * p.Ktot))));
    // Tuning switch: TCONT_UMMA_RASTER=<g> sets the number of tile rows (pair rows for CTA pairs) swept together.
    if (const char* e = std::getenv("TCONT_UMMA_RASTER"))
        u->raster_group = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(u->tiles_m, std::atoll(e))));
    // fused row modes: digit 0 carries no C stride of its own, the kernel splits the position (slab_elem_offset)
    for (int which = 0; which < 2; ++which) {
        UmmaOperand& o = which == 0 ? u->a : u->b;
        if (split_inner[which] > 0) {
            o.split_inner = split_inner[which];
            o.split_outer_cstride = split_outer_cstride[which];
            o.row_digit_cstride[0] = 0;
        }
    }
    if (f64) {
        auto multiples = [&](const UmmaOperand& o, int from_digit, int64_t of) {
            bool ok = o.split_inner == 0 || o.split_outer_cstride % of == 0;
            for (int d = from_digit; d < o.n_row_digits; ++d) ok = ok && o.row_digit_cstride[d] % of == 0;
            return ok;
        };
        for (const int of : {4, 2}) {
            // (across slabs the first digit is C's stride-1 mode, in whole eights, and the elements of a slab lie along another mode)
            const bool rows = u->store_across_slabs ? multiples(u->a, 1, of) && u->a.row_elem_cstride % of == 0
                                                    : multiples(u->a, 0, of) && u->a.row_elem_cstride == 1 && u->a.split_inner % of == 0 && u->a.slab_mode_ext % of == 0;
            if (u->piece < of && rows && multiples(u->b, 0, of) && u->b.row_elem_cstride % of == 0) u->piece = of;
        }
        // (not where a C larger than L2 is stored in pieces of 64 bytes after a short main loop: there the stores bound the time, and they
        //  go faster the slower they come, or with narrow tiles in place of 64 slim columns.  Slim and not, us: k chunks of 16,
        //  16 x 48 x 24 x 24 x 48 by 48 101 / 94.4, 48 x 400 x 24 x 128 by 48 297 / 246, 24 x 400 x 24 x 128 by 32 117 / 99.4 (two groups), 16 x 64 x
        //  32 x 48 x 72 by 16 392 / 298, 72 x 96 x 48 x 128 by 16 118 / 103.  Slim is better with a C of 126 MB, 48 x 32 x 16 x 20 x 32 by 48
        //  73.7 / 83.3; on 24 columns by 16 168 / 170 (454 MB) and by 64 220 / 233 (340 MB); on 48 columns by 32 108 / 118 (315 MB); in k chunks of 8,
        //  24 columns by 40 179 / 173 (340 MB) but 20 by 24 146 / 150 (283 MB); and where a fourth of the rows are padding, as with 24 rows in
        //  slabs of 16, 48 x 32 x 72 x 20 x 24 by 48 275 / 343.  Reading the old values slim is better with three chunks of k, 48 x 400 x 24 x 128 by 48
        //  318 / 346, but not with two, 48 x 32 x 32 x 24 x 48 by 32 309 / 286.)
        const bool stores_bound = u->store_across_slabs && u->BK == 16 && double(p.sizeC) * 8.0 > 150e6 && u->a.total_slabs * u->a.slab_w * 3 < p.Mtot * 4 &&
                                  (u->BN == 64 ? u->k_iters == 1 : u->k_iters == 2 || u->k_iters == 3);
        const bool slim = u->tiles_n == 1 && u->b.major == 0 && u->b.total_slabs * u->b.slab_w <= u->BN / 4 * 3 && !std::getenv("TCONT_NO_SLIM");
        u->slim[0] = slim && !stores_bound;
        u->slim[1] = slim && !(stores_bound && (u->BN == 64 || u->k_iters != 3));
    }
    u->eligible = true;
}

// The tcgen05 kernel is planned twice where that can pay: with a k chunk of 64 on CTA pairs, and, where that
// form does not apply (short or ragged contracted mode, too few tiles, a B tile that does not split), with the
// 32-wide chunk on one CTA per tile.  TCONT_UMMA_BK=32 and TCONT_UMMA_PAIR=0 keep the second form.
// Float32: what cannot be staged without operand-level fusion is not staged with it either.  Fusion makes tiles cheaper; it
// must not take a contraction from IEEE single precision to TF32 (a fused mode can hide a stride TMA does not accept).
void plan_umma(const Problem& p, const CostTable& cost, UmmaSpec* u, bool fuse_rows = true)
{
    if (p.scalar_type != 1) {
        UmmaSpec plain;
        plan_umma_impl(p, cost, &plain, 32, false);
        if (!plain.eligible) {
            *u = plain;
            return;
        }
        const char* bk = std::getenv("TCONT_UMMA_BK");
        const char* pr = std::getenv("TCONT_UMMA_PAIR");
        if (!(bk && std::atoi(bk) == 32) && !(pr && pr[0] == '0')) {
            UmmaSpec v;
            plan_umma_impl(p, cost, &v, 64, fuse_rows);
            if (v.eligible && v.BK == 64) {
                *u = v;
                return;
            }
        }
        UmmaSpec v;
        plan_umma_impl(p, cost, &v, 32, fuse_rows);
        *u = v.eligible ? v : plain;
        return;
    }
    *u = UmmaSpec();
    plan_umma_impl(p, cost, u, 32, true);
}

// FP64 with short contracted extents: 128 x 32 tiles, three of them in work on an SM, where a block of 128 x 64 tiles has two.  The
// store of a tile then falls into two main loops of others, and old values of C are copied to shared memory while a tile is
// computed, which 64 columns leave no room for.  Decided when route and kernel are (the estimates know 128 x 64 tiles).  Measured,
// 9216 x 4096 by K, us, 64 and 32 columns: K 8 55 and 48, K 24 81 and 74, K 48 125 and 120, K 96 226 and 221, K 192 433 and 426;
// 4096 x 4096 x 1024 976 and 997.  Accumulating: K 24 168 and 113, K 96 305 and 263, K 192 487 and 472; with rows along C K 24 124
// and 121, K 72 229 and 217, K 96 261 and 267, K 128 325 and 337; in k chunks of 8 4096 x 4096 x 64 86 and 94.  Not with slabs of 8 rows of A: their 64-byte rows are loaded with bank
// conflicts, which half as many columns a fragment do not hide (5184^3, 72 x 72 rows: 8 236 and 13 138).
UmmaSpec narrow_tiles(const Problem& p, const CostTable& cost, const UmmaSpec& u)
{
    const char* want = std::getenv("TCONT_DMMA_BN");   // tuning switch: 32 or 64 columns
    const bool short_k = u.k_computed <= (u.store_across_slabs ? 256 : u.BK == 8 ? 32 : 96) && !(u.a.major == 1 && u.a.slab_w == 8);
    UmmaSpec v;
    const bool whole = !u.slim[0] && ceil_div(u.b.total_slabs * u.b.slab_w, 32) * 32 <= u.tiles_n * 64;   // as many columns computed
    if (u.BN != 64 || u.k_splits != 1 || !whole || !(want ? std::atoi(want) == 32 : short_k)) return v;
    plan_umma_impl(p, cost, &v, 32, true, true);
    if (v.k_splits != 1) v.eligible = false;
    return v;
}

// Consumer groups of a block of 128 x 32 tiles, as time with three / time with two (the best of five bursts with pauses between them):
//   as many rounds of tiles either way (1, 2 or 4 tiles a block): two of them copy ahead further and finish a tile sooner.  40 x 4 x 96 x 24
//     by 1000 47.0 / 43.8 us, 3560 x 96 by 120 accumulating 11.5 / 10.3, 32 x 6 x 88 x 32 by 300 accumulating 21.6 / 18.4, 59976 x 8 by 48
//     12.7 / 11.9.  Not in short ranges of k, which end in stores of whole partial tensors (fewer than 12 k iterations: 56 x 8 x 8 x 8
//     by 1792 in 32 17.5 / 17.9, 24 x 8 x 32 x 8 by 2560 in 18 21.8 / 22.1, but 56 x 8 x 16 x 8 by 3584 in 16 27.8 / 26.8)
//   stores in pieces of 8 or 16 bytes: 29 x 19 x 31 x 22 x 23 x 15 by 18 604 / 521, 51 x 30 x 29 x 30 x 49 by 7 217 / 188; reading the old
//     values, in pieces of 8 bytes 402 / 300 and 819 / 707, in pieces of 16 555 / 769 (23 x 23 x 24 .. by 32, 25 x 16 .. by 17, 26 x 12 .. by 14)
//   rows along C, one or two k chunks of 16: 127776 x 88 by 16 23.3 / 21.4, 105984 x 512 by 16 90.0 / 84.1, 78080 x 128 by 32 28.9 / 27.0
//     (but 306904 x 16 by 16 16.5 / 17.4); more of them 67584 x 128 by 48 31.6 / 33.0
//   across slabs the same in one column of tiles, with a C of twice L2 and more: 48 x 32 x 24 x 32 x 48 by 32 211 / 181 (453 MB); with a C of
//     201 MB three are 9 % faster, with 637 MB on 20 columns by 16 3 %, on 48 columns (906 MB, by 32) 12 %
// Elsewhere three: 24 x 42 x 1024 x 32 by 16 across slabs 52.7 / 62.4, 259056 x 32 by 24 accumulating 33.6 / 44.9, 64 x 236 x 1024 by 24
// 33.5 / 37.4, and always where A's slabs and k chunks of 8 meet, whose loads the narrower warp tile repeats twice as often with
// conflicts (72 x 48 x 16 x 16 by 960 70.8 / 105).
void set_dmma_groups(const Problem& p, UmmaSpec* u, const CostTable& cost)
{
    const char* want = std::getenv("TCONT_DMMA_GROUPS");   // tuning switch: 2 or 3
    const bool slabs8 = u->a.major == 1 && u->a.slab_w == 8;
    const int64_t rounds = ceil_div(u->tiles_m * u->tiles_n * u->k_splits, cost.num_sms);
    for (int reads = 0; reads < 2; ++reads) {
        bool two = u->BN == 64;
        if (!two && !u->slim[reads] && !(slabs8 && u->BK == 8)) {
            if (u->k_splits > 1 ? u->k_iters_per_split >= 12 : true) two = rounds <= 2 || rounds == 4;
            if (!u->store_across_slabs && u->piece < (reads ? 2 : 4)) two = true;
            if (!reads && u->k_splits == 1 && u->BK == 16 && u->k_iters <= 2)
                two = two || !u->store_across_slabs || (u->tiles_n == 1 && double(p.sizeC) * 8.0 > 250e6);
        }
        if (want && u->BN == 32 && !u->slim[reads]) two = std::atoi(want) == 2;
        u->groups[reads] = two ? 2 : 3;
    }
}

// Whether launches that read the old values of C take the 128 x 64 tiles although plain ones are faster on narrow ones: rows along C, a C
// a fifth larger than L2 or more.  128 x 64 reads the values a tile ahead from L2, narrow tiles copy them while they compute (K up to 64) or
// ask for them at the end.  32 and 64 columns in us, C of 318 to 480 MB: 19456 x 2048 by 56 193 / 176, 39040 x 1024 by 56 196 / 189,
// 39472 x 1520 by 80 380 / 348, 16096 x 2816 by 80 281 / 269, 31912 x 1880 by 96 439 / 406, and of 165 MB 89008 x 232 by 72 139 / 133; but
// 624896 x 64 by 48 178 / 185, 156160 x 256 by 32 134 / 145, with a C of 135 MB 15424 x 1100 by 64 94.3 / 96.1 and of 80 MB 9728 x 1024 by 80
// 66.5 / 74.3, by 96 74.7 / 78.3.
bool wide_reads(const Problem& p, const UmmaSpec& wide, const UmmaSpec& narrow)
{
    return narrow.eligible && wide.BN == 64 && wide.k_splits == 1 && narrow.k_splits == 1 && !wide.store_across_slabs && wide.k_computed > 48 && double(p.sizeC) * 8.0 > 150e6;
}

// Time of the TMA-fed FP64 kernel in `s` ranges of k, for up to a few rounds of work units.  A block's SM has `groups` units in work: all
// of them together are bound by the FP64 pipe, each by itself by its chain of k iterations (no shorter than the copies of a stage
// take) and its store.  Fitted to 663 (128 x 32) and 446 (128 x 64) launches of 113 contractions of 4 MFLOP to 3 GFLOP in 1 to 48
// ranges: two thirds within 8 %, nine tenths within 15 %.
double split_us(const Problem& p, const UmmaSpec& u, int64_t s, const CostTable& cost)
{
    const bool narrow = u.BN == 32;
    const double setup = narrow ? 3.22 : 3.47, chain_it = narrow ? 0.362 : 0.966, store = narrow ? 1.52 : 2.1, pipe_it = narrow ? 0.614 : 1.2, copy0 = narrow ? 0.178 : -0.656,
                 copy1 = narrow ? 0.035 : 0.067, sum0 = narrow ? 1.46 : 1.59, sum1 = narrow ? 0.188 : 0.192;
    const int groups = narrow ? 3 : 2;
    const double c_mb = double(p.sizeC) * 8e-6, chunk = u.BK / 16.0, copies = double(u.a.slabs_per_tile) / u.a.slabs_per_op + double(u.b.slabs_per_tile) / u.b.slabs_per_op;
    const int64_t per = ceil_div(u.k_iters, s), units = ceil_div(u.tiles_m * u.tiles_n * ceil_div(u.k_iters, per), cost.num_sms);
    const double pipe = double(units * per) * pipe_it * (u.slim[0] ? 0.8 : 1.0) * chunk + store / groups;
    const double chain = double(ceil_div(units, groups)) * (double(per) * std::max(chain_it * chunk, copy0 + copy1 * copies) + store);
    const double us = setup + std::max(pipe, chain) + (s > 1 ? sum0 + (sum1 * c_mb + 0.12) * double(s) : 0.0);
    return std::max(us, setup + (c_mb + (double(p.sizeA) + double(p.sizeB)) * 8e-6) / (narrow ? 4.93 : 4.54));
}

// FP64 with few tiles: 128 x 32 tiles in the number of ranges of k with the smallest estimate, `*us` (eligible = false: none).  More and
// smaller units than the 128 x 64 tiles' even out better over the SMs: 16 x 16 outputs by 13 440 26.4 -> 20.9 us, 20 x 18 tiles by 384
// in three ranges 46.8 -> 42.3, 144 x 1 by 312 33.2 -> 27.2.
UmmaSpec narrow_ranges(const Problem& p, const CostTable& cost, const UmmaSpec& u, double* us)
{
    UmmaSpec v;
    *us = 1e300;
    if (!u.eligible || u.elt != 8 || std::getenv("TCONT_SPLITK") || std::getenv("TCONT_DMMA_BN")) return v;
    if ((u.a.row_elem_cstride != 1 && !u.store_across_slabs) || u.a.slab_mode_ext < 8) return v;   // (stores of single elements)
    // Where A's slabs and k chunks of 8 meet, a stage is 16 to 20 copies of 512 bytes, which three producers wait for each other with, more
    // than the estimate knows, and 64 columns halve: of 20 contractions half were faster on narrow tiles, 40 x 8 x 8 x 8 by 1536 18.6 us of
    // 21.2, half slower, 24 x 56 x 40 x 24 by 384 58.3 of 49.6.  With k chunks of 16 they gain: 72 x 16 x 72 x 64 by 2560 (27 GFLOP, one range
    // instead of three) 788 us of 847, and all but 5 of 48 others, which gain in two consumer groups.
    if (u.BK == 8 && u.a.major == 1 && u.a.slab_w == 8) return v;
    if (u.BN == 32) v = u;
    else plan_umma_impl(p, cost, &v, 32, true, true);
    if (!v.eligible) return v;
    int64_t best = 1;
    for (int64_t s = 1; s <= (p.c_strided ? 1 : std::min<int64_t>(64, std::max<int64_t>(1, v.k_iters / 2))); ++s) {
        if (double(s) * double(p.sizeC) * 8.0 > 512.0 * 1024 * 1024) break;   // workspace
        const double t = split_us(p, v, s, cost);
        if (t < 0.97 * *us) *us = t, best = s;
    }
    v.k_iters_per_split = ceil_div(v.k_iters, best);
    v.k_splits = static_cast<int>(ceil_div(v.k_iters, v.k_iters_per_split));
    return v;
}

std::string perm_modes(const Problem& p, const std::vector<int>& ids)
{
    std::string s;
    for (int id : ids) s += p.modes[static_cast<size_t>(id)].names;
    return s;
}

void fill_transpose(const std::string& src, const std::string& dst, const std::string& ext_mode,
                    const std::vector<int64_t>& ext_val, TransposeSpec* t, const std::vector<int64_t>& src_parent = {}, const std::vector<int64_t>& padded = {})
{
    t->needed = src != dst || !padded.empty();
    t->rank = static_cast<int>(src.size());
    t->elements = t->dst_elements = 1;
    t->strided_src = !src_parent.empty();
    int64_t st = 1;
    for (size_t i = 0; i < src.size(); ++i) {
        t->src_extent[i] = ext_val[static_cast<size_t>(find_char(ext_mode, src[i]))];
        t->elements *= t->src_extent[i];
        t->perm[i] = find_char(src, dst[i]);
        t->dst_extent[i] = padded.empty() ? ext_val[static_cast<size_t>(find_char(ext_mode, dst[i]))] : padded[i];
        t->dst_elements *= t->dst_extent[i];
        t->src_stride[i] = st;   // the source may be a view: strides from its parent's extents
        st *= src_parent.empty() ? t->src_extent[i] : src_parent[i];
    }
}

// Share of the last wave's SMs that have a tile: t tiles on n SMs take ceil(t / n) rounds.
double wave_efficiency(int64_t tiles, int sms)
{
    const int64_t t = std::max<int64_t>(tiles, 1);
    return double(t) / double(ceil_div(t, sms) * sms);
}

// Tile, cluster and form of the gather kernel: the smallest estimate over its tile shapes and 1, 2, 4, 8 or 16 CTAs per tile.
// CTAs spread evenly over the SMs; the CTAs an SM holds pass their k tiles together at the rate of a full GPU
// (throughput), but none faster than one alone (latency), which is what bounds small problems and what a split of k
// shortens.  Measured on 60 contractions of 2 MFLOP to 280 GFLOP with every tile, cluster and form: the choice is within
// 11 % of the best one on average.
// The 128 x 128 Float32 tile in four wide warps instead of eight.  A wide block takes longer to begin and to end, with
// half the threads, the more so in a large cluster, and has to make that good in its range of k.  Old / wide in us, by k per block:
// one block to a tile, 5003 x 3001: 101 108 / 111, 201 194 / 183, 601 513 / 442; clusters of 2, 1401 x 1401: 100 52 / 39, 300 87 / 73;
// of 4, 1801 x 1501: 75 77 / 80, 100 107 / 98; of 8, 701 x 701: 75 39 / 46, 400 170 / 142.  With no more blocks than SMs the one warp
// on each scheduler has its latencies to itself (301 x 301 x 9201 in clusters of 16: 103 / 102), so the old kind stays there.
// 64 x 64 tiles, one block to a tile and few k: direct stores of whole lines (126 x 145 x 95 by 27 10.6 us, 11.3 by way of shared memory).
int float32_form(const GatherSpec& g, const Problem& p, const CostTable& c)
{
    if (g.tile == GATHER_SQUARE && g.cluster == 1 && p.Ktot < 48) return GATHER_FORM_SHORT;
    const int64_t blocks = ceil_div(g.rows, 128) * ceil_div(p.Ntot, 128) * g.cluster, least_k = g.cluster == 1 ? 160 : g.cluster <= 4 ? 96 : 192;
    return g.tile == GATHER_BIG && blocks > c.num_sms && p.Ktot / g.cluster >= least_k ? GATHER_FORM_WIDE : GATHER_FORM_PLAIN;
}

GatherSpec plan_gather(const Problem& p, const CostTable& c, bool count_sectors = true)
{
    const bool f64 = p.scalar_type == 1;
    static const int kTile64[3][3] = {{64, 64, 3}, {128, 32, 2}, {32, 32, 4}};   // BM, BN, CTAs per SM
    static const int kTile32[4][3] = {{64, 64, 4}, {128, 32, 4}, {32, 32, 4}, {128, 128, 2}};
    const auto* kTile = f64 ? kTile64 : kTile32;
    const double elt = f64 ? 8.0 : 4.0;
    GatherSpec best;   // (what runs when no candidate below qualifies: a forced cluster this contraction cannot have, an unusable rate)
    best.rows = p.Mtot;
    best.est_us = 1e300;
    // FP64 sums of this length are off by close to 1e-14 of their norm as one chain of FMAs, and by a fifth of that when cut
    // into ranges.  They stay one chain here only so that results recorded with it do not move by that much; where tiles are
    // few it costs 15 times the time, and the TMA-fed kernel does cut them.
    const bool one_chain = f64 && p.Ktot > 49152;
    // An operand whose stride-1 mode is contracted, but not the first of the contracted modes (those are in the other operand's
    // order): every element of it is fetched as a 32-byte sector of its own, by every tile that needs it.  168 x 192 x 4096
    // FP64, 36 tiles of 32 x 32 in 16 ranges of k: 62 us, 38 of them for 151 MB of such sectors.  Counted where the TMA-fed
    // kernel behind a permutation is the alternative; the gather kernel behind one is not reliably faster (the same
    // contractions: 0.5 to 1.3 times the time).
    auto scattered = [&](const std::vector<int>& t) { return f64 && count_sectors && p.modes[static_cast<size_t>(t[0])].group == GROUP_K && t[0] != p.K[0] ? int64_t(1) : int64_t(0); };
    const int64_t scattered_a = scattered(p.A), scattered_b = scattered(p.B);
    double sector_us = 0;
    const char* force_tile = std::getenv("TCONT_GATHER_TILE");        // tuning switches: 0..3, 1..16 (1 where that many are impossible)
    const char* force_cluster = std::getenv("TCONT_GATHER_CLUSTER");
    const char* force_flat = std::getenv("TCONT_GATHER_FLAT");
    for (int t : {GATHER_BIG, GATHER_SQUARE, GATHER_TALL, GATHER_SMALL}) {   // (of equal estimates the larger tile)
        if (f64 && t == GATHER_BIG) continue;
        if (force_tile && std::atoi(force_tile) != t && std::atoi(force_tile) < (f64 ? 3 : 4)) continue;
        const int64_t bm = kTile[t][0], bn = kTile[t][1];
        GatherSpec g;
        g.tile = t;
        g.rows = p.Mtot;
        // A's stride-1 mode is a row mode, but not C's: a tile of t0 x t1 indices of the two lets both gathers and stores
        // run along memory.  Where C is the larger tensor, t0 = 32 keeps whole 128-byte (256-byte) runs of it; else the
        // least padded shape with 8 elements or more a side.
        if (p.A[0] != p.M[0] && p.modes[static_cast<size_t>(p.A[0])].group == GROUP_M && p.modes[static_cast<size_t>(p.M[0])].sC == 1) {
            const int64_t e0 = p.modes[static_cast<size_t>(p.M[0])].extent, e1 = p.modes[static_cast<size_t>(p.A[0])].extent;
            const int64_t rest = p.Mtot / e0 / e1;
            const bool c_larger = p.sizeC > p.sizeA;
            int64_t least = 0;
            for (int64_t t0 : c_larger ? std::vector<int64_t>{32} : std::vector<int64_t>{8, bm / 8, 16}) {
                const int64_t t1 = bm / t0, rows = ceil_div(e0, t0) * t0 * ceil_div(e1, t1) * t1 * rest;
                if (least == 0 || rows < least) {
                    least = rows;
                    g.t0 = static_cast<int>(t0);
                    g.t1 = static_cast<int>(t1);
                }
            }
            g.rows = least;
            if (double(least) > (c_larger ? 1.1 : 1.5) * double(p.Mtot)) {   // short modes: rows in C's order after all
                g.t0 = g.t1 = 0;
                g.rows = p.Mtot;
            }
        }
        const int64_t tiles_m = ceil_div(g.rows, bm), tiles_n = ceil_div(p.Ntot, bn);
        if (tiles_m > (int64_t(1) << 31) / kMaxGatherCluster / tiles_n) { if (t != GATHER_SQUARE) continue; }
        const double rate = f64 ? c.gather_f64_tflops[t] : c.gather_f32_tflops[t];
        const double iter_us = f64 ? c.gather_f64_iter_us[t] : c.gather_f32_iter_us[t];
        static const double kFixed[4] = {1.3, 1.7, 0.9, 1.7};   // set-up and stores of a tile, in units of gather_fixed_us
        const double fixed_us = c.gather_fixed_us * kFixed[t];
        const double sm_iter_us = 2.0 * double(bm) * double(bn) * 16.0 / (rate * 1e6 / c.num_sms);
        for (int s = 1; s <= kMaxGatherCluster; s *= 2) {
            if (force_cluster && std::atoi(force_cluster) != s) continue;
            const int64_t k_tiles = ceil_div(p.Ktot, 16);
            if (s > 1 && (one_chain || k_tiles < 2 * s || tiles_m * tiles_n * s > 8 * int64_t(c.num_sms))) break;
            const double iters = double(ceil_div(k_tiles, s));
            const int64_t per_sm = ceil_div(tiles_m * tiles_n * s, c.num_sms), resident = kTile[t][2];
            auto round_us = [&](int64_t ctas) { return ctas ? iters * std::max(iter_us, double(ctas) * sm_iter_us) + fixed_us : 0.0; };
            // Persistent CTAs where a CTA would otherwise be mostly set-up: more than one round of short k loops.  The small
            // FP64 tile takes that form for up to four k tiles anyway, because it has no k groups to add up at its end.
            const bool flat = s == 1 && (t == GATHER_SMALL ? one_chain || (f64 && iters <= 4) : per_sm > resident && iters <= 4);
            double us = flat ? fixed_us + std::max(double(per_sm) * (iters * sm_iter_us + c.gather_tile_us), double(ceil_div(per_sm, resident)) * iters * iter_us)
                             : double(per_sm / resident) * round_us(resident) + round_us(per_sm % resident);
            if (s > 1) us += c.gather_reduce_us;
            // tensors of up to half of L2 move at twice the rate (6912 x 240 x 4 FP64, 13 MB: 5.9 us)
            const double bytes = (double(p.sizeA) + double(p.sizeB) + double(p.sizeC)) * elt;
            us = std::max(us, fixed_us + bytes / ((bytes <= 64e6 ? 2.0 : 1.0) * c.gather_gbs * 1e3));
            // Rows in C's order although A's stride-1 mode is another row mode: every element of A comes in a sector of its own, which
            // the rates stand for once; 128 x 32 tiles on 33 to 64 columns fetch A twice (31185 x 35 x 311 FP64: 217 us, where
            // 64 x 64 tiles with rows cut 8 x 8 take 130; 2480625 x 35 x 87 Float32: 7884, 128 x 128 tiles 4155).  (An A in L2 can be: 9367 x
            // 33 x 63 Float32 takes 10 us in them, 14 in others.)
            if (t == GATHER_TALL && tiles_n == 2 && double(p.sizeA) * elt > 32e6 && g.t0 == 0 && p.A[0] != p.M[0] && p.modes[static_cast<size_t>(p.A[0])].group == GROUP_M)
                us += double(g.rows) * double(p.Ktot) * 32.0 / (c.gather_sector_gbs * 1e3);
            if (g.t0 > 0) us *= 1.6;   // (short runs on both sides: 12 x 12 by 124 FP64, rows cut 4 x 8, 18 us where the rule said 11)
            if (us < best.est_us) {
                best = g;
                best.cluster = s;
                // One column of Float32 tiles in two or three (64 x 64) and three or four (128 x 128) k tiles: blocks of one tile each, of which
                // more fit an SM at different stages, instead of a few persistent ones.  They read an A whose stride-1 mode is another row
                // mode than C's, a sector an element, in step.  Persistent / one tile a block in us: 2689715 x 35 x 19 1510 / 872, 4604655 x 45
                // x 33 5177 / 2979, 462231 x 113 x 43 315 / 250.  Elsewhere they multiply a last k tile whole, which the persistent ones cut
                // off: 64 x 64 by the k in it 2 149 / 172, 3 44 / 51, 8 70 / 74, 11 23.0 / 25.0 to 84 / 80, 12 295 / 281, 14 30.1 / 26.3; 128 x
                // 128 4 89 / 99, 7 350 / 362, 8 147 / 147, 9 190 / 177, 10 34.7 / 30.1, 14 196 / 176.  FP64 is up to twice as slow that way.
                const bool scattered_rows = g.t0 == 0 && p.A[0] != p.M[0] && p.modes[static_cast<size_t>(p.A[0])].group == GROUP_M;
                const int64_t last_k = (p.Ktot - 1) % 16 + 1;
                const bool few_k_tiles = (t == GATHER_SQUARE && iters >= 2 && iters <= 3 && (scattered_rows || last_k >= 12)) ||
                                         (t == GATHER_BIG && iters >= 3 && (scattered_rows || last_k >= 9));
                best.flat = flat && (f64 || tiles_n > 1 || !few_k_tiles);
                if (force_flat) best.flat = s == 1 && force_flat[0] == '1' && (f64 || t != GATHER_SMALL);   // (the small Float32 tile has no such form)
                best.est_us = us;
                sector_us = double(scattered_a * g.rows * tiles_n + scattered_b * p.Ntot * tiles_m) * double(p.Ktot) * 32.0 / (c.gather_sector_gbs * 1e3);
            }
        }
    }
    best.form = f64 || best.flat ? GATHER_FORM_PLAIN : float32_form(best, p, c);
    best.est_us += sector_us;   // (the choice of a tile is as good without it: its rates have it in part)
    return best;
}

double contraction_us(const Problem& p, int kernel, const UmmaSpec& u, const CostTable& c, bool count_sectors = true)
{
    if (kernel == KERNEL_DMMA_F64 || kernel == KERNEL_SIMT) return c.launch_us + plan_gather(p, c, count_sectors).est_us;
    const double elt = p.scalar_type == 1 ? 8.0 : 4.0;
    const double flops = 2.0 * double(p.Mtot) * double(p.Ntot) * double(p.Ktot);
    double c_bytes = double(p.sizeC) * elt;
    double rate = 0;
    double extra_us = 0, scatter_us = 0, extra_floor_us = 0;
    // (Whole tile columns, although `slim` computes fewer: charging what is computed here and for split-K changes 52 of 1434 drawn choices
    // of kernel and ranges, 24 of them for the worse, up to 2.2 times; the other constants are fitted with whole columns.)
    // TMA-fed kernels: slabs and k chunks are whole, ragged extents are zero-filled and multiplied anyway
    // (extents of 72 in 32-wide slabs and chunks: abcd-aefb-fdce ran at 138 TFLOP/s direct, 415 after a
    // transpose that fuses the ragged modes away)
    const double tma_padding = double(u.tiles_m * u.BM) / double(p.Mtot) * double(u.tiles_n * u.BN) / double(p.Ntot) *
                               u.k_computed / double(p.Ktot);
    if ((kernel == KERNEL_DMMA_F64_TMA || kernel == KERNEL_UMMA_TF32) && u.k_splits > 1) {
        // partial tensors written, read back and summed by a second kernel
        // (set up while the first kernel drains; partial tensors of up to half of L2 are read back from there)
        const double partials = 2.0 * double(u.k_splits) * double(p.sizeC) * elt;
        extra_us += 0.5 * c.launch_us + partials / (c.hbm_gbs * 1e3) * (partials < 128e6 ? 0.5 : 1.0);
    }
    if (kernel == KERNEL_DMMA_F64_TMA) {
        // A 128 x 64 tile keeps the FP64 pipe busy for 1.05 us per k chunk of 16 (128 MMAs a warp) and takes 4.5 us to set up,
        // fill and drain (M 192, N 384, K 52: 12 tiles in 15 us; M = N = 576, K 256 in four ranges: 21 us)
        extra_floor_us = 4.5 + double(ceil_div(u.tiles_m * u.tiles_n * u.k_splits, c.num_sms)) * double(u.k_iters_per_split) * (u.BK == 16 ? 1.05 : 0.55) * u.BN / 64.0;
        rate = c.dmma_f64_tflops * wave_efficiency(u.tiles_m * u.tiles_n * u.k_splits, c.num_sms) / tma_padding;
        // Rows of a slab that are not contiguous in C are stored element by element
        // (abcdef-dega-gfbc: 37.7 M elements of C, 1.08 ms against 0.10 ms for its coalesced siblings).
        // (runs shorter than 64 bytes count as scattered too: cfg3 cut to a = 6 ran at 17.6 TFLOP/s here
        // against 20.2 on the gather kernel, which sees those rows as one flat index)
        if ((u.a.row_elem_cstride != 1 && !u.store_across_slabs) || u.a.slab_mode_ext < 8)
            scatter_us = double(p.sizeC) * double(u.k_splits) * c.scatter_store_ps * 1e-6;
    }
    if (kernel == KERNEL_UMMA_TF32) {
        rate = c.umma_tf32_tflops * (1.0 - c.far_row_penalty * u.far_fraction) *
               wave_efficiency((u.pair ? ceil_div(u.tiles_m, 2) : u.tiles_m) * u.tiles_n * u.k_splits, u.pair ? c.num_sms / 2 : c.num_sms) / tma_padding;
        // Rows of a slab that are not contiguous in C are stored element by element, a 32-byte sector each
        // (abcd-dbea-ec, 9.0 M elements of C: 0.125 ms against a 0.022 ms traffic floor).
        if (u.a.row_elem_cstride != 1) scatter_us = double(p.sizeC) * double(u.k_splits) * c.scatter_store_f32_ps * 1e-6;
        // (one stage per umma_stage_us at best: see plan_umma_impl)
        const int64_t units = (u.pair ? ceil_div(u.tiles_m, 2) : u.tiles_m) * u.tiles_n * u.k_splits;
        const int64_t wave = u.pair ? c.num_sms / 2 : c.num_sms;
        // ... and a tile leaves an SM no faster than the epilogue stores it (cfg4: 7 776 tiles of 128 x 256 in 0.196 ms)
        const double tile_store_us = double(u.BM) * double(u.BN) * 4.0 / (c.umma_store_gbs_per_sm * 1e3);
        extra_floor_us = double(ceil_div(units, wave)) * std::max(double(u.k_iters_per_split) * c.umma_stage_us / u.producers, tile_store_us);
    }
    const double bytes = (double(p.sizeA) + double(p.sizeB)) * elt + c_bytes;
    // scattered stores are a third ceiling rather than an addition: one consumer group stores while the
    // other computes (abc-bda-dc, K = 312: 0.086 ms scattered against 0.072 ms for its coalesced sibling)
    return c.launch_us + std::max({flops / (rate * 1e6), bytes / (c.hbm_gbs * 1e3), scatter_us, extra_floor_us}) + extra_us;
}

// Float32 where A's stride-1 mode x is a row mode but not C's, y (across_tf32.cu).  Everything a tensor map needs is checked
// here, so that a plan that has it can run.
AcrossSpec plan_across(const Problem& p, const CostTable& c)
{
    AcrossSpec s;
    if (p.scalar_type != 0 || p.M.size() < 2 || p.N.empty() || p.K.empty() || p.K.size() > 3) return s;
    if (p.A.size() > kMaxTmaRank || p.B.size() > kMaxTmaRank || p.C.size() > kMaxTmaRank || p.B.size() < 2) return s;
    auto mode = [&](int id) -> const Mode& { return p.modes[static_cast<size_t>(id)]; };
    const int x = p.A[0], y = p.M[0];
    if (mode(x).group != GROUP_M || x == y || mode(y).sC != 1 || mode(x).sA != 1) return s;
    const bool b_kmajor = mode(p.B[0]).group == GROUP_K;
    int kc = p.K[0], n = p.B[0];
    if (b_kmajor) {
        kc = p.B[0];
        n = p.N[0];
        for (int id : p.N)
            if (mode(id).extent > mode(n).extent) n = id;
    } else {
        for (int id : p.K)   // rows of a box are one stride of this mode apart
            if (mode(id).sA < mode(kc).sA) kc = id;
    }
    const int64_t kc_ext = mode(kc).extent, n_ext = mode(n).extent;
    s.b_major = b_kmajor ? 0 : 1;
    s.BK = b_kmajor ? 32 : kc_ext <= 8 ? 8 : kc_ext <= 16 ? 16 : 32;
    if (!b_kmajor && kc_ext % 24 == 0 && double(ceil_div(kc_ext, 32) * 32) > 1.15 * double(kc_ext)) s.BK = 24;
    s.BN = n_ext <= 32 ? 32 : 64;
    s.n_ext = n_ext;
    s.x_ext = mode(x).extent;
    std::vector<int> rows, columns, ks;   // the other modes
    for (int id : p.M)
        if (id != x && id != y) rows.push_back(id);
    for (int id : p.N)
        if (id != n) columns.push_back(id);
    for (int id : p.K)
        if (id != kc) ks.push_back(id);
    auto fill = [&](AcrossSpec::Map& m, std::vector<int> order, const std::vector<int>& first, const std::vector<int>& second, int which) {
        order.insert(order.end(), first.begin(), first.end());
        order.insert(order.end(), second.begin(), second.end());
        int64_t span = 1;
        for (size_t d = 0; d < order.size(); ++d) {
            const Mode& q = mode(order[d]);
            m.ext[d] = q.extent;
            m.stride[d] = which == 0 ? q.sA : which == 1 ? q.sB : q.sC;
            if (d == 0 ? m.stride[0] != 1 : m.stride[d] % 4 != 0) return false;   // (16 bytes)
            span += (q.extent - 1) * m.stride[d];
        }
        for (size_t d = order.size(); d < kMaxTmaRank; ++d) m.stride[d] = (span + 3) / 4 * 4;
        return span < (int64_t(1) << 37);
    };
    if (!fill(s.a, {x, kc, y}, rows, ks, 0) || !fill(s.b, b_kmajor ? std::vector<int>{kc, n} : std::vector<int>{n, kc}, columns, ks, 1) ||
        !fill(s.c, {y, x, n}, rows, columns, 2)) return s;
    s.a.box[0] = 32; s.a.box[1] = s.BK; s.a.box[2] = 16;
    s.b.box[0] = 32; s.b.box[1] = b_kmajor ? s.BN : s.BK;
    s.c.box[0] = 16; s.c.box[1] = 16; s.c.box[2] = 8;
    s.row_others = static_cast<int>(rows.size());
    s.column_others = static_cast<int>(columns.size());
    if (!rows.empty()) s.o0 = mode(rows[0]).extent;
    if (rows.size() > 1) s.o1 = mode(rows[1]).extent;
    if (!columns.empty()) s.p0 = mode(columns[0]).extent;
    if (!ks.empty()) s.k1 = mode(ks[0]).extent;
    s.k_ext = kc_ext;
    s.y_chunks = ceil_div(mode(y).extent, 16);
    s.x_chunks = ceil_div(s.x_ext, 32);
    s.n_chunks = ceil_div(n_ext, s.BN);
    s.tiles_m = s.y_chunks * s.x_chunks;
    for (int id : rows) s.tiles_m *= mode(id).extent;
    s.tiles_n = s.n_chunks;
    for (int id : columns) s.tiles_n *= mode(id).extent;
    s.k_iters = ceil_div(kc_ext, s.BK);
    for (int id : ks) s.k_iters *= mode(id).extent;
    if (s.tiles_m >= (int64_t(1) << 30) / s.tiles_n || s.k_iters >= (int64_t(1) << 24)) return s;
    // Rows first, so that tiles that run together cover whole rows of C (C[a,b,c,d,e] of 251 MB from A of 1.3: 79 -> 43 us), and x
    // last among them, because its 32 rows lie far apart in C and the fewer of them are written at a time the better (C of 1.0 GB:
    // 339 us with x behind y, 210 behind all; of 453 MB: 208 and 118).  Unless A is too large to be read from L2 again by the other
    // columns' tiles later, and is read in its own order (A of 107 MB, two tile columns: 78 us rows first, 68 columns first; of 162
    // MB, four: 180 and 123; of 33 MB, four: 36.4 and 36.1; of 1.4 GB, one: 411 us with x last, 313 behind y).
    // TCONT_ACROSS_ROWS_FIRST=0|1 overrides the rule.
    s.rows_first = p.sizeA * 4 <= (int64_t(64) << 20);
    if (const char* e = std::getenv("TCONT_ACROSS_ROWS_FIRST")) s.rows_first = e[0] == '1';
    // two stages at least beside the staged pieces of C
    const int stage_bytes = 16 * 128 * s.BK + s.BN * s.BK * 4;
    s.stages = std::min(8, (227 * 1024 - 2 * 1024 - 64 * 1024) / stage_bytes);
    // A CTA passes a stage no faster than an SM takes it in: 110 GB/s, less where A's rows do not start on 128-byte lines (C of 55 MB, x = 24,
    // K 72: 34 us, 24 behind copies), less than half where they start in the middle of a 32-byte sector (C of 138 MB, x = 20, K 48:
    // 72 us, 42 behind copies), unless few SMs ask for them.  And a piece of 8 columns no faster than it is staged and stored, by
    // one bulk store or, with x > 16, by two.
    int64_t together = 32;
    for (int d = 1; d < kMaxTmaRank; ++d)
        while (s.a.ext[d] > 1 && s.a.stride[d] % together != 0) together /= 2;
    const double stage_gbs = together == 32 || s.tiles_m * s.tiles_n < c.num_sms ? 110.0 : together >= 8 ? 65.0 : 50.0;
    const double pieces = std::ceil(std::min<double>(double(n_ext), s.BN) / 8.0);
    const double tile_us = std::max(double(s.k_iters) * double(stage_bytes) / (stage_gbs * 1e3), c.across_piece_us * (s.x_ext > 16 ? 1.0 : 0.8) * pieces) + c.across_tile_us;
    // Rows of y that are no multiple of 32 bytes end inside a sector, which is then read first (C of 188 MB with y = 28: 91 us, y = 32
    // 33); a C that stays in L2 minds less (26 MB, y = 20: 18.3 us, where whole rows would take 14; 10 MB 8.5), and a small one does
    // not.  Rows that end in half of a chunk leave in 64 and 32 bytes (C of 151 MB, y = 24: 44.3 us, 37 by its bytes; of 106 MB 30.7 and 28).
    const double c_bytes = 4.0 * double(p.sizeC);
    const bool torn = mode(y).extent % 8 != 0, half = mode(y).extent % 16 == 8, beyond_l2 = c_bytes > 64e6;
    const double bytes = 4.0 * (double(p.sizeA) + double(p.sizeB)) + (beyond_l2 ? torn ? 3.0 : half ? 1.25 : 1.0 : 1.0) * c_bytes;
    const double us = std::max(double(ceil_div(s.tiles_m * s.tiles_n, c.num_sms)) * tile_us, bytes / (c.across_gbs * 1e3));
    s.est_us = c.launch_us + us * (torn && !beyond_l2 && c_bytes > 16e6 ? mode(y).extent < 32 ? 1.5 : 1.15 : 1.0);
    s.on = true;
    return s;
}

// What alpha and beta add to a Float32 contraction on the tensor cores (microseconds), `reads` = beta is not zero.  Tiles across two
// stride-1 modes go to a workspace that a second pass reads, with C, and writes C from: C three times or twice more.  The other
// form's epilogue reads C as it stores it, slower than its plain stores in either case; rows stored element by element are read that
// way, too.  Read off 176 contractions (C of 0.2 to 1000 MB) in both forms: C of 460 MB 314 us more across (226 without the old values),
// 167 (72) in the other form, of 75 MB 37 (24) and 24 (11), of 25 MB 10 (9) and 12 (7), of 1.8 MB 2.8 and, element by element, 16.
double scalars_us(bool across, double c_bytes, double scattered_us, bool reads)
{
    const double mb = c_bytes * 1e-6;
    if (across) return 2.3 + (reads ? 3.0 : 2.0) * mb / (mb > 67.2 ? 4.85 : mb > 48.0 ? 6.4 : 8.0);
    return (reads ? 1.5 + mb / 3.3 + 1.5 * scattered_us : 0.5 + 0.155 * mb + 0.6 * scattered_us) + (scattered_us > 0 ? 1.0 : 0.0);
}

// TF32 goes to the tcgen05 kernel whenever its tiles can be described to TMA.  FP64 takes the cheaper of the TMA-fed kernel
// and the gather kernel, by the cost table; Float32 that TMA cannot describe goes to the gather kernel.  The gather kernel
// is reported as KERNEL_DMMA_F64 where FP64 work fills the GPU with tiles, as KERNEL_SIMT otherwise.
int pick_kernel(const Problem& p, const UmmaSpec& u, const CostTable& c)
{
    if (u.eligible && u.elt == 4) return KERNEL_UMMA_TF32;
    if (p.scalar_type != 1) return KERNEL_SIMT;
    const char* k = std::getenv("TCONT_KERNEL");
    if (k && std::strcmp(k, "simt") == 0) return KERNEL_SIMT;
    const int64_t bn = p.Ntot <= 48 ? 32 : 64, bm = p.Ntot <= 48 ? 256 : 128;
    const int gather = ceil_div(p.Mtot, bm) * ceil_div(p.Ntot, bn) >= c.num_sms ? KERNEL_DMMA_F64 : KERNEL_SIMT;
    if (!u.eligible || u.elt != 8 || (k && std::strcmp(k, "gather") == 0)) return gather;
    if (k && std::strcmp(k, "tma") == 0) return KERNEL_DMMA_F64_TMA;
    if (std::getenv("TCONT_SPLITK")) return KERNEL_DMMA_F64_TMA;   // (a forced split of k is a switch of the TMA-fed kernel)
    // The smallest problems are a matter of latency, which both estimates know to a tenth; above 20 us the gather kernel has to
    // look 30 % better, because its whole-tile rate is 5 to 25 % more than it reaches on uneven tiles and long rows.  Where the
    // TMA-fed kernel's tiles run across slabs, A's stride-1 mode is not C's, and its gathers or C's stores are short runs:
    // there already above 10 us (1024 x 2048 x 40, estimated at 18 and 20 us, takes 22.5 and 15.8; 4096 x 128 x 8, at 8 and 9,
    // 3.8 and 7.3).
    const double tma_us = contraction_us(p, KERNEL_DMMA_F64_TMA, u, c), gather_us = contraction_us(p, gather, u, c);
    return tma_us <= (gather_us < (u.store_across_slabs ? 10.0 : 20.0) ? 1.05 : 1.3) * gather_us ? KERNEL_DMMA_F64_TMA : gather;
}

}  // namespace

bool read_cost_table_file(const std::string& path, CostTable* table)
{
    CostTable& c = *table;
    std::ifstream f(path);
    if (!f) return false;
    std::string key;
    double v;
    // "key value" pairs, one per line; unknown keys are ignored.
    while (f >> key >> v) {
        if (key == "hbm_gbs") c.hbm_gbs = v;
        else if (key == "umma_tf32_tflops") c.umma_tf32_tflops = v;
        else if (key == "launch_us") c.launch_us = v;
        else if (key == "simt_f32_tflops") c.line_f32_tflops = v;
        else if (key == "line_launch_us") c.line_launch_us = v;
        else if (key == "dmma_f64_tflops") c.dmma_f64_tflops = v;
        else if (key == "gather_fixed_us") c.gather_fixed_us = v;
        else if (key == "gather_reduce_us") c.gather_reduce_us = v;
        else if (key == "gather_tile_us") c.gather_tile_us = v;
        else if (key == "gather_gbs") c.gather_gbs = v;
        else if (key == "gather_sector_gbs") c.gather_sector_gbs = v;
        else if (key == "permute_tile_ns") c.permute_tile_ns = v;
        else if (key == "scatter_store_ps") c.scatter_store_ps = v;
        else if (key == "scatter_store_f32_ps") c.scatter_store_f32_ps = v;
        else if (key == "far_row_penalty") c.far_row_penalty = v;
        else if (key == "across_piece_us") c.across_piece_us = v;
        else if (key == "across_tile_us") c.across_tile_us = v;
        else if (key == "across_gbs") c.across_gbs = v;
        else if (key == "umma_stage_us") c.umma_stage_us = v;
        else if (key == "umma_store_gbs_per_sm") c.umma_store_gbs_per_sm = v;
        else if (key == "num_sms" && v >= 1) c.num_sms = static_cast<int>(v);
        else
            for (int t = 0; t < 4; ++t) {   // gather_f64_tflops_0 ... gather_f32_iter_us_3
                const std::string i = std::to_string(t);
                if (t < 3 && key == "gather_f64_tflops_" + i) c.gather_f64_tflops[t] = v;
                else if (t < 3 && key == "gather_f64_iter_us_" + i) c.gather_f64_iter_us[t] = v;
                else if (key == "gather_f32_tflops_" + i) c.gather_f32_tflops[t] = v;
                else if (key == "gather_f32_iter_us_" + i) c.gather_f32_iter_us[t] = v;
            }
    }
    return true;
}

CostTable load_cost_table()
{
    CostTable c;
    if (const char* path = std::getenv("TCONT_COST_TABLE")) read_cost_table_file(path, &c);
    return c;
}

int make_plan(const char* modeC, int nC, const char* modeA, int nA, const char* modeB, int nB, char op, int scalar_type,
              const char* ext_mode, const int64_t* ext_val, int n_ext, int backend_selection, const CostTable& cost,
              Plan* plan, std::string* err, const int64_t* parentC, const int64_t* parentA, const int64_t* parentB, bool fuse_rows, bool across)
{
    if (!plan || !err) return 1;
    if (nC < 0 || nA < 0 || nB < 0 || n_ext < 0 || nC > kMaxModes || nA > kMaxModes || nB > kMaxModes || n_ext > 64) {
        *err = "Mode counts out of range";
        return 1;
    }
    if ((nC && !modeC) || (nA && !modeA) || (nB && !modeB) || (n_ext && (!ext_mode || !ext_val))) {
        *err = "Null mode or extent array";
        return 1;
    }
    if (scalar_type != 0 && scalar_type != 1) {
        *err = "Unsupported scalar type";
        return 1;
    }
    if (backend_selection < 0 || backend_selection > 2) {
        *err = "Unknown backend selection";
        return 1;
    }
    if (nA == 0 || nB == 0 || nC == 0) {
        *err = "Each tensor needs at least one mode";
        return 1;
    }
    Plan pl;
    pl.modeC.assign(modeC, static_cast<size_t>(nC));
    pl.modeA.assign(modeA, static_cast<size_t>(nA));
    pl.modeB.assign(modeB, static_cast<size_t>(nB));
    pl.ext_mode.assign(ext_mode, static_cast<size_t>(n_ext));
    pl.ext_val.assign(ext_val, ext_val + n_ext);
    pl.op = op;
    pl.scalar_type = scalar_type;
    pl.backend_selection = backend_selection;
    if (parentC) pl.parentC.assign(parentC, parentC + nC);
    if (parentA) pl.parentA.assign(parentA, parentA + nA);
    if (parentB) pl.parentB.assign(parentB, parentB + nB);

    Problem direct;
    int rc = build_problem(pl.modeC, pl.modeA, pl.modeB, pl.ext_mode, pl.ext_val, scalar_type, &direct, err, pl.parentC, pl.parentA, pl.parentB);
    if (rc) return rc;
    if (direct.sizeA >= (int64_t(1) << 32) || direct.sizeB >= (int64_t(1) << 32)) {
        *err = "Input tensors with 2^32 or more elements are not supported";
        return 3;
    }
    auto count = [&](const std::string& s) {
        int64_t n = 1;
        for (char c : s) n *= pl.ext_val[static_cast<size_t>(find_char(pl.ext_mode, c))];
        return n;
    };
    pl.sizeL = count(pl.modeA);
    pl.sizeR = count(pl.modeB);
    pl.sizeC = count(pl.modeC);
    pl.flops = 2.0 * std::sqrt(double(pl.sizeL) * double(pl.sizeR) * double(pl.sizeC));

    UmmaSpec direct_umma;
    plan_umma(direct, cost, &direct_umma, fuse_rows);
    int direct_kernel = pick_kernel(direct, direct_umma, cost);

    // Transpose-assisted candidate.  A role's transposed layout is
    //     [lead | K modes | remaining row modes in C order]
    // where `lead` is the shortest run of the role's first row modes (consecutive in C) whose fused
    // extent is a multiple of 32: the slab mode stays stride-1 and the K rows of a tile follow it
    // directly, so a TMA box is one contiguous piece of memory.  An operand that already starts
    // with [lead, first K mode] (or is K-major on that K mode) is used where it lies.  Three K
    // orders are tried (by A's strides, by B's strides, the direct plan's); the one that moves
    // the fewest bytes wins.  C is written in its final order by the contraction kernel, so
    // there is never a third transpose (the reference's TTGT always pays C' -> C,
    // backends/ttgt_cutt/src/ttgt_cutt.cpp:811-816).
    const std::string& roleA_src = direct.swapped ? pl.modeB : pl.modeA;
    const std::string& roleB_src = direct.swapped ? pl.modeA : pl.modeB;
    auto ext_of = [&](char c) { return pl.ext_val[static_cast<size_t>(find_char(pl.ext_mode, c))]; };
    auto lead_of = [&](const std::string& src) {  // row modes of `src` in C order, split into (lead, rest)
        std::string rows;
        for (char c : pl.modeC)
            if (find_char(src, c) >= 0) rows.push_back(c);
        size_t n = 0;
        int64_t prod = 1;
        bool found = false;
        while (n < rows.size()) {
            if (n > 0 && find_char(pl.modeC, rows[n]) != find_char(pl.modeC, rows[n - 1]) + 1) break;
            prod *= ext_of(rows[n]);
            ++n;
            if (prod % 32 == 0) { found = true; break; }
        }
        if (!found) {  // no multiple of 32: keep the whole leading run together
            n = 1;
            while (n < rows.size() && find_char(pl.modeC, rows[n]) == find_char(pl.modeC, rows[n - 1]) + 1) ++n;
        }
        // FP64: a leading run too short for whole slabs (extent 6 or 12: a quarter of the rows empty) takes the
        // next run of row modes along, so that the kernel's planner can stage both as one fused mode
        // (operand-level row fusion in plan_umma)
        if (scalar_type == 1 && n < rows.size()) {
            int64_t lead_ext = 1;
            for (size_t i = 0; i < n; ++i) lead_ext *= ext_of(rows[i]);
            if (slab_padding_f64(lead_ext) > 1.08) {
                size_t m = n + 1;
                while (m < rows.size() && find_char(pl.modeC, rows[m]) == find_char(pl.modeC, rows[m - 1]) + 1) ++m;
                n = m;
            }
        }
        return std::make_pair(rows.substr(0, n), rows.substr(n));
    };
    const auto leadA = lead_of(roleA_src), leadB = lead_of(roleB_src);
    std::string kall;
    for (char c : roleA_src)
        if (find_char(pl.modeC, c) < 0) kall.push_back(c);
    auto sorted_by = [&](const std::string& src) {
        std::string k = kall;
        std::sort(k.begin(), k.end(), [&](char x, char y) { return find_char(src, x) < find_char(src, y); });
        return k;
    };
    auto starts_with = [](const std::string& s, const std::string& pre) { return s.compare(0, pre.size(), pre) == 0; };
    std::vector<std::pair<std::string, std::string>> candidates{{roleA_src, roleB_src}};
    {
        double best = 1e300;
        for (const std::string& korder : {sorted_by(roleB_src), sorted_by(roleA_src), perm_modes(direct, direct.K)}) {
            if (korder.empty()) continue;
            auto keep = [&](const std::string& src, const std::string& lead) {
                return src[0] == korder[0] || starts_with(src, lead + korder[0]);
            };
            const bool keepA = keep(roleA_src, leadA.first), keepB = keep(roleB_src, leadB.first);
            const double moved = (keepA ? 0.0 : double(direct.sizeA)) + (keepB ? 0.0 : double(direct.sizeB));
            if (moved < best) {
                best = moved;
                candidates[0] = {keepA ? roleA_src : leadA.first + korder + leadA.second,
                                 keepB ? roleB_src : leadB.first + korder + leadB.second};
            }
        }
    }
    // Float32, arithmetic-bound: both operands as matrices, A as [rows | K] and B as [K | columns], K in one order, so
    // that the contracted modes fuse into one and (operand-level fusion in plan_umma) the rows do: no slab and no k chunk
    // is padded.  abcd-aedf-fbec with extents of 72 computes 1.97 times its flops where the operands lie.
    if (scalar_type == 0 && fuse_rows) {
        std::string rowsA, rowsB;
        for (char c : pl.modeC) (find_char(roleA_src, c) >= 0 ? rowsA : rowsB).push_back(c);
        for (const std::string& korder : {sorted_by(roleB_src), sorted_by(roleA_src)})
            if (!korder.empty() && !rowsB.empty()) candidates.push_back({rowsA + korder, korder + rowsB});
    }
    // FP64 operands TMA cannot describe where they lie, because some stride is no multiple of 16 bytes: both as such matrices, the
    // last mode of the run that starts each padded where that makes every stride behind it even (61 x 53 rows of A: 61 x 54).
    // 3233 x 2773 x 851: 640 us on the gather kernel, 514 behind the two padded copies; 1297 x 1633 x 7859 3 444 and 1 230.  (Sums of more than 49 152 products stay
    // one chain of FMAs on the gather kernel, see plan_gather.)
    std::vector<int64_t> paddedA, paddedB;   // of the last candidate; empty = dense
    size_t padded_candidate = 0;
    const char* padded_env = std::getenv("TCONT_PADDED_COPIES");   // tuning switch: 0 never, 1 wherever they can be staged
    const bool padded_forced = padded_env && padded_env[0] == '1';
    if (scalar_type == 1 && !direct.strided && !direct_umma.eligible && direct.Ktot <= 49152 && direct.M.size() > 0 && direct.N.size() > 0 && !(padded_env && padded_env[0] == '0')) {
        std::string rowsA, rowsB;
        for (char c : pl.modeC) (find_char(roleA_src, c) >= 0 ? rowsA : rowsB).push_back(c);
        const std::string korder = sorted_by(roleB_src);
        // (rows that lie next to one another in C become one mode, and so do all contracted ones)
        size_t run = 1;
        while (run < rowsA.size() && find_char(pl.modeC, rowsA[run]) == find_char(pl.modeC, rowsA[run - 1]) + 1) ++run;
        auto pad = [&](const std::string& layout, size_t first_run) {
            std::vector<int64_t> v;
            int64_t product = 1;
            for (size_t i = 0; i < layout.size(); ++i) {
                v.push_back(ext_of(layout[i]));
                if (i < first_run) product *= v.back();
            }
            if (product % 2 == 0) return std::vector<int64_t>();
            ++v[first_run - 1];   // (all extents of the run are odd)
            return v;
        };
        if (!korder.empty()) {
            padded_candidate = candidates.size();
            candidates.push_back({rowsA + korder, korder + rowsB});
            paddedA = pad(candidates.back().first, run);
            paddedB = pad(candidates.back().second, korder.size());
        }
    }
    // (a transposed operand is a dense scratch tensor; one that is used where it lies keeps its parent's strides)
    const std::vector<int64_t>& roleA_parent = direct.swapped ? pl.parentB : pl.parentA;
    const std::vector<int64_t>& roleB_parent = direct.swapped ? pl.parentA : pl.parentB;
    const std::vector<int64_t> dense;
    const double elt = scalar_type == 1 ? 8.0 : 4.0;
    Problem ttgt;
    UmmaSpec ttgt_umma;
    int ttgt_kernel = KERNEL_SIMT;
    double ttgt_by_tiles_us = 1e300;   // with the permutations' tiles counted
    TransposeSpec tA, tB;
    pl.est_ttgt_us = 1e300;
    auto padded = [&](size_t candidate, bool is_a) -> const std::vector<int64_t>& {
        return candidate > 0 && candidate == padded_candidate ? (is_a ? paddedA : paddedB) : dense;
    };
    auto problem_of = [&](size_t candidate, Problem* q) {
        const auto& layouts = candidates[candidate];
        const std::vector<int64_t> &padA = padded(candidate, true), &padB = padded(candidate, false);
        const int rc_build = build_problem(pl.modeC, layouts.first, layouts.second, pl.ext_mode, pl.ext_val, scalar_type, q, err, pl.parentC,
                                           !padA.empty() ? padA : layouts.first == roleA_src ? roleA_parent : dense,
                                           !padB.empty() ? padB : layouts.second == roleB_src ? roleB_parent : dense);
        q->strided = direct.strided;   // (padding is not a view)
        return rc_build;
    };
    // `tiles`: also by the tiles of the permutation kernel, 64 x 64 at most along the stride-1 modes of source and destination.
    // Short ones on both sides make many small tiles: 15 x 15 of 50 MB take 171 us, not the 23 of the bandwidth.
    auto transpose_us = [&](const std::string& src, const std::string& dst, int64_t elements, const CostTable& c, bool tiles, bool padded_copy) {
        if (src == dst && !padded_copy) return 0.0;
        auto run = [&](const std::string& of, const std::string& in) {   // extent of the first modes that stay together
            int64_t e = ext_of(of[0]);
            for (size_t i = 1; i < of.size() && find_char(in, of[i]) == find_char(in, of[i - 1]) + 1; ++i) e *= ext_of(of[i]);
            return e;
        };
        double us = 2.0 * double(elements) * elt / (c.hbm_gbs * 0.7 * 1e3);
        if (tiles && src[0] != dst[0]) {
            const int64_t e0 = run(src, dst), e1 = run(dst, src);
            us = std::max(us, double(elements) / double(e0) / double(e1) * double(ceil_div(e0, 64) * ceil_div(e1, 64)) * c.permute_tile_ns * 1e-3);
        }
        return c.launch_us + us;
    };
    auto transposes_us = [&](size_t candidate, const CostTable& c, bool tiles) {
        const auto& layouts = candidates[candidate];
        return transpose_us(roleA_src, layouts.first, direct.sizeA, c, tiles, !padded(candidate, true).empty()) +
               transpose_us(roleB_src, layouts.second, direct.sizeB, c, tiles, !padded(candidate, false).empty());
    };
    // Whether Float32 runs as TF32 or in IEEE single precision is a question of precision, not only of time, and its answer
    // does not follow the kernels' speed: of the operands as they lie and the first transposed layout, the cheaper decides, by
    // whether the tcgen05 kernel can stage it.  Cheaper by launches of 6.9 us, CUDA cores at 23.7 TFLOP/s (line_launch_us and
    // line_f32_tflops of the cost table) and the tcgen05 kernel with every mode staged on its own.
    bool tf32 = true;
    if (scalar_type == 0) {
        CostTable line = cost;
        line.launch_us = cost.line_launch_us;
        const double flops = 2.0 * double(direct.Mtot) * double(direct.Ntot) * double(direct.Ktot);
        const double ieee_us = line.launch_us + std::max(flops / (line.line_f32_tflops * 1e6), (double(direct.sizeA) + double(direct.sizeB) + double(direct.sizeC)) * elt / (line.hbm_gbs * 1e3));
        auto line_us = [&](const Problem& q, bool* staged) {
            UmmaSpec u;
            plan_umma(q, line, &u, false);
            *staged = pick_kernel(q, u, line) == KERNEL_UMMA_TF32;
            if (!*staged) return ieee_us;
            double us = contraction_us(q, KERNEL_UMMA_TF32, u, line);
            if (u.k_splits > 1) {   // (a whole launch, and all partials through HBM)
                const double partials = 2.0 * double(u.k_splits) * double(q.sizeC) * elt;
                us += 0.5 * line.launch_us + (partials < 128e6 ? 0.5 : 0.0) * partials / (line.hbm_gbs * 1e3);
            }
            return us;
        };
        Problem q;
        rc = problem_of(0, &q);
        if (rc) return rc;
        bool direct_staged, moved_staged;
        const double direct_us = line_us(direct, &direct_staged), moved_us = line_us(q, &moved_staged);
        const double t_us = transposes_us(0, line, false);
        tf32 = (backend_selection == 0 ? t_us > 0 && t_us + moved_us < direct_us : backend_selection == 2) ? moved_staged : direct_staged;
        if (!tf32 && direct_kernel == KERNEL_UMMA_TF32) {
            direct_umma = UmmaSpec();
            direct_umma.why_not = "runs in IEEE single precision";
            direct_kernel = KERNEL_SIMT;
        }
    }
    pl.est_direct_us = contraction_us(direct, direct_kernel, direct_umma, cost);
    for (size_t i = 0; i < (tf32 ? candidates.size() : 1); ++i) {
        // (short contractions gain nothing by padded copies that the estimates could tell: 88 000 x 13 x 39 36 us, 38 behind them, 987 x
        // 1820 x 234 63 and 59)
        if (i > 0 && i == padded_candidate && pl.est_direct_us < 60.0 && !padded_forced) continue;
        Problem q;
        rc = problem_of(i, &q);
        if (rc) return rc;
        UmmaSpec u;
        if (tf32) plan_umma(q, cost, &u, fuse_rows);
        const int kernel = pick_kernel(q, u, cost);
        // (the TMA-fed kernels gain much more by another layout than the gather kernel does, so for them the tiles do not decide)
        const bool gathers = kernel == KERNEL_SIMT || kernel == KERNEL_DMMA_F64;
        double us = transposes_us(i, cost, gathers || (i > 0 && i == padded_candidate)) + contraction_us(q, kernel, u, cost);
        // (stores come on top of the arithmetic where they are not all of 32 aligned bytes: 10469 x 9025 x 63, odd, 798 us with 360 of
        // arithmetic, 580 on the gather kernel; 82431 x 2205 x 7 818 and 546)
        if (i > 0 && i == padded_candidate && kernel == KERNEL_DMMA_F64_TMA) us += double(q.sizeC) * double(u.k_splits) * (u.piece == 4 ? 0.8e-6 : 4.6e-6);
        if (padded_forced && i > 0 && i == padded_candidate && kernel == KERNEL_DMMA_F64_TMA) us = 0;
        // Partial sums behind the FP64 kernel: a thread adds its partials up one after the other, 0.12 us each (96 x 64 x 2992
        // in 41 ranges: 20.8 us without that, 24.6 measured).  Where the operands lie the kernels' estimates are compared as they were fitted.
        if (kernel == KERNEL_DMMA_F64_TMA && u.k_splits > 1) us += 0.12 * u.k_splits;
        if (us < 0.97 * pl.est_ttgt_us) {   // (an alternative has to be clearly better than the first)
            pl.est_ttgt_us = us;
            ttgt_by_tiles_us = us - transposes_us(i, cost, false) + transposes_us(i, cost, true);
            ttgt = q;
            ttgt_umma = u;
            ttgt_kernel = kernel;
            fill_transpose(roleA_src, candidates[i].first, pl.ext_mode, pl.ext_val, &tA, roleA_parent, padded(i, true));
            fill_transpose(roleB_src, candidates[i].second, pl.ext_mode, pl.ext_val, &tB, roleB_parent, padded(i, false));
        }
    }

    if (ttgt_kernel != KERNEL_UMMA_TF32 && ttgt_kernel != KERNEL_DMMA_F64_TMA)
        pl.est_direct_us = contraction_us(direct, direct_kernel, direct_umma, cost, false);
    // (the error-compensated mode and a contracted-mode split keep the other form)
    const char* x3 = std::getenv("TCONT_TF32X3");
    if (across && fuse_rows && tf32 && direct_kernel == KERNEL_UMMA_TF32 && backend_selection != 2 && !(x3 && x3[0] == '1') && !std::getenv("TCONT_NO_ROWS_ACROSS_SLABS")) {
        pl.across = plan_across(direct, cost);
        const char* force = std::getenv("TCONT_ACROSS");   // tuning switch: 1 wherever it can run
        // Clearly better than either (C of 524 MB, estimated at 112 us and at 113 behind a copy of A of 3 MB, takes 104 and 94).  The copy of a
        // large A by its tiles: with short modes on both sides it takes far longer than its bytes (A of 126 MB, 16 x 32: 227 us in all, not 97).
        const bool clear = pl.across.est_us < 0.97 * pl.est_direct_us && (backend_selection == 1 || !(tA.needed || tB.needed) || pl.across.est_us < 0.97 * ttgt_by_tiles_us);
        if (pl.across.on && (clear || (force && force[0] == '1'))) pl.est_direct_us = pl.across.est_us;
        else pl.across.on = false;
    }
    bool use_ttgt;
    if (backend_selection == 1) use_ttgt = false;
    else if (backend_selection == 2) use_ttgt = true;
    // (no margin for padded copies: 47 x 49 x 45 by 127 by 19, estimated level, takes 110 us on the gather kernel and 96 behind them)
    else use_ttgt = !pl.across.on && (tA.needed || tB.needed) && pl.est_ttgt_us < pl.est_direct_us;

    if (use_ttgt) {
        pl.backend = 1;
        pl.prob = ttgt;
        pl.prob.swapped = direct.swapped;  // roles still map to the caller's operands as in `direct`
        pl.tA = tA;
        pl.tB = tB;
        pl.kernel = ttgt_kernel;
        pl.umma = ttgt_umma;
    } else {
        pl.backend = 0;
        pl.prob = direct;
        pl.kernel = direct_kernel;
        pl.umma = direct_umma;
    }
    const Problem& p = pl.prob;
    pl.kernel_without_narrow = pl.kernel;
    if (pl.kernel == KERNEL_DMMA_F64_TMA) {
        pl.narrow = narrow_tiles(p, cost, pl.umma);
        double us;
        // (the smallest estimate has to be 5 % better than the one of what was planned: of 22 contractions in ranges 16 changed, 1.10 times as fast)
        if (!pl.narrow.eligible && pl.umma.k_splits > 1) {
            UmmaSpec v = narrow_ranges(p, cost, pl.umma, &us);
            if (v.eligible && us < 0.95 * split_us(p, pl.umma, pl.umma.k_splits, cost)) pl.narrow = v;
        }
    } else if (p.scalar_type == 1 && p.Ktot <= 49152 && !std::getenv("TCONT_KERNEL")) {
        // The gather kernel's estimate of the smallest contractions is off by up to a factor of two either way (10.9 us estimated: 5.8 to
        // 12.9): only above 13.5 us does it say enough (17.9 estimated, 18.2 taken; 14.7 here).  Longer sums stay one chain (plan_gather).
        const double gather_us = contraction_us(p, pl.kernel, pl.umma, cost);
        double us = 1e300;
        UmmaSpec v;
        if (gather_us >= 13.5) v = narrow_ranges(p, cost, pl.umma, &us);
        if (v.eligible && us < 0.9 * gather_us) {
            pl.narrow = v;
            pl.kernel = KERNEL_DMMA_F64_TMA;
        }
    }
    pl.wide_reads = pl.kernel_without_narrow == KERNEL_DMMA_F64_TMA && wide_reads(p, pl.umma, pl.narrow) && !std::getenv("TCONT_DMMA_BN");
    for (UmmaSpec* u : {&pl.umma, &pl.narrow})
        if (u->eligible && u->elt == 8) set_dmma_groups(p, u, cost);
    if (pl.kernel == KERNEL_UMMA_TF32)
        for (int reads = 0; reads < 2; ++reads)
            pl.est_scaled_us[reads] = (use_ttgt ? ttgt_by_tiles_us : pl.est_direct_us) +
                                      scalars_us(pl.across.on, double(p.sizeC) * elt, !pl.across.on && pl.umma.a.row_elem_cstride != 1 ? double(p.sizeC) * cost.scatter_store_f32_ps * 1e-6 : 0.0, reads != 0);
    auto first_is = [&](const std::vector<int>& t, const std::vector<int>& grp) {
        return !t.empty() && !grp.empty() && t[0] == grp[0];
    };
    // SIMT loads run along m (or n) when the operand's stride-1 mode is the fastest mode of the
    // flat m (n) index, along k when it is the fastest contracted mode.
    pl.simt.a_load_along_k = first_is(p.A, p.M) ? 0 : (first_is(p.A, p.K) ? 1 : 0);
    pl.simt.b_load_along_k = first_is(p.B, p.N) ? 0 : (first_is(p.B, p.K) ? 1 : 0);
    pl.gather = plan_gather(p, cost);
    *plan = pl;
    return 0;
}

bool cuts_into_ranges(const Plan& pl, int ranges, std::string* why)
{
    const Problem& p = pl.prob;
    const UmmaSpec& u = pl.umma;
    if (pl.across.on) {
        *why = "contracted-mode split: tiles across two stride-1 modes have no columns of their own per rank";
        return false;
    }
    if (pl.kernel != KERNEL_UMMA_TF32 || u.k_splits != 1) {
        *why = "contracted-mode split needs the tcgen05 kernel without split-K (Float32 operands TMA can stage; TCONT_SPLITK=1)";
        return false;
    }
    if (p.C.empty() || p.N.empty() || p.C.back() != p.N.back()) {
        *why = "contracted-mode split: C's slowest mode must belong to the operand that does not hold C's stride-1 mode";
        return false;
    }
    *why = "contracted-mode split: the extent of C's slowest mode does not cut into whole tile columns per rank";
    const Mode& slow = p.modes[static_cast<size_t>(p.C.back())];
    if (slow.extent % ranges || pl.sizeC % ranges || u.tiles_n % ranges) return false;
    const int64_t tile_slabs = u.b.slabs_per_tile;
    // One row digit: the slab mode is all of N (one mode, or two fused ones), so a range ends inside it, and has to end where
    // a tile does.  More digits: C's slowest mode is the most significant one, and a range is whole indices of it -- unless it
    // is the slab mode (B's stride-1 mode), whose chunks are the least significant digit.
    if (u.b.n_row_digits == 1) return (u.b.slab_mode_ext / ranges) % (u.b.slab_w * tile_slabs) == 0;
    if (u.b.major == 1 && p.B[0] == p.C.back()) return false;
    return u.b.total_slabs % ranges == 0 && (u.b.total_slabs / ranges) % tile_slabs == 0;
}

static const char* kernel_name(int kernel)
{
    return kernel == KERNEL_UMMA_TF32 ? "umma_tf32" : kernel == KERNEL_DMMA_F64 ? "dmma_f64" : kernel == KERNEL_DMMA_F64_TMA ? "dmma_f64_tma" : "simt";
}

std::string describe_plan(const Plan& pl)
{
    std::ostringstream o;
    const Problem& p = pl.prob;
    auto list = [&](const std::vector<int>& ids) {
        std::string s = "[";
        for (size_t i = 0; i < ids.size(); ++i) {
            const Mode& m = p.modes[static_cast<size_t>(ids[i])];
            s += (i ? "," : "") + std::string("\"") + m.names + ":" + std::to_string(m.extent) + "\"";
        }
        return s + "]";
    };
    auto perm = [&](const TransposeSpec& t) {
        std::string s = "[";
        for (int i = 0; i < t.rank; ++i) s += (i ? "," : "") + std::to_string(t.perm[i]);
        return s + "]";
    };
    o << "{\"backend\":\"" << (pl.backend == 0 ? "direct" : "ttgt") << "\",\"kernel\":\""
      << kernel_name(pl.kernel) << "\""
      << ",\"scalar\":\"" << (pl.scalar_type == 1 ? "f64" : "f32") << "\",\"swapped\":" << (p.swapped ? "true" : "false")
      << ",\"views\":" << (p.strided ? "true" : "false")
      << ",\"A\":" << list(p.A) << ",\"B\":" << list(p.B) << ",\"C\":" << list(p.C) << ",\"M\":" << list(p.M)
      << ",\"N\":" << list(p.N) << ",\"K\":" << list(p.K) << ",\"Mtot\":" << p.Mtot << ",\"Ntot\":" << p.Ntot
      << ",\"Ktot\":" << p.Ktot << ",\"transpose_a\":" << (pl.tA.needed ? perm(pl.tA) : "null")
      << ",\"transpose_b\":" << (pl.tB.needed ? perm(pl.tB) : "null") << ",\"est_direct_us\":" << pl.est_direct_us
      << ",\"est_ttgt_us\":" << pl.est_ttgt_us << ",\"simt\":{\"a_along_k\":" << pl.simt.a_load_along_k
      << ",\"b_along_k\":" << pl.simt.b_load_along_k << "},\"gather\":{\"tile\":" << pl.gather.tile
      << ",\"cluster\":" << pl.gather.cluster << ",\"flat\":" << (pl.gather.flat ? "true" : "false")
      << ",\"form\":\"" << (pl.gather.form == GATHER_FORM_WIDE ? "wide" : pl.gather.form == GATHER_FORM_SHORT ? "short" : "plain") << "\",\"t0\":" << pl.gather.t0 << ",\"t1\":" << pl.gather.t1 << ",\"rows\":" << pl.gather.rows << ",\"est_us\":" << pl.gather.est_us << "}";
    const UmmaSpec& u = pl.umma;
    if (pl.across.on)
        o << ",\"across\":{\"BN\":" << pl.across.BN << ",\"BK\":" << pl.across.BK << ",\"stages\":" << pl.across.stages << ",\"tiles_m\":" << pl.across.tiles_m
          << ",\"tiles_n\":" << pl.across.tiles_n << ",\"k_iters\":" << pl.across.k_iters << ",\"b_major\":\"" << (pl.across.b_major ? "MN" : "K") << "\"}";
    if (pl.narrow.eligible)
        o << ",\"narrow\":{\"BN\":" << pl.narrow.BN << ",\"BK\":" << pl.narrow.BK << ",\"stages\":" << pl.narrow.stages << ",\"slim\":" << (pl.narrow.slim[0] ? "true" : "false") << ",\"tiles_m\":" << pl.narrow.tiles_m
          << ",\"tiles_n\":" << pl.narrow.tiles_n << ",\"k_splits\":" << pl.narrow.k_splits << ",\"groups\":[" << pl.narrow.groups[0] << "," << pl.narrow.groups[1] << "],\"wide_reads\":" << (pl.wide_reads ? "true" : "false") << ",\"instead_of\":\"" << kernel_name(pl.kernel_without_narrow) << "\"}";
    o << ",\"umma\":{\"eligible\":" << (u.eligible ? "true" : "false");
    if (!u.eligible) o << ",\"why_not\":\"" << u.why_not << "\"";
    else {
        // (not in use: the gather kernel was cheaper, or tiles across two stride-1 modes or narrow ones run)
        o << ",\"in_use\":" << (!pl.across.on && !pl.narrow.eligible && (pl.kernel == KERNEL_UMMA_TF32 || pl.kernel == KERNEL_DMMA_F64_TMA) ? "true" : "false") << ",\"BM\":" << u.BM << ",\"BN\":" << u.BN << ",\"BK\":" << u.BK << ",\"stages\":" << u.stages
          << ",\"pair\":" << (u.pair ? "true" : "false") << ",\"kc\":\"" << u.kc_names << "\",\"k_iters\":" << u.k_iters << ",\"k_splits\":" << u.k_splits << ",\"tiles_m\":" << u.tiles_m << ",\"tiles_n\":" << u.tiles_n
          << ",\"a_major\":\"" << (u.a.major ? "MN" : "K") << "\",\"b_major\":\"" << (u.b.major ? "MN" : "K") << "\""
          << ",\"a_slab_w\":" << u.a.slab_w << ",\"b_slab_w\":" << u.b.slab_w << ",\"a_slabs_per_copy\":" << u.a.slabs_per_op << ",\"b_slabs_per_copy\":" << u.b.slabs_per_op << ",\"a_slabs\":" << u.a.slabs_per_tile
          << ",\"b_slabs\":" << u.b.slabs_per_tile << ",\"smem_bytes\":" << u.smem_bytes
          << ",\"coalesced_store\":" << (u.a.row_elem_cstride == 1 ? "true" : "false")
          << ",\"store_across_slabs\":" << (u.store_across_slabs ? "true" : "false") << ",\"slim\":" << (u.slim[0] ? "true" : "false") << ",\"slim_reads\":" << (u.slim[1] ? "true" : "false") << ",\"piece\":" << u.piece << ",\"groups\":[" << u.groups[0] << "," << u.groups[1] << "],\"producers\":" << u.producers
          << ",\"a_fused\":" << u.a.split_inner << ",\"b_fused\":" << u.b.split_inner << ",\"column_ranges\":[";
        std::string why;
        for (int r = 2, n = 0; r <= 8; ++r)
            if (cuts_into_ranges(pl, r, &why)) o << (n++ ? "," : "") << r;
        o << "]";
    }
    o << "}}";
    return o.str();
}

}  // namespace tcontb
