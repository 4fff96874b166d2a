// tile_common.cuh -- device helpers shared by the TMA-fed kernels (tcgen05 TF32 and FP64 tensor
// path): mbarrier and bulk-tensor-copy wrappers, bounded waits, tile rasterisation and the
// mixed-radix slab arithmetic that maps a tile row or column to its place in C.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "fast_div.cuh"
#include "kernels.hpp"

namespace tcontb {
namespace {

constexpr unsigned long long kWaitLimitNs = 2000000000ull;  // 2 s

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ unsigned long long global_timer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// One look at the barrier without waiting (try_wait may suspend the thread for a while).
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity)
{
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// Bounded wait.  Returns false (and raises the CTA's abort flag) when the limit passes, or
// immediately when another thread of the CTA already gave up.
__device__ __forceinline__ uint32_t ld_shared_u32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.volatile.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
__device__ __forceinline__ void st_shared_u32(uint32_t addr, uint32_t v)
{
    asm volatile("st.volatile.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_shared_s64(uint32_t addr, long long v)
{
    asm volatile("st.shared.b64 [%0], %1;" ::"r"(addr), "l"(v) : "memory");
}
__device__ __forceinline__ long long ld_shared_s64(uint32_t addr)
{
    long long v;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(v) : "r"(addr) : "memory");
    return v;
}

// Bounded wait.  The fast path is a bare try_wait; every 256 failed polls it looks at the CTA's
// abort flag (shared-memory word at `abort_addr`) and at the clock.  Returns false, and raises the
// flag, when the limit passes; returns false at once when another thread already gave up.
// `sleep_ns` > 0: the thread sleeps that long after a failed poll, for warps whose polling would
// otherwise take issue slots from the warps doing the arithmetic on the same scheduler.
// `limit_ns` = 0 means the default limit.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint32_t abort_addr, uint32_t sleep_ns = 0,
                                          unsigned long long limit_ns = 0)
{
    const unsigned long long limit = limit_ns ? limit_ns : kWaitLimitNs;
    unsigned long long t0 = 0;
    for (uint32_t spin = 0;; ++spin) {
        if (mbar_try_wait(bar, parity)) return true;
        if (sleep_ns) __nanosleep(sleep_ns);
        if ((spin & 255u) == 255u || spin == 0) {
            if (ld_shared_u32(abort_addr)) return false;
            if (spin == 0) continue;
            const unsigned long long now = global_timer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit) {
                st_shared_u32(abort_addr, 1u);
                return false;
            }
        }
    }
}

// Give the bulk copies issued into these barriers a bounded time to land before the CTA ends (after a wait gave up).
__device__ __forceinline__ void drain_copies(uint32_t bar_full, int stages, uint32_t issued_mask, uint32_t issued_parity)
{
    for (int s = 0; s < stages; ++s) {
        if (!(issued_mask & (1u << s))) continue;
        const unsigned long long t0 = global_timer();
        while (!mbar_try_wait(bar_full + 8u * static_cast<uint32_t>(s), (issued_parity >> s) & 1u))
            if (global_timer() - t0 > 100000000ull) break;
    }
}

__device__ __forceinline__ void tma_load_5d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1, int c2, int c3, int c4)
{
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(tmap)), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// Raster order: groups of raster_group tile rows are swept column by column, so the CTAs that run
// together share A and B panels in L2.  Tile and slab counts fit 31 bits (the planner checks).
__device__ __forceinline__ void decode_tile(uint32_t tile, const UmmaParams& p, uint32_t tiles_m, uint32_t tiles_n, uint32_t* tm, uint32_t* tn)
{
    const uint32_t g = static_cast<uint32_t>(p.raster_group);
    const uint32_t group = fast_div(tile, p.div_group);
    const uint32_t first_m = group * g;
    const bool whole = tiles_m - first_m >= g;
    const uint32_t local = tile - group * g * tiles_n;
    *tn = whole ? fast_div(local, p.div_rows) : fast_div(local, p.div_last_rows);
    *tm = first_m + local - *tn * (whole ? g : tiles_m - first_m);
}

// A unit of work: one tile, or with split-K one range of a tile's k iterations.  Units are numbered
// tile * k_splits + split.
struct WorkUnit {
    uint32_t tm, tn, split;
    int it0, n_it;
};
__device__ __forceinline__ WorkUnit decode_unit(uint32_t unit, const UmmaParams& p, uint32_t tiles_m, uint32_t tiles_n)
{
    WorkUnit w;
    const uint32_t splits = static_cast<uint32_t>(p.k_splits);
    const uint32_t tile = splits > 1 ? fast_div(unit, p.div_splits) : unit;
    w.split = splits > 1 ? unit - tile * splits : 0u;
    decode_tile(tile, p, tiles_m, tiles_n, &w.tm, &w.tn);
    w.tn += static_cast<uint32_t>(p.tn_rotate);   // (below tiles_n)
    if (w.tn >= tiles_n) w.tn -= tiles_n;
    w.it0 = static_cast<int>(w.split) * p.k_iters_per_split;
    w.n_it = p.k_iters - w.it0 < p.k_iters_per_split ? p.k_iters - w.it0 : p.k_iters_per_split;
    return w;
}

// Splits a slab index into its mixed-radix digits and returns the C offset of the slab start.
// valid = false when the slab lies beyond the tensor.
__device__ __forceinline__ long long slab_c_offset(const UmmaOperandDev& o, uint32_t slab, int* digit0, bool* valid)
{
    *valid = slab < static_cast<uint32_t>(o.total_slabs);
    uint32_t rem = slab;
    long long off = 0;
#pragma unroll
    for (int d = 0; d < kMaxTmaRank; ++d) {
        if (d < o.n_row_digits) {
            const uint32_t q = fast_div(rem, o.row_digit_ext[d]);
            const uint32_t idx = rem - q * o.row_digit_ext[d].d;
            rem = q;
            off += static_cast<long long>(idx) * o.row_digit_cstride[d];
            if (d == o.chunk_digit) *digit0 = static_cast<int>(idx);
        }
    }
    return off;
}

// C offset of position `in` of a slab whose digit-0 index is `digit0`, relative to what slab_c_offset returned.
// With operand-level row fusion (split_inner > 0) the slab mode is two C modes, and digit 0 carries no C
// stride of its own: the position inside the fused mode is split here.
__device__ __forceinline__ long long slab_elem_offset(const UmmaOperandDev& o, int digit0, int in)
{
    if (o.split_inner > 0) {
        const int pos = digit0 * o.slab_w + in;
        const int outer = static_cast<int>(fast_div(static_cast<uint32_t>(pos), o.split_div));
        return static_cast<long long>(pos - outer * o.split_inner) * o.row_elem_cstride +
               static_cast<long long>(outer) * o.split_outer_cstride;
    }
    return static_cast<long long>(in) * o.row_elem_cstride;
}

// TMA coordinates of the box that starts at slab `s` (the k coordinates come on top).
__device__ __forceinline__ void slab_coords(const UmmaOperandDev& o, uint32_t s, int (&base)[kMaxTmaRank])
{
#pragma unroll
    for (int t = 0; t < kMaxTmaRank; ++t) base[t] = 0;
    if (s < static_cast<uint32_t>(o.total_slabs)) {
        uint32_t rem = s;
#pragma unroll
        for (int d = 0; d < kMaxTmaRank; ++d) {
            if (d < o.n_row_digits) {
                const uint32_t q = fast_div(rem, o.row_digit_ext[d]);
                const int idx = static_cast<int>(rem - q * o.row_digit_ext[d].d);
                rem = q;
                const int v = d == o.chunk_digit ? idx * o.digit0_scale : idx;
#pragma unroll
                for (int t = 0; t < kMaxTmaRank; ++t)
                    if (o.row_digit_dim[d] == t) base[t] = v;
            }
        }
    } else {
        // Slab beyond the tensor: start the box past the slab mode's end, TMA fills zeros.
#pragma unroll
        for (int t = 0; t < kMaxTmaRank; ++t)
            if (o.row_digit_dim[o.chunk_digit] == t) base[t] = o.oob_coord;
    }
}

// What one step of k digit 0, 1, 2 adds to each TMA coordinate of an operand, and the coordinates themselves.
struct KSteps {
    int s0[kMaxTmaRank], s1[kMaxTmaRank], s2[kMaxTmaRank];
};
__device__ __forceinline__ void k_steps(const UmmaOperandDev& o, KSteps& k)
{
#pragma unroll
    for (int t = 0; t < kMaxTmaRank; ++t) {
        k.s0[t] = o.k_digit_dim[0] == t ? o.k0_scale : 0;
        k.s1[t] = o.k_digit_dim[1] == t ? 1 : 0;
        k.s2[t] = o.k_digit_dim[2] == t ? 1 : 0;
    }
}
// (a tensor dimension carries either a row digit or a k digit, so the two parts never meet in one coordinate)
__device__ __forceinline__ void k_coords(const int (&base)[kMaxTmaRank], const KSteps& k, int kd0, int kd1, int kd2, int (&c)[kMaxTmaRank])
{
#pragma unroll
    for (int t = 0; t < kMaxTmaRank; ++t) c[t] = base[t] + kd0 * k.s0[t] + kd1 * k.s1[t] + kd2 * k.s2[t];
}

}  // namespace
}  // namespace tcontb
