// across_tf32.cu -- TF32 contraction on the tensor cores (tcgen05, sm_100a) where A's stride-1 mode x is not C's, y:
// C[y, ..., x, ...] = sum A[x, k, ..., y] B.  umma_tf32.cu stores rows along A's stride-1 mode, here 4-byte pieces of C each in a
// sector of its own, or needs a copy of A with its modes exchanged first.
//
// A tile is 16 indices of y times 32 of x (one copy: 16 slabs of 32 x, MN-major, 128-byte swizzle in 32-byte units) by up to 64
// columns.  It is contracted as four groups of 128 rows; group g takes slabs g, g + 4, g + 8, g + 12 (the leading byte offset of
// the operand descriptor skips three slabs), so that a thread of the epilogue, which owns tensor-memory lane 32 q + x of all
// four accumulators, holds y = 4 q .. 4 q + 3 for one x: 16 neighbouring bytes of C.  Pieces of eight columns go through
// shared memory in 64-byte rows of y (64-byte swizzle, no bank conflicts either way) and leave by bulk tensor stores, whose
// bounds take care of ragged y, x and columns.
//
//   warp 0      producer: one elected thread, two or three copies a stage
//   warp 1      allocates tensor memory; an elected thread issues the MMAs (M 128, N 32 or 64, K 8) into one of two accumulator sets
//   warps 2-5   epilogue: tcgen05.ld -> shared memory, a ring of four buffers of eight columns
//   warp 6      one elected thread issues the bulk stores of filled buffers and frees them when they have been read
//
// What bounds it: the tensors' traffic (C of 226 MB from A of 302, 48 x 32 x 24 x 32 x 48 by 32: 311 us with the copy of A, 106
// here, 5.0 TB/s), for short contracted extents C leaving in pieces of 64 bytes (24 x 32 x 24 x 24 x 32 by 8, 57 MB: 22 -> 13.5 us),
// for the smallest the way through one tile (16 x 8 x 8 x 8 x 16 by 8: 7.4 -> 4.5 us).  A first form without warp 6, its epilogue
// working out every tile's coordinates, took 2.0 us a tile beside the pieces (109 and 29.7 us).
// Every wait is bounded as in umma_tf32.cu, with the same test hooks.
//
// Stands where the reference runs its generated TF32 WMMA kernels (backends/cogent/plan/generators/kernels/kernel_store.py:280-507).
#include <cuda.h>

#include "chain.cuh"
#include "kernels.hpp"
#include "tcgen05.cuh"
#include "tile_common.cuh"

namespace tcontb {
namespace {

constexpr int kAcrossThreads = 224;
constexpr int kBuffers = 4;                    // staged pieces of C: 512 rows x 8 columns each
constexpr uint32_t kHalfBytes = 16 * 16 * 8 * 4, kBufferBytes = 2 * kHalfBytes;

__device__ __forceinline__ void tma_store_5d(const void* tmap, uint32_t src, int c0, int c1, int c2, int c3, int c4)
{
    asm volatile("cp.async.bulk.tensor.5d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5, %6}], [%1];"
                 ::"l"(reinterpret_cast<uint64_t>(tmap)), "r"(src), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
                 : "memory");
}

// A tile's indices: chunks of y, x and n and the other modes of its rows and columns.  The planner puts the other row modes
// first among the last dimensions of A's and C's maps, the other column modes first among B's, so that a coordinate is a choice
// between two or three of them; a mode that is not there has extent 1.
struct TileIndex {
    int y, x, o0, o1, n, p0, p1;
};
__device__ __forceinline__ TileIndex tile_index(uint32_t unit, const AcrossParams& p)
{
    TileIndex t;
    uint32_t q = fast_div(unit, p.inner), tm = unit - q * p.inner.d, tn = q;
    if (!p.rows_first) {
        tn = tm;
        tm = q;
    }
    q = fast_div(tm, p.y_chunks);
    t.y = static_cast<int>(tm - q * p.y_chunks.d) * 16;
    if (!p.rows_first) {
        tm = fast_div(q, p.x_chunks);
        t.x = static_cast<int>(q - tm * p.x_chunks.d) * 32;
        q = tm;
    }
    tm = fast_div(q, p.o0);
    t.o0 = static_cast<int>(q - tm * p.o0.d);
    q = fast_div(tm, p.o1);
    t.o1 = static_cast<int>(tm - q * p.o1.d);
    if (p.rows_first) t.x = static_cast<int>(q) * 32;
    q = fast_div(tn, p.n_chunks);
    t.n = static_cast<int>(tn - q * p.n_chunks.d) * p.BN;
    tn = fast_div(q, p.p0);
    t.p0 = static_cast<int>(q - tn * p.p0.d);
    t.p1 = static_cast<int>(tn);
    return t;
}

__global__ void __launch_bounds__(kAcrossThreads, 1)
across_tf32_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB, const __grid_constant__ CUtensorMap tmapC,
                   const __grid_constant__ AcrossParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // 1024-byte aligned
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t slab_bytes = static_cast<uint32_t>(p.BK) * 128u, a_bytes = 16u * slab_bytes;
    const uint32_t b_bytes = static_cast<uint32_t>(p.BN * p.BK) * 4u, stage_bytes = a_bytes + b_bytes;
    const uint32_t buffers = smem_u32(smem) + static_cast<uint32_t>(p.stages) * stage_bytes;
    uint8_t* aux = smem + static_cast<size_t>(p.stages) * stage_bytes + kBuffers * kBufferBytes;
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(aux);  // [8]
    uint64_t* bar_empty = bar_full + 8;                     // [8]
    uint64_t* bar_tfull = bar_empty + 8;                    // [2]
    uint64_t* bar_tempty = bar_tfull + 2;                   // [2]
    uint64_t* bar_staged = bar_tempty + 2;                  // [kBuffers]
    uint64_t* bar_free = bar_staged + kBuffers;             // [kBuffers]
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bar_free + kBuffers);
    const uint32_t abort_flag = smem_u32(tmem_slot + 1);
    const uint32_t bar_drain = smem_u32(tmem_slot + 2);
    const uint32_t tmem_cols = static_cast<uint32_t>(8 * p.BN);   // two sets of four accumulators: 256 or 512

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(bar_full + s), 1);
            mbar_init(smem_u32(bar_empty + s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(smem_u32(bar_tfull + a), 1);
            mbar_init(smem_u32(bar_tempty + a), 128);
        }
        for (int b = 0; b < kBuffers; ++b) {
            mbar_init(smem_u32(bar_staged + b), 128);
            mbar_init(smem_u32(bar_free + b), 1);
        }
        mbar_init(bar_drain, 1);
        st_shared_u32(abort_flag, 0u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tcgen05_fence_before();
    if (!p.release_late) chain_release();
    chain_wait();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    auto wait = [&](uint32_t bar, uint32_t parity) { return mbar_wait(bar, parity, abort_flag, 0, p.wait_limit_ns); };
    // columns of a tile that lie inside C
    auto columns_of = [&](uint32_t unit) {
        uint32_t tn = fast_div(unit, p.inner);
        if (!p.rows_first) tn = unit - tn * p.inner.d;
        const uint32_t q = fast_div(tn, p.n_chunks);
        const int left = p.n_ext - static_cast<int>(tn - q * p.n_chunks.d) * p.BN;
        return left < p.BN ? left : p.BN;
    };

    if (warp == 0) {
        if (elect_one()) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmapA)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmapB)) : "memory");
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmapC)) : "memory");
            int stage = 0, cta_iter = 0;
            uint32_t phase = 0, issued_mask = 0, issued_parity = 0;
            const int b_copies = p.b_major ? p.BN / 32 : 1;
            TileIndex next = tile_index(blockIdx.x, p);
            for (uint32_t unit = blockIdx.x; unit < p.units; unit += gridDim.x) {
                const TileIndex t = next;
                int k0 = 0, k1 = 0, k2 = 0;
                for (int it = 0; it < p.k_iters; ++it, ++cta_iter) {
                    if (wait(smem_u32(bar_empty + stage), phase ^ 1u) && cta_iter != p.test_skip_iter) {
                        const uint32_t bar = smem_u32(bar_full + stage), dst = smem_u32(smem) + static_cast<uint32_t>(stage) * stage_bytes;
                        mbar_arrive_expect_tx(bar, stage_bytes);
                        tma_load_5d(dst, &tmapA, bar, t.x, k0, t.y, p.row_others > 0 ? t.o0 : k1, p.row_others > 1 ? t.o1 : p.row_others == 1 ? k1 : k2);
                        const int b2 = p.column_others > 0 ? t.p0 : k1, b3 = p.column_others > 1 ? t.p1 : p.column_others == 1 ? k1 : k2;
                        const int b4 = p.column_others > 1 ? k1 : p.column_others == 1 ? k2 : 0;
                        for (int c = 0; c < b_copies; ++c)
                            tma_load_5d(dst + a_bytes + static_cast<uint32_t>(c) * slab_bytes, &tmapB, bar, p.b_major ? t.n + c * 32 : k0, p.b_major ? k0 : t.n, b2, b3, b4);
                        issued_mask |= 1u << stage;
                        issued_parity = (issued_parity & ~(1u << stage)) | (phase << stage);
                    }
                    if (it == 0) next = tile_index(unit + gridDim.x, p);   // (behind the first copies of this tile; not used past the last)
                    k0 += p.BK;
                    if (k0 >= p.k_ext) {
                        k0 = 0;
                        if (++k1 == p.k1_ext) {
                            k1 = 0;
                            ++k2;
                        }
                    }
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (p.release_late) chain_release();
            if (ld_shared_u32(abort_flag)) drain_copies(smem_u32(bar_full), p.stages, issued_mask, issued_parity);
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (1u << 15) | (static_cast<uint32_t>(p.b_major) << 16) |
                                   (static_cast<uint32_t>(p.BN >> 3) << 17) | ((128u >> 4) << 24);
            const uint64_t a_desc = smem_desc(0u, 4u * slab_bytes, 512u, 1u);   // rows of a group: every fourth slab
            const uint64_t b_desc = smem_desc(0u, p.b_major ? slab_bytes : 16u, p.b_major ? 512u : 1024u, p.b_major ? 1u : 2u);
            const uint32_t b_step = p.b_major ? 1024u : 32u;
            const int ksteps = p.BK / 8;
            int stage = 0;
            uint32_t phase = 0, tile = 0;
            for (uint32_t unit = blockIdx.x; unit < p.units; unit += gridDim.x, ++tile) {
                const uint32_t acc = tile & 1u;
                bool ok = wait(smem_u32(bar_tempty + acc), ((tile >> 1) & 1u) ^ 1u);
                tcgen05_fence_after();
                const uint32_t tmem_c = tmem_base + acc * 4u * static_cast<uint32_t>(p.BN);
                for (int it = 0; it < p.k_iters; ++it) {
                    ok = ok && wait(smem_u32(bar_full + stage), phase);
                    if (ok) {
                        tcgen05_fence_after();
                        const uint32_t a = smem_u32(smem) + static_cast<uint32_t>(stage) * stage_bytes, b = a + a_bytes;
                        for (int kk = 0; kk < ksteps; ++kk) {
                            const uint64_t db = b_desc + ((b + static_cast<uint32_t>(kk) * b_step) >> 4);
#pragma unroll
                            for (uint32_t g = 0; g < 4; ++g)
                                umma_tf32(tmem_c + g * static_cast<uint32_t>(p.BN), a_desc + ((a + g * slab_bytes + static_cast<uint32_t>(kk) * 1024u) >> 4), db,
                                          idesc, (it | kk) != 0 ? 1u : 0u);
                        }
                        umma_commit(smem_u32(bar_empty + stage));
                    }
                    if (++stage == p.stages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (ok) umma_commit(smem_u32(bar_tfull + acc));
            }
            if (ld_shared_u32(abort_flag)) {   // MMAs of stages that did arrive may be running: they end before tensor memory is given back
                umma_commit(bar_drain);
                drain_copies(bar_drain, 1, 1u, 0u);
            }
        }
        __syncwarp();
    } else if (warp < 6) {
        const uint32_t q = static_cast<uint32_t>(warp & 3), xi = static_cast<uint32_t>(lane & 15);   // tensor-memory quadrant = quarter of the y
        const uint32_t piece = static_cast<uint32_t>(lane >> 4) * kHalfBytes + xi * 64u + ((q ^ ((xi >> 1) & 3u)) << 4);
        uint32_t tile = 0, buffer = 0, round = 0;
        for (uint32_t unit = blockIdx.x; unit < p.units; unit += gridDim.x, ++tile) {
            const uint32_t acc = tile & 1u;
            const int columns = columns_of(unit);
            bool ok = wait(smem_u32(bar_tfull + acc), (tile >> 1) & 1u);
            ok = __all_sync(0xffffffffu, ok);
            tcgen05_fence_after();
            const uint32_t taddr = tmem_base + (q << 21) + acc * 4u * static_cast<uint32_t>(p.BN);   // (lane 32 q in bits 16 and up)
            for (int j0 = 0; j0 < columns; j0 += 8) {
                uint32_t v[4][8];
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) tmem_ld_32x8(taddr + g * static_cast<uint32_t>(p.BN) + static_cast<uint32_t>(j0), v[g]);
                ok = __all_sync(0xffffffffu, wait(smem_u32(bar_free + buffer), (round & 1u) ^ 1u)) && ok;
                tmem_ld_wait();
                if (j0 + 8 >= columns) {   // all of the tile is in registers
                    tcgen05_fence_before();
                    mbar_arrive(smem_u32(bar_tempty + acc));
                }
                const uint32_t to = buffers + buffer * kBufferBytes + piece;
                if (ok) {
#pragma unroll
                    for (uint32_t j = 0; j < 8; ++j)
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + j * 1024u), "r"(v[0][j]), "r"(v[1][j]), "r"(v[2][j]), "r"(v[3][j]) : "memory");
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                mbar_arrive(smem_u32(bar_staged + buffer));
                if (++buffer == kBuffers) {
                    buffer = 0;
                    ++round;
                }
            }
        }
    } else {
        if (elect_one()) {
            uint32_t buffer = 0, round = 0, last = kBuffers;   // (last: the buffer whose store may still be reading)
            for (uint32_t unit = blockIdx.x; unit < p.units; unit += gridDim.x) {
                const TileIndex t = tile_index(unit, p);
                const int columns = columns_of(unit);
                const int c3 = p.row_others > 0 ? t.o0 : t.p0, c4 = p.row_others > 1 ? t.o1 : p.row_others == 1 ? t.p0 : t.p1;
                for (int j0 = 0; j0 < columns; j0 += 8) {
                    if (wait(smem_u32(bar_staged + buffer), round & 1u) && !ld_shared_u32(abort_flag)) {   // (a piece that was not staged is not stored)
                        const uint32_t from = buffers + buffer * kBufferBytes;
                        tma_store_5d(&tmapC, from, t.y, t.x, t.n + j0, c3, c4);
                        if (t.x + 16 < p.x_ext) tma_store_5d(&tmapC, from + kHalfBytes, t.y, t.x + 16, t.n + j0, c3, c4);
                    }
                    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
                    asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                    if (last < kBuffers) mbar_arrive(smem_u32(bar_free + last));
                    last = buffer;
                    if (++buffer == kBuffers) {
                        buffer = 0;
                        ++round;
                    }
                }
            }
            asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
        __syncwarp();
    }

    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols) : "memory");
    if (threadIdx.x == 0 && ld_shared_u32(abort_flag)) atomicMax(p.status, 1);
}

}  // namespace

int across_tf32_smem(int stages, int BN, int BK) { return stages * (16 * 128 * BK + BN * BK * 4) + kBuffers * static_cast<int>(kBufferBytes) + 256 + 1024; }

cudaError_t across_tf32_configure()
{
    return cudaFuncSetAttribute(across_tf32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmemBytes);
}

cudaError_t launch_across_tf32(const AcrossParams& p, const void* tmapA, const void* tmapB, const void* tmapC, int num_sms, cudaStream_t stream)
{
    if (p.units == 0 || p.stages < 2 || p.stages > 8 || (p.BN != 32 && p.BN != 64) || p.BK < 8 || p.BK > 32 || p.BK % 8) return cudaErrorInvalidValue;
    const unsigned grid = p.units < static_cast<uint32_t>(num_sms) ? p.units : static_cast<unsigned>(num_sms);
    int smem = across_tf32_smem(p.stages, p.BN, p.BK);
    smem = smem > kMaxDynamicSmemBytes / 2 + 1024 ? smem : kMaxDynamicSmemBytes / 2 + 1024;   // (one persistent CTA an SM, see launch_umma_tf32)
    return launch_chained(across_tf32_kernel, dim3(grid), dim3(kAcrossThreads), static_cast<size_t>(smem), stream, 1, *static_cast<const CUtensorMap*>(tmapA),
                          *static_cast<const CUtensorMap*>(tmapB), *static_cast<const CUtensorMap*>(tmapC), p);
}

}  // namespace tcontb
