// dmma_tma_f64.cu -- FP64 direct contraction: TMA-staged operand tiles feeding mma.sync m8n8k4.
//
// tcgen05 has no FP64 kind, so the arithmetic is warp-level DMMA (37.0 TFLOP/s measured on B200).
// What the gather kernel (gather_contract.cu) spends on address arithmetic is done here by the copy
// engine: the planner's slab machinery, the same as for the tcgen05 kernel but with 16 doubles per
// 128-byte row, describes every operand tile as a few multi-mode TMA boxes.
//
// One block per SM, three warpgroups; setmaxnreg moves the register budget from the first (56 per
// thread) to the other two (224):
//   warps 0, 1  producers, one per consumer group: lane i issues copy i of a stage (5-D tensor
//               maps, 128-byte swizzle, no multicast) into the group's own ring of stages,
//               full/empty mbarriers per stage, the ring runs across tile boundaries
//   warps 2, 3  table builders: for every tile, ahead of time, the C offset of each of its 128 rows
//               and 64 columns (mixed-radix slab arithmetic, the same as the tcgen05 epilogue),
//               double-buffered per group behind mbarriers
//   warps 4-7   consumer group 0, warps 8-11 consumer group 1.  A group is 2 x 2 warps with a
//               64 x 32 warp tile (8 x 4 accumulator fragments; 64 x 16 in the 128 x 32 variant for
//               narrow N) and takes every other tile of the block.  Group 1 starts half a main loop late, so one group's stores fall into the
//               other's main loop instead of both storing with the FP64 pipe idle.
// Fragment rows are permuted so that one 16-byte shared load of an MN-major operand feeds two
// fragments (rows 2 r and 2 r + 1 of a 16-row slab; two-way bank conflicts with k in ascending order, which cost nothing that could be timed:
// 2048 x 8000 x 24 36.7 us, 36.6 with an order without them), and the MMA is issued
// transposed (B fragment as the row operand): a thread then owns four consecutive elements of C's
// stride-1 mode per fragment pair and a warp store instruction writes eight whole 128-byte lines.
// The loads of the next k step are issued between the MMAs of the current one.
// Every wait is bounded and raises the run's status word instead of hanging.
//
// Stands where the reference runs its generated FP64 WMMA kernels
// (backends/cogent/plan/generators/kernels/kernel_compute.py:127-850) and its cublasGemmEx FP64
// call (backends/ttgt_cutt/src/ttgt_cutt.cpp:764-809).
#include <cuda.h>

#include <type_traits>

#include "chain.cuh"
#include "kernels.hpp"
#include "tile_common.cuh"

namespace tcontb {
namespace {

constexpr int kThreads64 = 384;
constexpr int kBM = 128, kMaxBN = 64;
constexpr uint32_t kTabBytes = (kBM + kMaxBN) * 8u;  // one tile's row and column offsets
constexpr long long kBeyond = -(1ll << 61);          // entry of a row or column beyond C: a sum with any other entry is negative

__device__ __forceinline__ double ld_shared_f64(uint32_t addr)
{
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void ld_shared_v2f64(uint32_t addr, double& x, double& y)
{
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(x), "=d"(y) : "r"(addr));
}

__device__ __forceinline__ void dmma_m8n8k4(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}

__device__ __forceinline__ void st_global_cs_v4f64(double* p, double a, double b, double c, double d)
{
    asm volatile("st.global.cs.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(a), "d"(b), "d"(c), "d"(d) : "memory");
}

// The same at C + offset, by predicate: not where `offset` is negative.
__device__ __forceinline__ void st_global_cs_v4f64_in(double* C, long long offset, double a, double b, double c, double d)
{
    asm volatile("{\n .reg .pred in;\n setp.ge.s64 in, %5, 0;\n @in st.global.cs.v4.f64 [%0], {%1, %2, %3, %4};\n}" ::"l"(C + offset), "d"(a), "d"(b), "d"(c),
                 "d"(d), "l"(offset)
                 : "memory");
}

__device__ __forceinline__ void st_global_cs_v2f64_in(double* C, long long offset, double a, double b)
{
    asm volatile("{\n .reg .pred in;\n setp.ge.s64 in, %3, 0;\n @in st.global.cs.v2.f64 [%0], {%1, %2};\n}" ::"l"(C + offset), "d"(a), "d"(b), "l"(offset) : "memory");
}

__device__ __forceinline__ void ld_global_cs_v4f64(double (&o)[4], const double* p)
{
    asm volatile("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3]) : "l"(p) : "memory");
}

// Which k a lane feeds into step t of a stage: k = 4 t + fk, fk = lane % 4, so that an unsplit sum is one chain of FMAs in
// ascending order of k, the same bits as the gather kernel's.
__device__ __forceinline__ uint32_t step_k(uint32_t t, uint32_t fk) { return 4u * t + fk; }

// Where a thread finds its fragments of one operand, as byte offsets from the start of the stage:
//   MN-major (rows of the stage are k, 16 consecutive m per 128-byte row, slabs of 16 m one slab apart;
//   or 8 m per 64-byte row, two slabs per 16 m):
//     one 16-byte load at  step + pair * PITCH  holds fragments 2 pair and 2 pair + 1
//   K-major (rows of the stage are m, BK consecutive k per row: 128 bytes, or 64 with a k chunk of 8):
//     fragment i at  step + (i odd ? odd : 0) + (i / 2) * PITCH,  PITCH = 16 rows
// The 16-byte chunk index inside a row is XORed with (row % 8) (128-byte rows, 128-byte swizzle) or
// with (row / 2) % 4 (64-byte rows, 64-byte swizzle).  In all of them 16 m are BK * 128 bytes apart, step 1 differs from step 0
// and steps 2, 3 from 0, 1 by a thread's own constant: worked out once per block, because between two MMAs of a warp every
// instruction is time in which it feeds the pipe nothing (5184^3: 8 670 us with the offsets worked out per step and two ways
// through a stage, 8 246 now; the pipe is active in 95 % of the cycles of 2304^3).
template <int BK>
struct FragOffsets {
    static constexpr uint32_t PITCH = BK * 128u;
    uint32_t step0, step1, later, odd;
    uint32_t single;   // K-major, from row 2 fr to row 2 (fr % 4) + fr / 4: a fragment that is not one of a pair

    // `slabs8`: MN-major rows of 64 bytes (slabs of 8); the thread's slab, fr / 4, is already part of thread_base
    template <bool MN>
    __device__ __forceinline__ void set(uint32_t thread_base, uint32_t fr, uint32_t fk, bool slabs8)
    {
        auto offset = [&](uint32_t t) {
            const uint32_t k = step_k(t, fk);
            if (MN) return slabs8 ? thread_base + k * 64u + (((fr & 3u) ^ ((k >> 1) & 3u)) << 4) : thread_base + k * 128u + ((fr ^ (k & 7u)) << 4);
            const uint32_t kk = (k & 1u) * 8u, kc = k >> 1;
            return thread_base + kk + (BK == 8 ? (kc ^ (fr & 3u)) << 4 : (kc ^ ((2u * fr) & 7u)) << 4);   // (rows 2 fr and 2 fr + 1 share (row / 2) % 4)
        };
        step0 = offset(0);
        step1 = offset(1);
        later = offset(2) - step0;
        odd = MN ? 0u : BK == 8 ? 64u : (fk & 2u) ? 112u : 144u;   // the next row, its chunk index with bit 0 flipped
        single = fr < 4u ? 0u : odd - 8u * (BK * 8u);
    }
};

template <bool MN, int N, int BK>
__device__ __forceinline__ void load_frag(double (&f)[N], int i, uint32_t q, uint32_t odd)
{
    if (MN) {
        if ((i & 1) == 0) ld_shared_v2f64(q + static_cast<uint32_t>(i >> 1) * FragOffsets<BK>::PITCH, f[i], f[i + 1]);
    } else {
        f[i] = ld_shared_f64(q + ((i & 1) ? odd : 0u) + static_cast<uint32_t>(i >> 1) * FragOffsets<BK>::PITCH);
    }
}

// The last of an odd number of K-major fragments: eight rows of its own.
template <int N, int BK>
__device__ __forceinline__ void load_single(double (&f)[N], uint32_t q, uint32_t single)
{
    f[N - 1] = ld_shared_f64(q + single + static_cast<uint32_t>(N >> 1) * FragOffsets<BK>::PITCH);
}

// load N fragments (8 of A, 1 to 4 of B), all at once
template <bool MN, int N, int BK>
__device__ __forceinline__ void load_all(double (&f)[N], uint32_t q, const FragOffsets<BK>& o)
{
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if ((N & 1) && i == N - 1) load_single<N, BK>(f, q, o.single);
        else load_frag<MN, N, BK>(f, i, q, o.odd);
    }
}

// One k4 step of a warp: 8 NF MMAs on the current fragments (NF column fragments); the fragment loads of the next
// step are issued between them, where the FP64 tensor pipe leaves issue slots free.
// acc[i][j][h]: row m = 16 (i / 2) + 4 (lane % 4) + 2 h + (i % 2), column n = column_of(j).
template <bool AMN, bool BMN, int NF, int BK, bool HALVES>
__device__ __forceinline__ void mma_step(double (&acc)[8][NF][2], const double (&ac)[8], const double (&bc)[NF], double (&an)[8],
                                         double (&bn)[NF], uint32_t qa, const FragOffsets<BK>& oa, uint32_t qb, const FragOffsets<BK>& ob, bool second)
{
    static_assert(!BMN || NF % 2 == 0, "fragments along the rows come in pairs");
    if (HALVES && !second) {   // (one branch a step: with one at every MMA 373 248 x 24 x 72 gained nothing)
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            dmma_m8n8k4(acc[i][0], bc[0], ac[i]);
            load_frag<AMN, 8, BK>(an, i, qa, oa.odd);
            if (i == 0) load_frag<false, NF, BK>(bn, 0, qb, ob.odd);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int j = 0; j < NF; ++j) dmma_m8n8k4(acc[i][j], bc[j], ac[i]);
        load_frag<AMN, 8, BK>(an, i, qa, oa.odd);
        if (BMN) {
            if ((i == 1 || i == 3) && i < NF) load_frag<true, NF, BK>(bn, i - 1, qb, ob.odd);
        } else if ((NF & 1) && i == NF - 1) {
            load_single<NF, BK>(bn, qb, ob.single);
        } else {
            if (i < NF) load_frag<false, NF, BK>(bn, i, qb, ob.odd);
        }
    }
}
// Column of a warp's fragment j that a lane's accumulators belong to (fr = lane / 4): pairs of fragments take 16 columns, a last
// one by itself eight.
template <int NF>
__device__ __forceinline__ uint32_t column_of(int j, uint32_t fr)
{
    if ((NF & 1) && j == NF - 1) return 16u * (NF >> 1) + 2u * (fr & 3u) + (fr >> 2);
    return 16u * static_cast<uint32_t>(j >> 1) + static_cast<uint32_t>(j & 1) + 2u * fr;
}

// SCALED: C = alpha A B + beta C in the epilogue (C read only when beta is not zero); a template parameter because the
// overwriting kernel has no registers to spare for it.  PIECES: every store is 32 aligned bytes (UmmaSpec::piece); one kernel with both
// epilogues is slower in either (9216 x 4096 x 24 102.5 us, 94.5 in a kernel of its own; 2050 x 8000 x 16 54.8 and 48.7).
// SLIM: one column of tiles, of at most 48 of its 64 columns or 24 of its 32 (B K-major).  Three column fragments a warp instead of
// four; or (HALVES) two for the warps of one half and one for the others, the other way round in the second group, so that every
// scheduler has three.  373 248 x 24 x 72 70.1 -> 65.0 us, 48 columns 128.5 -> 106.2, 200 000 x 24 x 200 83.8 -> 72.8.
template <bool AMN, bool BMN, int NF, int BK, bool SCALED, bool SLIM, bool PIECES>
__global__ void __launch_bounds__(kThreads64, 1)
dmma_tma_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                const __grid_constant__ UmmaParams p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // 1024-byte aligned
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int SA = p.a.slabs_per_tile, SB = p.b.slabs_per_tile;
    const uint32_t a_tile_bytes = static_cast<uint32_t>(SA * p.a.slab_bytes);
    const uint32_t stage_bytes = a_tile_bytes + static_cast<uint32_t>(SB * p.b.slab_bytes);

    uint8_t* aux = smem + static_cast<size_t>(p.stages) * stage_bytes;
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(aux);  // [8]
    uint64_t* bar_empty = bar_full + 8;                     // [8]
    const uint32_t abort_flag = smem_u32(bar_empty + 8);
    uint64_t* tab_full = bar_empty + 10;   // [group][buffer]
    uint64_t* tab_empty = tab_full + 4;    // [group][buffer]
    const uint32_t ragged = smem_u32(tab_empty + 4);   // [group][buffer]: 1 + number of the last tile with rows (not SLIM: or columns) beyond C
    const uint32_t tabs = smem_u32(aux + 256);  // [group][buffer]: long long [128] row offsets, [64] column offsets (kBeyond = beyond C)

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(bar_full + s), 1);
            mbar_init(smem_u32(bar_empty + s), 4);  // one arrival per consumer warp
        }
        for (int s = 0; s < 4; ++s) {
            mbar_init(smem_u32(tab_full + s), 64);  // every builder thread
            mbar_init(smem_u32(tab_empty + s), 4);  // one arrival per consumer warp
        }
        for (uint32_t t = 0; t < 4; ++t) st_shared_u32(ragged + t * 4u, 0u);
        st_shared_u32(abort_flag, 0u);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    chain_release();
    chain_wait();
    __syncthreads();

    const uint32_t tiles_m = static_cast<uint32_t>(p.tiles_m), tiles_n = static_cast<uint32_t>(p.tiles_n);
    const uint32_t total_tiles = tiles_m * tiles_n * static_cast<uint32_t>(p.k_splits);  // work units (tile, k range)
    const uint32_t my_tiles = blockIdx.x < total_tiles ? (total_tiles - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;
    const uint32_t ring = static_cast<uint32_t>(p.stages) / 2u;  // stages per group

    if (warp < 4) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp < 2) {
            // ---------------- TMA producer of group `warp`: lane i owns copy i of the stage ----------------
            const uint32_t first = static_cast<uint32_t>(warp) * ring;  // first stage of this group's ring
            const int OA = SA / p.a.slabs_per_op, OB = SB / p.b.slabs_per_op;
            const bool is_a = lane < OA;
            const bool active = lane < OA + OB;
            const UmmaOperandDev& o = is_a ? p.a : p.b;
            const void* tmap = is_a ? static_cast<const void*>(&tmapA) : static_cast<const void*>(&tmapB);
            const int slab = is_a ? lane * p.a.slabs_per_op : (lane - OA) * p.b.slabs_per_op;
            const uint32_t my_off = is_a ? static_cast<uint32_t>(slab * p.a.slab_bytes)
                                         : a_tile_bytes + static_cast<uint32_t>(slab * p.b.slab_bytes);
            if (lane == 0) {
                asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmapA)) : "memory");
                asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmapB)) : "memory");
            }
            KSteps ks;
            k_steps(o, ks);
            uint32_t stage = 0, phase = 0;
            uint32_t issued_mask = 0, issued_parity = 0;
            for (uint32_t i = static_cast<uint32_t>(warp); i < my_tiles; i += 2) {
                const WorkUnit w = decode_unit(blockIdx.x + i * gridDim.x, p, tiles_m, tiles_n);
                const uint32_t tm = w.tm, tn = w.tn;
                int base[kMaxTmaRank];
                slab_coords(o, (is_a ? tm * SA : tn * SB) + slab, base);
                int kd0 = 0, kd1 = 0, kd2 = 0;
                if (w.it0) {   // (a later k range of a split)
                    kd0 = w.it0 % p.k_digit_ext[0];
                    kd1 = w.it0 / p.k_digit_ext[0] % p.k_digit_ext[1];
                    kd2 = w.it0 / (p.k_digit_ext[0] * p.k_digit_ext[1]);
                }
                for (int it = 0; it < w.n_it; ++it) {
                    const uint32_t ps = first + stage;
                    const bool ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar_empty + ps), phase ^ 1u, abort_flag, 200u));
                    if (ok) {
                        if (lane == 0) mbar_arrive_expect_tx(smem_u32(bar_full + ps), stage_bytes);
                        __syncwarp();
                        if (active) {
                            int c[kMaxTmaRank];
                            k_coords(base, ks, kd0, kd1, kd2, c);
                            tma_load_5d(smem_u32(smem + static_cast<size_t>(ps) * stage_bytes + my_off), tmap,
                                        smem_u32(bar_full + ps), c[0], c[1], c[2], c[3], c[4]);
                        }
                        issued_mask |= 1u << ps;
                        issued_parity = (issued_parity & ~(1u << ps)) | (phase << ps);
                    }
                    if (++kd0 == p.k_digit_ext[0]) {
                        kd0 = 0;
                        if (++kd1 == p.k_digit_ext[1]) {
                            kd1 = 0;
                            ++kd2;
                        }
                    }
                    if (++stage == ring) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (ld_shared_u32(abort_flag) && lane == 0) {
                // Give the bulk copies issued into these barriers a bounded time to land before the block ends.
                for (int s = 0; s < p.stages; ++s) {
                    if (!(issued_mask & (1u << s))) continue;
                    const unsigned long long t0 = global_timer();
                    while (!mbar_try_wait(smem_u32(bar_full + s), (issued_parity >> s) & 1u))
                        if (global_timer() - t0 > 100000000ull) break;
                }
            }
        } else {
            // ---------------- table builders: 64 threads, three entries each per tile ----------------
            const int bt = threadIdx.x - 64;
            for (uint32_t i = 0; i < my_tiles; ++i) {
                const WorkUnit w = decode_unit(blockIdx.x + i * gridDim.x, p, tiles_m, tiles_n);
                const uint32_t tm = w.tm, tn = w.tn;
                const uint32_t slot = (i & 1u) * 2u + ((i >> 1) & 1u);  // group, buffer
                const uint32_t use = i >> 2;                            // how often this slot was filled before
                if (!mbar_wait(smem_u32(tab_empty + slot), (use & 1u) ^ 1u, abort_flag, 500u)) break;
                const uint32_t tab = tabs + slot * kTabBytes;
#pragma unroll
                for (int e3 = 0; e3 < 3; ++e3) {
                    const int e = bt + e3 * 64;
                    const bool is_row = e < kBM;
                    if (!is_row && e - kBM >= NF * 16) continue;
                    const UmmaOperandDev& o = is_row ? p.a : p.b;
                    const int idx = is_row ? e : e - kBM;
                    const int sl = idx >> o.slab_shift, in = idx & (o.slab_w - 1);
                    bool ok;
                    int d0 = 0;
                    const long long off = slab_c_offset(o, (is_row ? tm * SA : tn * SB) + sl, &d0, &ok);
                    ok = ok && (d0 * o.slab_w + in < o.slab_mode_ext);
                    if (SCALED && PIECES && (is_row || !SLIM) && !ok) st_shared_u32(ragged + slot * 4u, i + 1u);
                    st_shared_s64(tab + static_cast<uint32_t>(e) * 8u, ok ? off + slab_elem_offset(o, d0, in) : kBeyond);
                }
                mbar_arrive(smem_u32(tab_full + slot));
                if (SCALED && p.beta != 0.0) {
                    // The tile's old values are wanted about two tiles from now: bring them into L2.  Eight warps cannot keep
                    // enough reads of C in flight to hide DRAM behind the store phase, which had them wait there.
                    if (!mbar_wait(smem_u32(tab_full + slot), use & 1u, abort_flag)) break;   // the other builders' entries
                    const double* C = p.C64;
                    // one look per four rows (32 bytes), or across slabs per group of eight slabs (64 bytes)
                    const int step = p.store_across_slabs ? 1 : 4, looks = p.store_across_slabs ? 16 : kBM / 4;
                    for (int q = bt; q < looks * NF * 16; q += 64) {
                        const long long r = ld_shared_s64(tab + static_cast<uint32_t>((q % looks) * step) * 8u);
                        const long long c = ld_shared_s64(tab + static_cast<uint32_t>(kBM + q / looks) * 8u);
                        if (r >= 0 && c >= 0 && (step == 1 || (q % looks) % 4 == 0 || ((reinterpret_cast<uintptr_t>(C + r + c) & 127u) < 32u)))
                            asm volatile("prefetch.global.L2 [%0];" ::"l"(C + r + c));
                    }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
        // ---------------- consumers: two groups of 2 x 2 warps, warp tile 64 x 32 ----------------
        const int cw = warp & 3, grp = (warp >> 2) - 1, wm = cw & 1, wn = cw >> 1;
        const uint32_t fr = static_cast<uint32_t>(lane >> 2), fk = static_cast<uint32_t>(lane & 3);
        const uint32_t first = static_cast<uint32_t>(grp) * ring;
        const bool a8 = AMN && p.a.slab_w == 8, b8 = BMN && p.b.slab_w == 8;  // 16 m = two slabs of 8
        constexpr uint32_t PITCH = FragOffsets<BK>::PITCH;
        FragOffsets<BK> fa, fb;
        fa.template set<AMN>(AMN ? static_cast<uint32_t>(wm * 4) * PITCH + (a8 ? (fr >> 2) * static_cast<uint32_t>(p.a.slab_bytes) : 0u)
                                 : (static_cast<uint32_t>(wm * 64) + 2u * fr) * (BK * 8u), fr, fk, a8);
        const bool narrow = SLIM && NF == 2 && (wn ^ grp) != 0;
        const uint32_t col0 = SLIM ? (NF == 2 ? (narrow ? 16u : 0u) : static_cast<uint32_t>(wn) * 24u) : static_cast<uint32_t>(wn * NF * 8);   // the warp's columns
        fb.template set<BMN>(a_tile_bytes + (BMN ? static_cast<uint32_t>(wn * (NF / 2)) * PITCH + (b8 ? (fr >> 2) * static_cast<uint32_t>(p.b.slab_bytes) : 0u)
                                                 : (col0 + 2u * fr) * (BK * 8u)), fr, fk, b8);

        if (narrow) {   // its one fragment is not one of a pair
            fb.step0 += fb.single;
            fb.step1 += fb.single;
        }
        const bool second = !narrow;
        constexpr int W = SLIM && NF == 4 ? 3 : NF;   // column fragments of a warp (narrow: the first of them)
        constexpr bool HALVES = SLIM && NF == 2;
        double acc[8][W][2];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < W; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

        uint32_t stage = 0, phase = 0;
        const bool prof = p.prof != nullptr && (threadIdx.x & 127) == 0 && grp == 0;
        long long t_all = prof ? clock64() : 0, t_full = 0, t_main = 0, t_tab = 0, t_store = 0;

        for (uint32_t i = static_cast<uint32_t>(grp); i < my_tiles; i += 2) {
            long long t0 = prof ? clock64() : 0;
            // group 1 starts half a main loop behind group 0 (named barrier 1: 128 waiting, 128 arriving)
            if (i == 1) asm volatile("bar.sync 1, 256;" ::: "memory");

            const WorkUnit w = decode_unit(blockIdx.x + i * gridDim.x, p, tiles_m, tiles_n);
            double* __restrict__ C = p.C64 + static_cast<long long>(w.split) * p.split_stride;
            bool tile_ok;
            // One path through a stage, with few instructions that are not between two MMAs: the last step of a stage fetches the
            // first fragments of the next one, whose barrier is looked at a step earlier (behind the last stage of a tile the
            // fragments are fetched from that stage again and not used).  A wait that gave up leaves wrong fragments, and
            // tile_ok says so.
            double fa0[8], fb0[W], fa1[8], fb1[W];
            uint32_t chunk = static_cast<uint32_t>(w.it0 ? w.it0 % p.k_digit_ext[0] : 0);   // chunk of the chunked mode
            {
                const long long tw = prof ? clock64() : 0;
                tile_ok = mbar_wait(smem_u32(bar_full + first + stage), phase, abort_flag);
                tile_ok = __all_sync(0xffffffffu, tile_ok);
                if (prof) t_full += clock64() - tw;
            }
            uint32_t sb = smem_u32(smem) + (first + stage) * stage_bytes;
            load_all<AMN, 8, BK>(fa0, sb + fa.step0, fa);
            load_all<BMN, W, BK>(fb0, sb + fb.step0, fb);
            for (int left = w.n_it; left > 0; --left) {
                if (i == 0 && my_tiles > 1 && left == w.n_it - w.n_it / 2) asm volatile("bar.arrive 1, 256;" ::: "memory");
                const uint32_t bar_done = smem_u32(bar_empty + first + stage);
                if (++stage == ring) {
                    stage = 0;
                    phase ^= 1u;
                }
                uint32_t later_a = 0, later_b = 0;
                // (the last chunk of a mode that is 1 to 8 past a multiple of 16 holds zeros in its second half: 5184^3 with
                // contracted modes of 72 computed a tenth of its k for nothing, 9 520 us)
                if (BK == 16 && chunk < static_cast<uint32_t>(p.full_chunks)) {
                    mma_step<AMN, BMN, W, BK, HALVES>(acc, fa0, fb0, fa1, fb1, sb + fa.step1, fa, sb + fb.step1, fb, second);
                    later_a = fa.later;
                    later_b = fb.later;
                    mma_step<AMN, BMN, W, BK, HALVES>(acc, fa1, fb1, fa0, fb0, sb + fa.step0 + later_a, fa, sb + fb.step0 + later_b, fb, second);
                }
                const uint32_t bar_next = smem_u32(bar_full + first + stage);
                const bool more = left > 1, landed = !more || mbar_test_wait(bar_next, phase);
                mma_step<AMN, BMN, W, BK, HALVES>(acc, fa0, fb0, fa1, fb1, sb + fa.step1 + later_a, fa, sb + fb.step1 + later_b, fb, second);
                if (!__all_sync(0xffffffffu, landed)) tile_ok = __all_sync(0xffffffffu, mbar_wait(bar_next, phase, abort_flag)) && tile_ok;
                if (more) sb = smem_u32(smem) + (first + stage) * stage_bytes;
                mma_step<AMN, BMN, W, BK, HALVES>(acc, fa1, fb1, fa0, fb0, sb + fa.step0, fa, sb + fb.step0, fb, second);
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_done);  // this warp is done reading the stage
                if (++chunk == static_cast<uint32_t>(p.k_digit_ext[0])) chunk = 0;
            }
            if (prof) { const long long t1 = clock64(); t_main += t1 - t0; t0 = t1; }

            // the tile's offset tables were built while it was being computed
            const uint32_t slot = static_cast<uint32_t>(grp) * 2u + ((i >> 1) & 1u);
            tile_ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(tab_full + slot), (i >> 2) & 1u, abort_flag)) && tile_ok;
            const uint32_t row_tab = tabs + slot * kTabBytes, col_tab = row_tab + kBM * 8u;
            if (prof) { const long long t1 = clock64(); t_tab += t1 - t0; t0 = t1; }

            // Store.  Four elements of C a thread holds for each of 4 x W (u, column fragment) lie next to each other:
            //   rows along C    : rows 16 u + 4 fk + q, element q in acc[2 u + (q & 1)][j][q >> 1]
            //   rows across slabs: the warp's 64 rows are four slabs of 16, slab q is index a0 + q of C's stride-1 mode; row
            //                      4 fk + u of the four slabs, element q in acc[2 q + (u & 1)][j][u >> 1]
            long long cn[W];
#pragma unroll
            for (int j = 0; j < W; ++j)
                cn[j] = HALVES && narrow ? (j == 0 ? ld_shared_s64(col_tab + (col0 + column_of<1>(0, fr)) * 8u) : kBeyond)
                                         : ld_shared_s64(col_tab + (col0 + column_of<W>(j, fr)) * 8u);
            const uint32_t row_u = p.store_across_slabs ? 8u : 128u, row_q = p.store_across_slabs ? 128u : 8u;   // table bytes from u to u + 1, q to q + 1
            const uint32_t rows = row_tab + (static_cast<uint32_t>(wm * 64) + 4u * fk) * 8u;
            auto row_of = [&](int u, uint32_t q) { return ld_shared_s64(rows + static_cast<uint32_t>(u) * row_u + q * row_q); };   // C offset of element q of the four
            const bool whole = SCALED && PIECES && ld_shared_u32(ragged + slot * 4u) != i + 1u;
            // Straight-line: a warp alone on its scheduler takes 5 to 20 cycles for every instruction and branch between two stores (with
            // alignment and bounds tested per store 4 200 cycles a tile, whatever the pieces' layout; 1 700 here).  Pieces beyond C are
            // left out by predicate (tested per store, 300 000 x 40 x 24 took 50.1 us and accumulating 124, here 40.4 and 65.6); a whole
            // tile's old values are not (9216 x 4096 x 24 accumulating: 176 us by predicate, 167 without).
            auto store_pieces = [&](auto&& at, auto all) {
                constexpr bool ALL = decltype(all)::value;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const long long cm = row_of(u, 0);
                    if constexpr (SCALED) {   // the old values of all column fragments are asked for before the first is used
                        double old[W][4];
#pragma unroll
                        for (int j = 0; j < W; ++j) {
                            if (p.beta != 0.0 && (ALL ? !SLIM || cn[j] >= 0 : cm + cn[j] >= 0)) ld_global_cs_v4f64(old[j], C + cm + cn[j]);
                            else old[j][0] = old[j][1] = old[j][2] = old[j][3] = 0.0;
                        }
#pragma unroll
                        for (int j = 0; j < W; ++j)
#pragma unroll
                            for (int q = 0; q < 4; ++q) at(u, j, q) = p.alpha * at(u, j, q) + p.beta * old[j][q];
                    }
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        if (!ALL) st_global_cs_v4f64_in(C, cm + cn[j], at(u, j, 0), at(u, j, 1), at(u, j, 2), at(u, j, 3));
                        else if (!SLIM || cn[j] >= 0) st_global_cs_v4f64(C + cm + cn[j], at(u, j, 0), at(u, j, 1), at(u, j, 2), at(u, j, 3));
                    }
                }
            };
            auto store_tile = [&](auto&& at) {
                if constexpr (PIECES) {
                    if (!tile_ok) return;
                    if (SCALED && whole) store_pieces(at, std::bool_constant<SCALED>());
                    else store_pieces(at, std::false_type());
                } else if (tile_ok && p.piece == 2) {
                    // halves of 16 bytes, straight-line as above
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const long long r[2] = {row_of(u, 0), row_of(u, 2)};
                        if constexpr (SCALED) {
                            double2 old[W][2];
#pragma unroll
                            for (int j = 0; j < W; ++j)
#pragma unroll
                                for (int h = 0; h < 2; ++h)
                                    old[j][h] = p.beta != 0.0 && r[h] + cn[j] >= 0 ? __ldcs(reinterpret_cast<const double2*>(C + r[h] + cn[j])) : make_double2(0.0, 0.0);
#pragma unroll
                            for (int j = 0; j < W; ++j)
#pragma unroll
                                for (int q = 0; q < 4; ++q) at(u, j, q) = p.alpha * at(u, j, q) + p.beta * (q & 1 ? old[j][q >> 1].y : old[j][q >> 1].x);
                        }
#pragma unroll
                        for (int j = 0; j < W; ++j)
#pragma unroll
                            for (int h = 0; h < 2; ++h) st_global_cs_v2f64_in(C, r[h] + cn[j], at(u, j, 2 * h), at(u, j, 2 * h + 1));
                    }
                } else if (tile_ok) {
                    // 32 bytes where they can be, 16 where two elements are neighbours, else one by one
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        long long r[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) r[q] = row_of(u, static_cast<uint32_t>(q));
                        const bool run4 = r[0] >= 0 && r[1] == r[0] + 1 && r[2] == r[0] + 2 && r[3] == r[0] + 3;
                        auto aligned32 = [&](int j) { return run4 && (reinterpret_cast<uintptr_t>(C + r[0] + cn[j]) & 31u) == 0; };
                        if constexpr (SCALED) {   // (two fragments at a time: more spill)
#pragma unroll
                            for (int j0 = 0; j0 < W; j0 += 2) {
                                double old[2][4];
#pragma unroll
                                for (int t = 0; t < 2 && j0 + t < W; ++t) {
                                    const int j = j0 + t;
                                    old[t][0] = old[t][1] = old[t][2] = old[t][3] = 0.0;
                                    if (p.beta == 0.0 || cn[j] < 0) continue;
                                    if (aligned32(j)) {
                                        ld_global_cs_v4f64(old[t], C + r[0] + cn[j]);
                                    } else {
#pragma unroll
                                        for (int q = 0; q < 4; ++q)
                                            if (r[q] >= 0) old[t][q] = __ldcs(C + r[q] + cn[j]);
                                    }
                                }
#pragma unroll
                                for (int t = 0; t < 2 && j0 + t < W; ++t)
#pragma unroll
                                    for (int q = 0; q < 4; ++q) at(u, j0 + t, q) = p.alpha * at(u, j0 + t, q) + p.beta * old[t][q];
                            }
                        }
#pragma unroll
                        for (int j = 0; j < W; ++j) {
                            if (cn[j] < 0) continue;
                            if (aligned32(j)) {
                                st_global_cs_v4f64(C + r[0] + cn[j], at(u, j, 0), at(u, j, 1), at(u, j, 2), at(u, j, 3));
                                continue;
                            }
#pragma unroll
                            for (int q = 0; q < 4; q += 2) {
                                double* d = C + r[q] + cn[j];
                                if (r[q] >= 0 && r[q + 1] == r[q] + 1 && (reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
                                    __stcs(reinterpret_cast<double2*>(d), make_double2(at(u, j, q), at(u, j, q + 1)));
                                } else {
                                    if (r[q] >= 0) __stcs(d, at(u, j, q));
                                    if (r[q + 1] >= 0) __stcs(C + r[q + 1] + cn[j], at(u, j, q + 1));
                                }
                            }
                        }
                    }
                }
            };
            if (p.store_across_slabs) store_tile([&](int u, int j, int q) -> double& { return acc[2 * q + (u & 1)][j][u >> 1]; });
            else store_tile([&](int u, int j, int q) -> double& { return acc[2 * u + (q & 1)][j][q >> 1]; });
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < W; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(tab_empty + slot));  // this warp is done with the tables
            if (prof) t_store += clock64() - t0;
        }
        if (prof) {
            long long* q = p.prof + static_cast<size_t>(blockIdx.x) * 8;
            q[0] = clock64() - t_all;
            q[1] = t_full;
            q[2] = t_main;
            q[3] = t_tab;
            q[4] = t_store;
            q[5] = 0;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && ld_shared_u32(abort_flag)) atomicMax(p.status, 1);
}

// The kernel's forms, one function per (majors, columns, k chunk, slim, scaled, pieces); `use` is called with the one that matches.
template <bool AMN, bool BMN, int NF, int BK, bool SLIM, typename Use>
cudaError_t with_epilogue(bool scaled, bool pieces, Use&& use)
{
    if (pieces) return scaled ? use(dmma_tma_kernel<AMN, BMN, NF, BK, true, SLIM, true>) : use(dmma_tma_kernel<AMN, BMN, NF, BK, false, SLIM, true>);
    return scaled ? use(dmma_tma_kernel<AMN, BMN, NF, BK, true, SLIM, false>) : use(dmma_tma_kernel<AMN, BMN, NF, BK, false, SLIM, false>);
}
template <int NF, int BK, typename Use>
cudaError_t with_majors(bool amn, bool bmn, bool slim, bool scaled, bool pieces, Use&& use)
{
    if (slim) return bmn ? cudaErrorInvalidValue : amn ? with_epilogue<true, false, NF, BK, true>(scaled, pieces, use) : with_epilogue<false, false, NF, BK, true>(scaled, pieces, use);
    if (amn) return bmn ? with_epilogue<true, true, NF, BK, false>(scaled, pieces, use) : with_epilogue<true, false, NF, BK, false>(scaled, pieces, use);
    return bmn ? with_epilogue<false, true, NF, BK, false>(scaled, pieces, use) : with_epilogue<false, false, NF, BK, false>(scaled, pieces, use);
}
template <typename Use>
cudaError_t with_kernel(const UmmaParams& p, bool scaled, bool pieces, Use&& use)
{
    const bool amn = p.a.major != 0, bmn = p.b.major != 0, slim = p.slim != 0;
    if (p.BK == 16) return p.BN == 64 ? with_majors<4, 16>(amn, bmn, slim, scaled, pieces, use) : with_majors<2, 16>(amn, bmn, slim, scaled, pieces, use);
    return p.BN == 64 ? with_majors<4, 8>(amn, bmn, slim, scaled, pieces, use) : with_majors<2, 8>(amn, bmn, slim, scaled, pieces, use);
}

// Whether every piece of `of` elements starts on a multiple of its size.
bool stores_pieces(const UmmaParams& p, int of)
{
    return p.piece >= of && reinterpret_cast<uintptr_t>(p.C64) % (8u * of) == 0 && (p.k_splits == 1 || p.split_stride % of == 0);
}

}  // namespace

// The dynamic shared-memory cap is per function and device: every run sets the same opt-in maximum, for the forms that it can launch.
cudaError_t dmma_tma_configure(const UmmaParams& p)
{
    cudaError_t e = cudaSuccess;
    for (int form = 0; form < 4 && e == cudaSuccess; ++form)
        e = with_kernel(p, form & 1, form & 2, [](auto* kernel) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxDynamicSmemBytes); });
    return e;
}

cudaError_t launch_dmma_tma(const UmmaParams& p, const void* tmapA, const void* tmapB, int smem_bytes, int num_sms, cudaStream_t stream)
{
    const long long total = p.tiles_m * p.tiles_n * p.k_splits;
    if (total <= 0 || p.k_splits < 1 || p.stages < 2 || (p.stages & 1) || (p.BN != 64 && p.BN != 32) || (p.BK != 16 && p.BK != 8)) return cudaErrorInvalidValue;
    const unsigned grid = static_cast<unsigned>(total < num_sms ? total : num_sms);
    const CUtensorMap &ta = *static_cast<const CUtensorMap*>(tmapA), &tb = *static_cast<const CUtensorMap*>(tmapB);
    UmmaParams q = p;
    // Strides of 2 modulo 4 elements: half of the columns could take 32 bytes at a time, but a test per store costs more than that spares
    // where the epilogue is most of a tile (2050 x 8000, K 24 57.3 us tested, 49.9 in halves, K 48 74.9 and 67.2; accumulating 103 and 75).
    // With more k iterations the stores fall into the other group's main loop (3002 x 3002, K 64 46.3 and 50.6, K 96 63.3 and 67.5), but
    // for the old values (79.8 and 69.1).
    q.piece = stores_pieces(p, 2) && (p.scaled || p.k_iters_per_split <= 3) ? 2 : 1;
    return with_kernel(q, p.scaled != 0, stores_pieces(p, 4), [&](auto* kernel) {
        return launch_chained(kernel, dim3(grid), dim3(kThreads64), static_cast<size_t>(smem_bytes), stream, 1, ta, tb, q);
    });
}

}  // namespace tcontb
