// dmma_tma_f64.cu -- FP64 direct contraction: TMA-staged operand tiles feeding mma.sync m8n8k4.
//
// tcgen05 has no FP64 kind, so the arithmetic is warp-level DMMA (37.0 TFLOP/s measured on B200).
// What the gather kernel (gather_contract.cu) spends on address arithmetic is done here by the copy
// engine: the planner's slab machinery, the same as for the tcgen05 kernel but with 16 doubles per
// 128-byte row, describes every operand tile as a few multi-mode TMA boxes.
//
// One block per SM.  128 x 64 tiles: three warpgroups, two of them consumer groups of 2 x 2 warps with a 64 x 32 warp tile.  128 x 32
// tiles (narrow N, and short contracted extents: narrow_tiles in planner.cpp): the same with a 64 x 16 warp tile, or four warpgroups,
// three of them consumer groups of 4 x 1 warps with a 32 x 32 warp tile (set_dmma_groups in planner.cpp has the choice and its figures).
// G consumer groups take every G-th tile of the block; setmaxnreg moves registers from the first warpgroup to them (72 and 216 a
// thread with two of them, 56 and 152 with three).
//   warps 0 .. G-1    producers, one per consumer group: lane i issues copy i of a stage (5-D tensor
//                     maps, no multicast) into the group's own ring of stages,
//                     full/empty mbarriers per stage, the ring runs across tile boundaries
//   warps G .. 3      table builders: for every tile, ahead of time, where its slabs, columns and (128 x 64) rows lie in C
//                     (mixed-radix slab arithmetic, the same as the tcgen05 epilogue),
//                     double-buffered per group behind mbarriers
//   the others        consumer groups.  They start one after the other, so that one's stores fall into the main loops of the others
//                     instead of all storing with the FP64 pipe idle.
// Fragment rows are permuted so that one 16-byte shared load of an MN-major operand feeds two
// fragments (rows 2 r and 2 r + 1 of a 16-row slab), and the MMA is issued
// transposed (B fragment as the row operand): a thread then owns four consecutive elements of C's
// stride-1 mode per fragment pair and a warp store instruction writes eight whole 128-byte lines (across slabs two elements, of the
// 64 bytes that four lanes have together: with 32-byte pieces of one lane each 9216 x 4096 x 24 took 94 us, with these 76).
// The loads of the next k step are issued between the MMAs of the current one, which go column fragment by column fragment
// (5184^3 8 225 us, row by row 8 266).
// Every wait is bounded and raises the run's status word instead of hanging.  Behind one that gave up a group stores nothing, and the
// block ends when the copies that were issued have landed.
//
// Stands where the reference runs its generated FP64 WMMA kernels
// (backends/cogent/plan/generators/kernels/kernel_compute.py:127-850) and its cublasGemmEx FP64
// call (backends/ttgt_cutt/src/ttgt_cutt.cpp:764-809).
#include <cuda.h>

#include <algorithm>
#include <type_traits>

#include "chain.cuh"
#include "kernels.hpp"
#include "tile_common.cuh"

namespace tcontb {
namespace {

constexpr int kMaxGroups = 3, kMaxStages64 = 12;
template <int FM>   // row fragments of a warp: 8 with two groups, 4 with three
constexpr int kGroups = FM == 8 ? 2 : 3;
// Three groups: every thread copies the old values of C that it will need to shared memory of its own when a tile begins.
template <int FM>
constexpr bool kOldInSmem = FM == 4;
constexpr int kOldBytes = 128 * 32 * 8;   // of one group
template <int FM>
constexpr int kThreads64 = 128 * (1 + kGroups<FM>);
constexpr int kBM = 128, kMaxBN = 64;
constexpr int kAuxBytes = 512;   // barriers, abort flag, ragged tiles
static_assert(8 * (2 * kMaxStages64 + 4 * kMaxGroups) + 4 + 8 * kMaxGroups + 48 <= kAuxBytes);
// Where a tile lies in C: an entry for each of its slabs, A's first, the offset of each column and, with two groups, of each row
// (which a thread of three groups works out from its slab: one warp has not the time to write them).
constexpr uint32_t kColumnTab = 32 * 16u, kRowTab = kColumnTab + kMaxBN * 8u;
template <int FM>
constexpr uint32_t kTabBytes = FM == 8 ? kRowTab + kBM * 8u : kColumnTab + 32 * 8u;
// (a ring of one stage would wait for its next one before it is read)
static_assert(1024 + kAuxBytes + 3 * (2 * static_cast<int>(kTabBytes<4>) + kOldBytes) + 2 * 3 * (kBM + 32) * 128 <= kMaxDynamicSmemBytes, "two stages a group beside the old values");
constexpr long long kBeyond = -(1ll << 61);          // offset of a row or column beyond C: a sum with any other offset is negative

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

__device__ __forceinline__ void st_global_cs_v2f64(double* p, double a, double b)
{
    asm volatile("st.global.cs.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(a), "d"(b) : "memory");
}

// Copies 16 or 8 bytes to shared memory, without waiting; not where `offset` is negative.
template <int BYTES>
__device__ __forceinline__ void cp_async_in(uint32_t dst, const double* C, long long offset)
{
    if constexpr (BYTES == 16)
        asm volatile("{\n .reg .pred in;\n setp.ge.s64 in, %2, 0;\n @in cp.async.cg.shared.global [%0], [%1], 16;\n}" ::"r"(dst), "l"(C + offset), "l"(offset) : "memory");
    else
        asm volatile("{\n .reg .pred in;\n setp.ge.s64 in, %2, 0;\n @in cp.async.ca.shared.global [%0], [%1], 8;\n}" ::"r"(dst), "l"(C + offset), "l"(offset) : "memory");
}

__device__ __forceinline__ void ld_global_cs(double (&o)[2], const double* p)
{
    asm volatile("ld.global.cs.v2.f64 {%0, %1}, [%2];" : "=d"(o[0]), "=d"(o[1]) : "l"(p) : "memory");
}
__device__ __forceinline__ void ld_global_cs(double (&o)[4], const double* p)
{
    asm volatile("ld.global.cs.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3]) : "l"(p) : "memory");
}

// Which k a lane feeds into step t of a stage: k = 4 t + fk, fk = lane % 4, so that an unsplit sum is one chain of FMAs in
// ascending order of k, the same bits as the gather kernel's.
__device__ __forceinline__ uint32_t step_k(uint32_t t, uint32_t fk) { return 4u * t + fk; }

// How the rows of an A tile lie in its stage, and in which rows of C they are stored.
enum RowLayout {
    ROWS_K_MAJOR,   // rows of the stage are m, BK consecutive k per row
    ROWS_MN,        // rows of the stage are k, slabs of 16 (or 8) consecutive m, which lie along C's stride-1 mode
    ROWS_ACROSS     // the same in slabs of 16, but slab s is index s of C's stride-1 mode
};

// Where a thread finds its fragments of one operand, as byte offsets from the start of the stage:
//   MN-major (rows of the stage are k, 16 consecutive m per 128-byte row, slabs of 16 m one slab apart;
//   or 8 m per 64-byte row, two slabs per 16 m):
//     one 16-byte load at  step + pair * PITCH  holds fragments 2 pair and 2 pair + 1
//   across slabs: a pair of fragments is 4 rows of each of 4 slabs, pairs 0 and 1 (2 and 3) the slabs of even and odd numbers,
//     pairs 2 and 3 the next 4 rows
//   K-major (rows of the stage are m, BK consecutive k per row: 128 bytes, or 64 with a k chunk of 8):
//     fragment i at  step + (i odd ? odd : 0) + (i / 2) * PITCH,  PITCH = 16 rows
// MN-major rows of 128 bytes are swizzled in units of 32 bytes (the unit's index XORed with row % 4): the four k and two row pairs
// that eight lanes load then lie in different banks, and a thread's offset is the same in every step.  Else the 16-byte chunk index
// inside a row is XORed with (row % 8) (128-byte rows, 128-byte swizzle) or with (row / 2) % 4 (64-byte rows, 64-byte swizzle).
// In all of them 16 m are BK * 128 bytes apart, step 1 differs from step 0
// and steps 2, 3 from 0, 1 by a thread's own constant: worked out once per block, because between two MMAs of a warp every
// instruction is time in which it feeds the pipe nothing (5184^3: 8 670 us with the offsets worked out per step and two ways
// through a stage, 8 246 now; the pipe is active in 95 % of the cycles of 2304^3).
template <int BK>
struct FragOffsets {
    static constexpr uint32_t PITCH = BK * 128u;
    uint32_t step0, step1, later, odd;
    uint32_t single;   // K-major, from row 2 fr to row 2 (fr % 4) + fr / 4: a fragment that is not one of a pair

    // `unit`: first 32-byte unit of the warp's rows in a slab (across slabs, else 0).  `slabs8`: MN-major rows of 64 bytes (slabs of 8);
    // the thread's slab, fr / 4 (across slabs: 2 (fr / 2)), is already part of thread_base
    template <RowLayout L>
    __device__ __forceinline__ void set(uint32_t thread_base, uint32_t fr, uint32_t fk, bool slabs8, uint32_t unit = 0)
    {
        auto offset = [&](uint32_t t) {
            const uint32_t k = step_k(t, fk);
            if (L != ROWS_K_MAJOR && !slabs8) return thread_base + k * 128u + (((L == ROWS_ACROSS ? unit : fr >> 1) ^ (k & 3u)) << 5) + ((fr & 1u) << 4);
            if (L != ROWS_K_MAJOR) return thread_base + k * 64u + (((fr & 3u) ^ ((k >> 1) & 3u)) << 4);
            const uint32_t kk = (k & 1u) * 8u, kc = k >> 1;
            return thread_base + kk + (BK == 8 ? (kc ^ (fr & 3u)) << 4 : (kc ^ ((2u * fr) & 7u)) << 4);   // (rows 2 fr and 2 fr + 1 share (row / 2) % 4)
        };
        step0 = offset(0);
        step1 = offset(1);
        later = offset(2) - step0;
        // K-major: the next row, its chunk index with bit 0 flipped.  Across slabs: the next unit.
        odd = L == ROWS_MN ? 0u : L == ROWS_ACROSS ? (((unit ^ fk) & 1u) ? 0u - 32u : 32u) : BK == 8 ? 64u : (fk & 2u) ? 112u : 144u;
        single = fr < 4u ? 0u : odd - 8u * (BK * 8u);
    }
};

template <RowLayout L, int N, int BK>
__device__ __forceinline__ void load_frag(double (&f)[N], int i, uint32_t q, uint32_t odd)
{
    if (L == ROWS_ACROSS) {
        if ((i & 1) == 0) ld_shared_v2f64(q + (i >= 4 ? odd : 0u) + static_cast<uint32_t>((i >> 1) & 1) * FragOffsets<BK>::PITCH, f[i], f[i + 1]);
    } else if (L == ROWS_MN) {
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

// load N fragments (8 or 4 of A, 4 or 3 of B), all at once
template <RowLayout L, int N, int BK>
__device__ __forceinline__ void load_all(double (&f)[N], uint32_t q, const FragOffsets<BK>& o)
{
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if ((N & 1) && i == N - 1) load_single<N, BK>(f, q, o.single);
        else load_frag<L, N, BK>(f, i, q, o.odd);
    }
}

// One k4 step of a warp: FM x W MMAs on the current fragments (FM row and W column fragments); the fragment loads of the next
// step are issued between them, where the FP64 tensor pipe leaves issue slots free.
// acc[i][j][h]: row 16 (i / 2) + 4 (lane % 4) + 2 h + (i % 2) of the warp (across slabs: row 4 (i / 4) + 2 h + i % 2 of slab
// 2 (lane % 4) + (i / 2) % 2), column n = column_of(j).
template <RowLayout L, bool BMN, int FM, int W, int BK>
__device__ __forceinline__ void mma_step(double (&acc)[FM][W][2], const double (&ac)[FM], const double (&bc)[W], double (&an)[FM],
                                         double (&bn)[W], uint32_t qa, const FragOffsets<BK>& oa, uint32_t qb, const FragOffsets<BK>& ob)
{
    static_assert(!BMN || W % 2 == 0, "fragments along the rows come in pairs");
#pragma unroll
    for (int i = 0; i < FM; ++i) {
#pragma unroll
        for (int t = i * W; t < (i + 1) * W; ++t) dmma_m8n8k4(acc[t % FM][t / FM], bc[t / FM], ac[t % FM]);
        load_frag<L, FM, BK>(an, i, qa, oa.odd);
        if (BMN) {
            if ((i == 1 || i == 3) && i < W) load_frag<ROWS_MN, W, BK>(bn, i - 1, qb, ob.odd);
        } else if ((W & 1) && i == W - 1) {
            load_single<W, BK>(bn, qb, ob.single);
        } else {
            if (i < W) load_frag<ROWS_K_MAJOR, W, BK>(bn, i, qb, ob.odd);
        }
    }
}
// Where a slab of a tile lies in C.
struct SlabEntry {
    long long off;   // of its first element, unless operand-level row fusion splits the position (slab_elem_offset)
    int left, pos;   // how many of its elements are inside the slab mode, position of the first one there
    __device__ __forceinline__ void store(uint32_t addr) const
    {
        asm volatile("st.shared.b64 [%0], %1;\n st.shared.v2.b32 [%0 + 8], {%2, %3};" ::"r"(addr), "l"(off), "r"(left), "r"(pos) : "memory");
    }
    __device__ __forceinline__ void load(uint32_t addr)
    {
        asm volatile("ld.shared.b64 %0, [%3];\n ld.shared.v2.b32 {%1, %2}, [%3 + 8];" : "=l"(off), "=r"(left), "=r"(pos) : "r"(addr) : "memory");
    }
    // C offset of the slab's element `in`, kBeyond where it is not in C
    __device__ __forceinline__ long long c_offset(const UmmaOperandDev& o, int in) const
    {
        const long long at = o.split_inner > 0 ? off + slab_elem_offset(o, 0, pos + in) : off + static_cast<long long>(in) * o.row_elem_cstride;
        return in < left ? at : kBeyond;
    }
};
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
// SLIM: one column of tiles, of at most three quarters of its columns (B K-major): three column fragments a warp instead of four.
template <RowLayout L, bool BMN, int FM, int BN, int BK, bool SCALED, bool SLIM, bool PIECES>
__global__ void __launch_bounds__(kThreads64<FM>, 1)
dmma_tma_kernel(const __grid_constant__ CUtensorMap tmapA, const __grid_constant__ CUtensorMap tmapB,
                const __grid_constant__ UmmaParams p)
{
    constexpr int G = kGroups<FM>, W = SLIM ? 3 : FM == 8 ? BN / 16 : 4;   // W: column fragments of a warp
    static_assert(FM == 8 ? BN == 64 || !SLIM : BN == 32);
    constexpr uint32_t kBuilders = 4 - G;   // warps of the first warpgroup that build tables
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);  // 1024-byte aligned
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int SA = p.a.slabs_per_tile, SB = p.b.slabs_per_tile;
    const uint32_t a_tile_bytes = static_cast<uint32_t>(SA * p.a.slab_bytes);
    const uint32_t stage_bytes = a_tile_bytes + static_cast<uint32_t>(SB * p.b.slab_bytes);

    uint8_t* aux = smem + static_cast<size_t>(p.stages) * stage_bytes;
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(aux);
    uint64_t* bar_empty = bar_full + kMaxStages64;
    uint64_t* tab_full = bar_empty + kMaxStages64;   // [group][buffer]
    uint64_t* tab_empty = tab_full + 2 * kMaxGroups; // [group][buffer]
    const uint32_t abort_flag = smem_u32(tab_empty + 2 * kMaxGroups);
    const uint32_t ragged = abort_flag + 4u;   // [group][buffer]: 1 + number of the last tile with rows (not SLIM: or columns) beyond C
    const uint32_t profile = smem_u32(aux + kAuxBytes - 48);   // long long [5] counters, time of the last mark
    const uint32_t tabs = smem_u32(aux + kAuxBytes);  // [group][buffer]

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(smem_u32(bar_full + s), 1);
            mbar_init(smem_u32(bar_empty + s), 4);  // one arrival per consumer warp
        }
        for (int s = 0; s < 2 * G; ++s) {
            mbar_init(smem_u32(tab_full + s), 1);
            mbar_init(smem_u32(tab_empty + s), 4);  // one arrival per consumer warp
        }
        for (uint32_t t = 0; t < 2 * G; ++t) st_shared_u32(ragged + t * 4u, 0u);
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
    const uint32_t ring = static_cast<uint32_t>(p.stages) / G;  // stages per group
    auto block_done = [] { asm volatile("bar.sync 0;" ::: "memory"); };   // the role's last act, but for what is in flight

    if (warp < 4) {
        if (G == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 72;");
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
        if (warp < G) {
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
            bool ok = true;
            const uint32_t filled = my_tiles < static_cast<uint32_t>(p.test_skip_iter) ? my_tiles : static_cast<uint32_t>(p.test_skip_iter);   // (test hook)
            for (uint32_t i = static_cast<uint32_t>(warp); ok && i < filled; i += G) {
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
                    ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar_empty + ps), phase ^ 1u, abort_flag, 200u));
                    // A stage given back behind a wait that gave up may never have been filled, or is still on its way: not filled again.  (One
                    // read for the warp, converged behind the vote, so its lanes go the same way; the word inside the vote costs 3 % where a
                    // stage is 20 copies, and 9216 x 4096 x 24 accumulating into a 6-D C 123 us instead of 121 where the warps that gave up
                    // keep their stages.)
                    ok = ok && ld_shared_u32(abort_flag) == 0u;
                    if (!ok) break;
                    if (lane == 0) mbar_arrive_expect_tx(smem_u32(bar_full + ps), stage_bytes);
                    __syncwarp();
                    if (active) {
                        int c[kMaxTmaRank];
                        k_coords(base, ks, kd0, kd1, kd2, c);
                        tma_load_5d(smem_u32(smem + static_cast<size_t>(ps) * stage_bytes + my_off), tmap,
                                    smem_u32(bar_full + ps), c[0], c[1], c[2], c[3], c[4]);
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
            if (filled < my_tiles) {   // (test hook: the group's waits end as if one of the block had run out)
                const unsigned long long t0 = global_timer();
                while (global_timer() - t0 < p.wait_limit_ns) __nanosleep(1000);
                st_shared_u32(abort_flag, 1u);
            }
            // Here, and not when the last copy is issued: a group may give up, or pass over stages that are still on their way, later on.
            // (stages before `stage` were filled in this phase, the others in the last one, or never, which a barrier takes for the last one)
            block_done();
            if (ld_shared_u32(abort_flag) && lane == 0)
                drain_copies(smem_u32(bar_full + first), static_cast<int>(ring), 0xffffffffu, phase ? (1u << stage) - 1u : ~((1u << stage) - 1u));
        } else {
            // ---------------- table builders: one warp a tile, lane s works out its slab s (at most 32) ----------------
            const bool of_a = lane < SA;
            const UmmaOperandDev& o = of_a ? p.a : p.b;
            uint32_t last_tab = 0;
            // Brings the old values of the tile with these entries into L2: the warps that compute cannot keep enough reads of C in flight to
            // hide DRAM behind the store phase.  One tile ahead: two ahead, with more of C on its way, 9216 x 4096 x 48 took 180 us, not 165.
            auto prefetch = [&](uint32_t tab) {
                const double* C = p.C64;
                // A look is 16 rows of a column (8 where a slab has no more), one line of C or parts of two; across slabs the 64 bytes of a row.
                const int run = L == ROWS_ACROSS ? 1 : p.a.slab_w < 16 ? 8 : 16, shift = L == ROWS_ACROSS || p.a.slab_w < 16 ? 4 : 3, looks = 1 << shift;
                for (int q = lane; q < looks * BN; q += 32) {
                    const uint32_t row = tab + kRowTab + static_cast<uint32_t>((q & (looks - 1)) * run) * 8u;
                    const long long c = ld_shared_s64(tab + kColumnTab + static_cast<uint32_t>(q >> shift) * 8u), first = ld_shared_s64(row) + c;
                    if (first >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + first));
                    if (L == ROWS_ACROSS) continue;
                    const long long last = ld_shared_s64(row + static_cast<uint32_t>(run - 4) * 8u) + c;
                    if (last >= 0 && (first < 0 || (((reinterpret_cast<uintptr_t>(C + first) ^ reinterpret_cast<uintptr_t>(C + last)) >> 7) != 0)))
                        asm volatile("prefetch.global.L2 [%0];" ::"l"(C + last));
                }
            };
            for (uint32_t i = static_cast<uint32_t>(warp) - G; i < my_tiles; i += kBuilders) {
                const WorkUnit w = decode_unit(blockIdx.x + i * gridDim.x, p, tiles_m, tiles_n);
                const uint32_t round = i / G, slot = (i - round * G) * 2u + (round & 1u);   // group, buffer
                if (!mbar_wait(smem_u32(tab_empty + slot), (round >> 1 & 1u) ^ 1u, abort_flag, 100u)) break;
                const uint32_t tab = tabs + slot * kTabBytes<FM>;
                SlabEntry entry;
                int d0 = 0;
                bool ok;
                entry.off = slab_c_offset(o, of_a ? w.tm * SA + lane : w.tn * SB + (lane - SA), &d0, &ok);
                entry.pos = d0 * o.slab_w;
                entry.left = ok ? o.slab_mode_ext - entry.pos : 0;
                entry.store(tab + static_cast<uint32_t>(lane) * 16u);
                auto offsets = [&](const UmmaOperandDev& of, int slab0, int count, uint32_t to) {
                    for (int c = lane; c < count; c += 32) {
                        const int from = slab0 + (c >> of.slab_shift);
                        SlabEntry e;
                        e.off = __shfl_sync(0xffffffffu, entry.off, from);
                        e.left = __shfl_sync(0xffffffffu, entry.left, from);
                        e.pos = __shfl_sync(0xffffffffu, entry.pos, from);
                        st_shared_s64(to + static_cast<uint32_t>(c) * 8u, e.c_offset(of, c & (of.slab_w - 1)));
                    }
                };
                offsets(p.b, SA, BN, tab + kColumnTab);
                if (FM == 8) offsets(p.a, 0, kBM, tab + kRowTab);
                if (SCALED && PIECES && !kOldInSmem<FM> && lane < (SLIM ? SA : SA + SB) && entry.left < o.slab_w) st_shared_u32(ragged + slot * 4u, i + 1u);
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(tab_full + slot));
                // The old values of the tile that the group begins now (behind the first one: its slot is what the wait above was for)
                if (SCALED && !kOldInSmem<FM> && p.beta != 0.0 && round != 1) prefetch(round == 0 ? tab : tabs + (slot ^ 1u) * kTabBytes<FM>);
                last_tab = tab;
            }
            if (SCALED && !kOldInSmem<FM> && p.beta != 0.0 && last_tab != 0) prefetch(last_tab);
            block_done();
        }
    } else {
        if (G == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");
        else asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
        // ---------------- consumers: groups of 2 x 2 warps (64 x 32 or 64 x 16 warp tiles) or 4 x 1 (32 x 32) ----------------
        constexpr int WM = 16 / FM;   // warps along the rows
        const int cw = warp & 3, grp = (warp >> 2) - 1, wm = cw % WM, wn = cw / WM;
        const uint32_t fr = static_cast<uint32_t>(lane >> 2), fk = static_cast<uint32_t>(lane & 3);
        const uint32_t first = static_cast<uint32_t>(grp) * ring;
        const bool a8 = L == ROWS_MN && p.a.slab_w == 8, b8 = BMN && p.b.slab_w == 8;  // 16 m = two slabs of 8
        constexpr uint32_t PITCH = FragOffsets<BK>::PITCH;
        const uint32_t col0 = static_cast<uint32_t>(wn * W * 8);   // the warp's columns
        FragOffsets<BK> fa, fb;
        fa.template set<L>(L == ROWS_ACROSS ? (fr >> 1) * 2u * PITCH
                           : L == ROWS_MN ? static_cast<uint32_t>(wm * (FM / 2)) * PITCH + (a8 ? (fr >> 2) * static_cast<uint32_t>(p.a.slab_bytes) : 0u)
                                          : (static_cast<uint32_t>(wm * FM * 8) + 2u * fr) * (BK * 8u), fr, fk, a8, static_cast<uint32_t>(wm * (FM / 4)));
        fb.template set<BMN ? ROWS_MN : ROWS_K_MAJOR>(a_tile_bytes + (BMN ? static_cast<uint32_t>(wn * (W / 2)) * PITCH + (b8 ? (fr >> 2) * static_cast<uint32_t>(p.b.slab_bytes) : 0u)
                                                                          : (col0 + 2u * fr) * (BK * 8u)), fr, fk, b8);
        double acc[FM][W][2];
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
            for (int j = 0; j < W; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

        // Old values: where a thread copies unit s of 16 bytes (8 where elements go one by one) is old_to + s * 2048 (1024), where it finds
        // its own ones is said by old_from.
        const bool staged = kOldInSmem<FM> && p.old_staged != 0;
        const uint32_t old_unit = PIECES || p.piece >= 2 ? 16u : 8u, old_base = tabs + 2u * G * kTabBytes<FM> + static_cast<uint32_t>(grp) * kOldBytes;
        const uint32_t old_to = old_base + (threadIdx.x & 127u) * old_unit;
        const uint32_t old_from = L == ROWS_ACROSS ? old_to
                                  : old_base + (threadIdx.x & 124u) * old_unit + (old_unit == 16u ? (fk >> 1) * (W * 2048u) + (fk & 1u) * 32u : fk * (W * 1024u));
        // A thread's elements of a tile.  Neighbouring ones for each of its row pieces and W column fragments:
        //   rows along C    : rows 16 u + 4 fk + q of the warp, q < 4, element q in acc[2 u + (q & 1)][j][q >> 1]
        //   rows across slabs: row 4 (u / 4) + u % 4 of slabs 2 fk + q, q < 2, element q in acc[4 (u / 4) + 2 q + (u & 1)][j][(u >> 1) & 1];
        //                      four lanes hold the same row of eight slabs, 64 bytes of C
        constexpr bool ACROSS = L == ROWS_ACROSS;
        constexpr int PIECE = ACROSS ? 2 : 4, ROWS = FM * 2 / PIECE;
        auto at = [&](int u, int j, int q) -> double& { return ACROSS ? acc[4 * (u >> 2) + 2 * q + (u & 1)][j][(u >> 1) & 1] : acc[2 * u + (q & 1)][j][q >> 1]; };
        const uint32_t my_row = ACROSS ? fk * 32u + static_cast<uint32_t>(wm * FM) : static_cast<uint32_t>(wm * FM * 8) + 4u * fk;
        uint32_t tab = 0;
        SlabEntry lead;   // across slabs: the thread's even slab
        auto row_at = [&](uint32_t row) {   // C offset of a row of the tile
            if (FM == 8) return ld_shared_s64(tab + kRowTab + row * 8u);
            SlabEntry e;
            e.load(tab + (row >> p.a.slab_shift) * 16u);
            return e.c_offset(p.a, static_cast<int>(row) & (p.a.slab_w - 1));
        };
        auto row_of = [&](uint32_t u, uint32_t q) {   // of element q of a piece
            if (!ACROSS) return row_at(my_row + 16u * u + q);
            if (FM == 8) return row_at(my_row + u + 16u * q);
            return lead.c_offset(p.a, wm * FM + static_cast<int>(u)) + q;   // (the slabs come in whole eights, next to each other in C)
        };
        auto tile_cols = [&](uint32_t slot, long long (&cn)[W]) {   // (and the rows of the tile in this slot from here on)
            tab = tabs + slot * kTabBytes<FM>;
#pragma unroll
            for (int j = 0; j < W; ++j) cn[j] = ld_shared_s64(tab + kColumnTab + (col0 + column_of<W>(j, fr)) * 8u);
            if (ACROSS && FM == 4) lead.load(tab + fk * 32u);
        };
        constexpr int kCopySteps = FM;   // ROWS * PIECE / 2
        bool sound = true;
        uint32_t stage = 0, phase = 0, round = 0;   // round: tiles of this group so far
        // Cycle counters of group 0, in shared memory: a mark adds the time since the last one to counter `to`.
        auto mark = [&](uint32_t to) {
            if (p.prof == nullptr || grp != 0 || (threadIdx.x & 127) != 0) return;
            const long long now = clock64();
            st_shared_s64(profile + to * 8u, ld_shared_s64(profile + to * 8u) + now - ld_shared_s64(profile + 40u));
            st_shared_s64(profile + 40u, now);
        };
        if (p.prof != nullptr && threadIdx.x == 128) {
            for (uint32_t c = 0; c < 5; ++c) st_shared_s64(profile + c * 8u, 0);
            st_shared_s64(profile + 40u, clock64());
        }

        for (uint32_t i = static_cast<uint32_t>(grp); i < my_tiles; i += G) {
            // group g starts g / G of a main loop behind group 0 (named barrier g: 128 waiting, 128 arriving)
            if (i == static_cast<uint32_t>(grp) && grp > 0) asm volatile("bar.sync %0, 256;" ::"r"(grp) : "memory");

            const WorkUnit w = decode_unit(blockIdx.x + i * gridDim.x, p, tiles_m, tiles_n);
            double* __restrict__ C = p.C64 + static_cast<long long>(w.split) * p.split_stride;
            bool tile_ok = sound;   // (behind a wait that gave up the parities of later ones mean nothing)
            const uint32_t slot = static_cast<uint32_t>(grp) * 2u + (round & 1u);
            // Old values of C: a step copies what the four lanes of a quad need of one piece of their rows (two elements a lane, W columns),
            // neighbouring lanes neighbouring bytes at both ends (with the bytes a lane needs lying together instead, each 16 were a request
            // of their own: 9216 x 4096 x 24, rows along C, 163 us).
            int copied = SCALED && staged ? 0 : kCopySteps;   // (staged: beta is not zero)
            long long cc[W];
            if (SCALED && staged) {
                tile_ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(tab_full + slot), (round >> 1) & 1u, abort_flag)) && tile_ok;
                if (!tile_ok) copied = kCopySteps;
                tile_cols(slot, cc);
            }
            auto copy_old = [&](uint32_t step) {
                // rows along C: step = 2 u + t, elements 8 t to 8 t + 7 of the quad's 16 rows; across slabs: step = row of the quad's eight slabs
                const uint32_t row = my_row + 16u * (step >> 1) + 8u * (step & 1u) - 4u * fk;
                if (PIECES || p.piece >= 2) {
                    const long long cm = ACROSS ? row_of(step, 0) : row_at(row + 2u * fk);
#pragma unroll
                    for (int j = 0; j < W; ++j) cp_async_in<16>(old_to + (step * W + static_cast<uint32_t>(j)) * 2048u, C, cm + cc[j]);
                } else {
#pragma unroll
                    for (uint32_t h = 0; h < 2; ++h) {
                        const long long cm = ACROSS ? row_of(step, h) : row_at(row + 4u * h + fk);
#pragma unroll
                        for (int j = 0; j < W; ++j) cp_async_in<8>(old_to + ((2u * step + h) * W + static_cast<uint32_t>(j)) * 1024u, C, cm + cc[j]);
                    }
                }
            };
            // One path through a stage, with few instructions that are not between two MMAs: the last step of a stage fetches the
            // first fragments of the next one, whose barrier is looked at a step earlier (behind the last stage of a tile the
            // fragments are fetched from that stage again and not used).  A wait that gave up leaves wrong fragments, and
            // tile_ok says so.
            double fa0[FM], fb0[W], fa1[FM], fb1[W];
            uint32_t chunk = static_cast<uint32_t>(w.it0 ? w.it0 % p.k_digit_ext[0] : 0);   // chunk of the chunked mode
            {
                const bool landed = mbar_wait(smem_u32(bar_full + first + stage), phase, abort_flag);
                tile_ok = __all_sync(0xffffffffu, landed) && tile_ok;
                mark(1);
            }
            uint32_t sb = smem_u32(smem) + (first + stage) * stage_bytes;
            load_all<L, FM, BK>(fa0, sb + fa.step0, fa);
            load_all<BMN ? ROWS_MN : ROWS_K_MAJOR, W, BK>(fb0, sb + fb.step0, fb);
            // (measured: k chunks of 8 once a turn 671 us for 5184^2 x 384, twice 651; chunks of 16 506 and 521 for 3233 x 2773 x 851)
            constexpr int kUnroll = BK == 8 ? 2 : 1;
#pragma unroll kUnroll
            for (int left = w.n_it; left > 0; --left) {
                if (i == 0) {
#pragma unroll
                    for (int g = 1; g < G; ++g)
                        if (my_tiles > static_cast<uint32_t>(g) && left == w.n_it - (w.n_it > 64 || (my_tiles % G == 0 && w.n_it > 4 * G) ? 4 * g : w.n_it * g / G)) asm volatile("bar.arrive %0, 256;" ::"r"(g) : "memory");
                }
                const uint32_t bar_done = smem_u32(bar_empty + first + stage);
                if (++stage == ring) {
                    stage = 0;
                    phase ^= 1u;
                }
                // (A step behind each of the first iterations, two where there are only few short ones, the rest behind the last: all at once
                // they are in the way of the fragment loads.  9216 x 4096 by K: 64 219 us at once, 196; 24 121 one at a time, 114.)
                if (SCALED && kOldInSmem<FM>)
                    for (; copied < kCopySteps && (copied < (w.n_it - left + 1) * (BK == 8 && w.n_it <= 4 ? 2 : 1) || left == 1); ++copied) copy_old(static_cast<uint32_t>(copied));
                uint32_t later_a = 0, later_b = 0;
                // (the last chunk of a mode that is 1 to 8 past a multiple of 16 holds zeros in its second half: 5184^3 with
                // contracted modes of 72 computed a tenth of its k for nothing, 9 520 us)
                if (BK == 16 && chunk < static_cast<uint32_t>(p.full_chunks)) {
                    mma_step<L, BMN, FM, W, BK>(acc, fa0, fb0, fa1, fb1, sb + fa.step1, fa, sb + fb.step1, fb);
                    later_a = fa.later;
                    later_b = fb.later;
                    mma_step<L, BMN, FM, W, BK>(acc, fa1, fb1, fa0, fb0, sb + fa.step0 + later_a, fa, sb + fb.step0 + later_b, fb);
                }
                const uint32_t bar_next = smem_u32(bar_full + first + stage);
                const bool more = left > 1, landed = !more || mbar_test_wait(bar_next, phase);
                mma_step<L, BMN, FM, W, BK>(acc, fa0, fb0, fa1, fb1, sb + fa.step1 + later_a, fa, sb + fb.step1 + later_b, fb);
                if (!__all_sync(0xffffffffu, landed)) tile_ok = __all_sync(0xffffffffu, mbar_wait(bar_next, phase, abort_flag)) && tile_ok;
                if (more) sb = smem_u32(smem) + (first + stage) * stage_bytes;
                mma_step<L, BMN, FM, W, BK>(acc, fa1, fb1, fa0, fb0, sb + fa.step0, fa, sb + fb.step0, fb);
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_done);  // this warp is done reading the stage
                if (++chunk == static_cast<uint32_t>(p.k_digit_ext[0])) chunk = 0;
            }
            mark(2);

            // the tile's offset tables were built while it was being computed
            tile_ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(tab_full + slot), (round >> 1) & 1u, abort_flag)) && tile_ok;
            if (SCALED && staged) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();   // (a thread's old values were copied by the four lanes of its rows)
#pragma unroll
                for (int u = 0; u < ROWS; ++u)
#pragma unroll
                    for (int q = 0; q < PIECE; q += 2)
#pragma unroll
                        for (int j = 0; j < W; ++j) {
                            double x, y;
                            if (PIECES || p.piece >= 2) {
                                ld_shared_v2f64(old_from + static_cast<uint32_t>(u * PIECE / 2 * W + j) * 2048u + static_cast<uint32_t>(q) * 8u, x, y);
                            } else {
                                const uint32_t at_u = old_from + static_cast<uint32_t>(u * PIECE * W + j) * 1024u;
                                x = ld_shared_f64(at_u + static_cast<uint32_t>(q) * (ACROSS ? W * 1024u : 8u));
                                y = ld_shared_f64(at_u + static_cast<uint32_t>(q + 1) * (ACROSS ? W * 1024u : 8u));
                            }
                            at(u, j, q) = p.alpha * at(u, j, q) + p.beta * x;
                            at(u, j, q + 1) = p.alpha * at(u, j, q + 1) + p.beta * y;
                        }
            }
            mark(3);

            long long cn[W];
            tile_cols(slot, cn);
            const bool whole = SCALED && !kOldInSmem<FM> && PIECES && ld_shared_u32(ragged + slot * 4u) != i + 1u;
            // Straight-line: a warp alone on its scheduler takes 5 to 20 cycles for every instruction and branch between two stores (with
            // alignment and bounds tested per store 4 200 cycles a tile, whatever the pieces' layout; 1 700 here).  Pieces beyond C are
            // left out by predicate (tested per store, 300 000 x 40 x 24 took 50.1 us and accumulating 124, here 40.4 and 65.6); a whole
            // tile's old values are not (9216 x 4096 x 24 accumulating: 176 us by predicate, 167 without).
            auto store_pieces = [&](auto all) {
                constexpr bool ALL = decltype(all)::value;
                constexpr int UB = FM == 4 ? ROWS : ACROSS ? 2 : 1;   // row pieces whose old values are asked for together
#pragma unroll
                for (int u0 = 0; u0 < ROWS; u0 += UB) {
                    long long cm[UB];
#pragma unroll
                    for (int v = 0; v < UB; ++v) cm[v] = row_of(u0 + v, 0);
                    if (SCALED && !staged) {   // the old values of all column fragments are asked for before the first is used
                        double old[UB][W][PIECE];
#pragma unroll
                        for (int v = 0; v < UB; ++v)
#pragma unroll
                            for (int j = 0; j < W; ++j) {
                                if (p.beta != 0.0 && (ALL ? !SLIM || cn[j] >= 0 : cm[v] + cn[j] >= 0)) ld_global_cs(old[v][j], C + cm[v] + cn[j]);
                                else
#pragma unroll
                                    for (int q = 0; q < PIECE; ++q) old[v][j][q] = 0.0;
                            }
#pragma unroll
                        for (int v = 0; v < UB; ++v)
#pragma unroll
                            for (int j = 0; j < W; ++j)
#pragma unroll
                                for (int q = 0; q < PIECE; ++q) at(u0 + v, j, q) = p.alpha * at(u0 + v, j, q) + p.beta * old[v][j][q];
                    }
#pragma unroll
                    for (int v = 0; v < UB; ++v)
#pragma unroll
                        for (int j = 0; j < W; ++j) {
                            const double piece[4] = {at(u0 + v, j, 0), at(u0 + v, j, 1), ACROSS ? 0.0 : at(u0 + v, j, 2 % PIECE), ACROSS ? 0.0 : at(u0 + v, j, 3 % PIECE)};
                            if (ALL && SLIM && cn[j] < 0) continue;
                            if (ACROSS) ALL ? st_global_cs_v2f64(C + cm[v] + cn[j], piece[0], piece[1]) : st_global_cs_v2f64_in(C, cm[v] + cn[j], piece[0], piece[1]);
                            else ALL ? st_global_cs_v4f64(C + cm[v] + cn[j], piece[0], piece[1], piece[2], piece[3])
                                     : st_global_cs_v4f64_in(C, cm[v] + cn[j], piece[0], piece[1], piece[2], piece[3]);
                        }
                }
            };
            if (!tile_ok) {
            } else if constexpr (PIECES) {
                if (!kOldInSmem<FM> && SCALED && whole) store_pieces(std::bool_constant<SCALED && !kOldInSmem<FM>>());
                else store_pieces(std::false_type());
            } else if (ACROSS || p.piece != 2) {
                // rows along C: 32 bytes where they can be, 16 where two elements are neighbours, else one by one; across slabs one by one
#pragma unroll
                for (int u = 0; u < ROWS; ++u) {
                    long long r[PIECE];
#pragma unroll
                    for (int q = 0; q < PIECE; ++q) r[q] = row_of(u, q);
                    const bool run4 = !ACROSS && r[0] >= 0 && r[1] == r[0] + 1 && r[2 % PIECE] == r[0] + 2 && r[3 % PIECE] == r[0] + 3;
                    auto aligned32 = [&](int j) { return run4 && (reinterpret_cast<uintptr_t>(C + r[0] + cn[j]) & 31u) == 0; };
                    if (SCALED && !staged) {   // (two fragments at a time: more spill)
#pragma unroll
                        for (int j0 = 0; j0 < W; j0 += 2) {
                            double old[2][PIECE];
#pragma unroll
                            for (int t = 0; t < 2 && j0 + t < W; ++t) {
                                const int j = j0 + t;
#pragma unroll
                                for (int q = 0; q < PIECE; ++q) old[t][q] = 0.0;
                                if (p.beta == 0.0 || cn[j] < 0) continue;
                                if (aligned32(j)) {
                                    ld_global_cs(old[t], C + r[0] + cn[j]);
                                } else {
#pragma unroll
                                    for (int q = 0; q < PIECE; ++q)
                                        if (r[q] >= 0) old[t][q] = __ldcs(C + r[q] + cn[j]);
                                }
                            }
#pragma unroll
                            for (int t = 0; t < 2 && j0 + t < W; ++t)
#pragma unroll
                                for (int q = 0; q < PIECE; ++q) at(u, j0 + t, q) = p.alpha * at(u, j0 + t, q) + p.beta * old[t][q];
                        }
                    }
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        if (cn[j] < 0) continue;
                        if (aligned32(j)) {
                            st_global_cs_v4f64(C + r[0] + cn[j], at(u, j, 0), at(u, j, 1), at(u, j, 2 % PIECE), at(u, j, 3 % PIECE));
                            continue;
                        }
#pragma unroll
                        for (int q = 0; q < PIECE; q += 2) {
                            double* d = C + r[q] + cn[j];
                            if (!ACROSS && r[q] >= 0 && r[q + 1] == r[q] + 1 && (reinterpret_cast<uintptr_t>(d) & 15u) == 0) {
                                __stcs(reinterpret_cast<double2*>(d), make_double2(at(u, j, q), at(u, j, q + 1)));
                            } else {
                                if (r[q] >= 0) __stcs(d, at(u, j, q));
                                if (r[q + 1] >= 0) __stcs(C + r[q + 1] + cn[j], at(u, j, q + 1));
                            }
                        }
                    }
                }
            } else if constexpr (!ACROSS) {
                // halves of 16 bytes, straight-line as above
#pragma unroll
                for (int u = 0; u < ROWS; ++u) {
                    const long long r[2] = {row_of(u, 0), row_of(u, 2)};
                    if (SCALED && !staged) {
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
            }
#pragma unroll
            for (int i = 0; i < FM; ++i)
#pragma unroll
                for (int j = 0; j < W; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(tab_empty + slot));  // this warp is done with the tables
            ++round;
            sound = tile_ok;
            mark(4);
        }
        if (p.prof != nullptr && threadIdx.x == 128) {
            long long* q = p.prof + static_cast<size_t>(blockIdx.x) * 8;
            q[0] = 0;
            for (uint32_t c = 1; c < 5; ++c) q[0] += q[c] = ld_shared_s64(profile + c * 8u);
            q[5] = 0;
        }
        block_done();
    }
    if (threadIdx.x == 0 && ld_shared_u32(abort_flag)) atomicMax(p.status, 1);
}

// The kernel's forms, one function per (layouts, row fragments, columns, k chunk, slim, scaled, pieces); `use` is called with the one that matches.
template <RowLayout L, bool BMN, int FM, int BN, int BK, bool SLIM, typename Use>
cudaError_t with_epilogue(bool scaled, bool pieces, Use&& use)
{
    if (pieces) return scaled ? use(dmma_tma_kernel<L, BMN, FM, BN, BK, true, SLIM, true>) : use(dmma_tma_kernel<L, BMN, FM, BN, BK, false, SLIM, true>);
    return scaled ? use(dmma_tma_kernel<L, BMN, FM, BN, BK, true, SLIM, false>) : use(dmma_tma_kernel<L, BMN, FM, BN, BK, false, SLIM, false>);
}
template <RowLayout L, int FM, int BN, int BK, typename Use>
cudaError_t with_columns(bool bmn, bool slim, bool scaled, bool pieces, Use&& use)
{
    if (slim) {
        if constexpr (FM == 8 && BN == 32) return cudaErrorInvalidValue;
        else return bmn ? cudaErrorInvalidValue : with_epilogue<L, false, FM, BN, BK, true>(scaled, pieces, use);
    }
    return bmn ? with_epilogue<L, true, FM, BN, BK, false>(scaled, pieces, use) : with_epilogue<L, false, FM, BN, BK, false>(scaled, pieces, use);
}
template <int FM, int BN, int BK, typename Use>
cudaError_t with_rows(const UmmaParams& p, bool scaled, bool pieces, Use&& use)
{
    const bool bmn = p.b.major != 0, slim = p.slim != 0;
    if (p.a.major == 0) return with_columns<ROWS_K_MAJOR, FM, BN, BK>(bmn, slim, scaled, pieces, use);
    if (!p.store_across_slabs) return with_columns<ROWS_MN, FM, BN, BK>(bmn, slim, scaled, pieces, use);
    return with_columns<ROWS_ACROSS, FM, BN, BK>(bmn, slim, scaled, pieces, use);
}
template <typename Use>
cudaError_t with_kernel(const UmmaParams& p, bool scaled, bool pieces, Use&& use)
{
    if (p.BN == 64) return p.BK == 16 ? with_rows<8, 64, 16>(p, scaled, pieces, use) : with_rows<8, 64, 8>(p, scaled, pieces, use);
    if (p.groups == 2) return p.BK == 16 ? with_rows<8, 32, 16>(p, scaled, pieces, use) : with_rows<8, 32, 8>(p, scaled, pieces, use);
    return p.BK == 16 ? with_rows<4, 32, 16>(p, scaled, pieces, use) : with_rows<4, 32, 8>(p, scaled, pieces, use);
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

cudaError_t launch_dmma_tma(const UmmaParams& p, const void* tmapA, const void* tmapB, int num_sms, cudaStream_t stream)
{
    const long long total = p.tiles_m * p.tiles_n * p.k_splits;
    if (total <= 0 || p.k_splits < 1 || (p.BN != 64 && p.BN != 32) || (p.BK != 16 && p.BK != 8)) return cudaErrorInvalidValue;
    const int groups = p.groups;
    if (groups != kGroups<8> && (groups != kGroups<4> || p.BN != 32)) return cudaErrorInvalidValue;
    if (p.stages < 2 * groups || p.stages > kMaxStages64) return cudaErrorInvalidValue;
    const unsigned grid = static_cast<unsigned>(total < num_sms ? total : num_sms);
    const CUtensorMap &ta = *static_cast<const CUtensorMap*>(tmapA), &tb = *static_cast<const CUtensorMap*>(tmapB);
    UmmaParams q = p;
    // test hooks: tiles of a block below this one are filled, the rest given up after the limit (in the waits themselves a limit that is
    // not a constant cost 32 x 512 x 3824 by 16 95 -> 101 us by way of other registers; a test per stage in the producer 3 % where it
    // issues 20 copies)
    q.test_skip_iter = p.test_skip_iter < 0 ? -1 : p.test_skip_iter / p.k_iters_per_split;
    if (q.wait_limit_ns == 0) q.wait_limit_ns = kWaitLimitNs;
    const int stage_bytes = p.a.slabs_per_tile * p.a.slab_bytes + p.b.slabs_per_tile * p.b.slab_bytes;
    // a ring of as many of the planned stages as the groups can share and `bytes` of other things leave room for
    auto share_stages = [&](int bytes) { q.stages = std::min(p.stages, (kMaxDynamicSmemBytes - bytes) / stage_bytes) / groups * groups; };
    int fixed = 1024 + kAuxBytes + 2 * groups * static_cast<int>(groups == 2 ? kTabBytes<8> : kTabBytes<4>);
    share_stages(fixed);
    // Room for the old values leaves two or three stages a group (four with k chunks of 8), where the tile's main loop is long enough to hide them behind anyway:
    // 172032 x 72 x 112, rows along C, 149 us staged, 137 read in the epilogue; K 48 168 and 174; across slabs K 72 73 and 86, K 128 342 and 344.
    q.old_staged = groups == 3 && p.scaled && p.beta != 0.0 && p.k_iters * p.BK <= (p.store_across_slabs ? 128 : 64) ? 1 : 0;
    if (q.old_staged) share_stages(fixed += groups * kOldBytes);
    if (q.stages < 2 * groups) return cudaErrorInvalidValue;
    const int smem = fixed + q.stages * stage_bytes;
    // Strides of 2 modulo 4 elements: half of the columns could take 32 bytes at a time, but a test per store costs more than that spares
    // where the epilogue is most of a tile (2050 x 8000, K 24 57.3 us tested, 49.9 in halves, K 48 74.9 and 67.2; accumulating 103 and 75).
    // With more k iterations the stores fall into the other group's main loop (3002 x 3002, K 64 46.3 and 50.6, K 96 63.3 and 67.5), but
    // for the old values (79.8 and 69.1).
    q.piece = stores_pieces(p, 2) && (p.scaled || p.k_iters_per_split <= 3) ? 2 : 1;
    return with_kernel(q, p.scaled != 0, stores_pieces(p, p.store_across_slabs ? 2 : 4), [&](auto* kernel) {
        return launch_chained(kernel, dim3(grid), dim3(128 * (1 + groups)), static_cast<size_t>(smem), stream, 1, ta, tb, q);
    });
}

}  // namespace tcontb
