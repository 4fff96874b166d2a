// gather_contract.cu -- direct contraction of ANY descriptor: operand tiles gathered element by element with cp.async,
// FP64 on the tensor path (mma.sync m8n8k4), Float32 on the CUDA cores with packed IEEE FMAs (fma.rn.f32x2).
//
// What TMA cannot describe runs here (ragged extents whose strides are no multiple of 16 bytes, operands that are K-major
// on different modes, views), and what is too small for the TMA-fed kernels.  Every address is a sum of per-mode terms; the
// rows, columns and contracted indices of a tile are split into their modes inside the kernel (multiply-shift division), so
// nothing has to be built or read from global memory before the first gather.
//
// Blocks are persistent where there are more tiles than resident blocks: the ring of operand stages runs over the flat
// sequence of (tile, k tile) steps, so that the gathers of the next tiles are in flight while this one is multiplied and
// stored.  Few tiles and a long contracted extent: a cluster of S CTAs shares one output tile, each CTA contracts a range
// of k, and the partial tiles are added through distributed shared memory in ascending rank order (one launch,
// deterministic).
//
// What bounds it: large problems the FP64 pipe or the FP32 pipe (5 184^3: FP64 30.0 TFLOP/s; 5 329^3 Float32 49.7, of the 66 that FMAs on
// registers alone reach, 40 in warps of 128 x 16; 3233 x 2773 x 851 FP64 1 055 -> 640 us), small ones the time a lone block needs per k tile (0.5 us
// in the 32 x 32 Float32 tile, 1.1 with a fourth of its warps; 0.7 / 1.5 us in the FP64 tiles of 32 / 64) and the way from
// launch to launch (693 x 47 x 41 Float32 8.2 -> 4.0 us), short contracted extents the stores of C (48825 x 2627 x 7 Float32
// 332 -> 208 us, 2.5 TB/s of odd-aligned runs).
//
// Stands where the reference runs its generated kernels for descriptors of any shape
// (backends/cogent/plan/generators/kernels/kernel_body.py:1253+, kernel_compute.py:127-850).
#include <cooperative_groups.h>

#include "chain.cuh"
#include "fast_div.cuh"
#include "kernels.hpp"

namespace tcontb {
namespace {

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

template <int BYTES>
__device__ __forceinline__ void cp_async(uint32_t dst, const void* src, bool valid)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(valid ? BYTES : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Splits flat index i of a mode group into its modes; x and y are the element offsets in the group's two tensors.
// Returns false, with offset 0, where a cut mode's index lies past its extent.
__device__ __forceinline__ bool radix_offsets(const RadixGroup& g, long long i, long long* x, long long* y)
{
    long long ox = 0, oy = 0;
    uint32_t cut0 = 0, cut1 = 0;
    if (!g.wide) {
        uint32_t rem = static_cast<uint32_t>(i);
        for (int d = 0; d < g.n; ++d) {
            uint32_t q = 0;
            if (d + 1 < g.n) q = fast_div(rem, g.ext[d]);
            const uint32_t idx = rem - q * g.ext[d].d;
            ox += static_cast<long long>(idx) * g.sx[d];
            oy += static_cast<long long>(idx) * g.sy[d];
            if (d == 0) cut0 = idx;
            if (d == 1) cut1 = idx;
            if (d == 2) cut0 += idx * g.t0;
            if (d == 3) cut1 += idx * g.t1;
            rem = q;
        }
    } else {
        for (int d = 0; d < g.n; ++d) {
            const long long q = i / g.ext[d].d;
            const long long idx = i - q * g.ext[d].d;
            ox += idx * g.sx[d];
            oy += idx * g.sy[d];
            if (d == 0) cut0 = static_cast<uint32_t>(idx);
            if (d == 1) cut1 = static_cast<uint32_t>(idx);
            if (d == 2) cut0 += static_cast<uint32_t>(idx) * g.t0;
            if (d == 3) cut1 += static_cast<uint32_t>(idx) * g.t1;
            i = q;
        }
    }
    const bool inside = g.lim0 == 0 || (cut0 < g.lim0 && cut1 < g.lim1);
    *x = inside ? ox : 0;
    *y = inside ? oy : 0;
    return inside;
}

__device__ __forceinline__ void dmma_m8n8k4(double (&c)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(c[0]), "+d"(c[1])
                 : "d"(a), "d"(b));
}
// Two IEEE single-precision FMAs in one instruction: half the issue slots of scalar FFMAs at the same pipe rate.
__device__ __forceinline__ void ffma2(unsigned long long& c, unsigned long long a, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long dup2(float a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float lo2(unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v)); }
__device__ __forceinline__ float hi2(unsigned long long v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }

// Block tile BM x BN, KG groups of WM x WN warps; a warp owns (BM / WM) x (BN / WN), a group one KG-th of every k tile (the
// small tile is bound by the time one block needs per k tile: more warps on it shorten that, and the sums of the groups are
// added up once at the end).
//   double: a warp tile is a grid of 8 x 8 DMMA fragments.
//   float : a warp tile is (32 TM) x 16, lane l holding rows l, l + 32, ... and all 16 columns as 8 packed pairs, so that A
//           fragments are conflict-free 4-byte loads, B fragments broadcast 16-byte loads, and stores whole 128-byte lines.
template <typename T, int BM_, int BN_, int WM_, int WN_, int KG_, bool FLAT_, int STAGES_, int MINB_>
struct GatherCfg {
    using type = T;
    static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, KG = KG_, BK = 16, STAGES = STAGES_, THREADS = WM * WN * KG * 32, MINB = MINB_;
    static constexpr bool F64 = sizeof(T) == 8;
    // FLAT: persistent blocks, the ring runs across tiles (short contracted ranges).  Else one tile per block: without the
    // bookkeeping of tiles the registers hold a longer main loop (Float32 128 x 128 on a 5184^3 problem: 38.5 against 30.6 TFLOP/s).
    static constexpr bool FLAT = FLAT_;
    // Row pitches.  double: 4 past a multiple of 16, so that a fragment load (k = lane % 4, row = lane / 4) touches 16
    // different 8-byte banks per half warp.  float: A 2 past a multiple of 32 (K-major gathers without conflicts), B a
    // multiple of 4 (16-byte fragment loads).
    // GRID: a Float32 warp tile of 32 x 32 or 64 x 64, lanes as 8 x 4, lane (m, n) holding rows 4 m .. 4 m + 3 (+ 32) and columns
    // 4 n .. 4 n + 3 (+ 16, 32, 48): all fragments are 16-byte loads, 3 of them to 16 packed FMAs instead of 6, or 6 to 64 instead of 8 to
    // 32, and the results leave through shared memory, whole columns of the tile.  45 drawn contractions on 64 x 64 tiles are 1.11 times
    // as fast (675 x 825 x 990 94 -> 75 us); on 128 x 32 tiles, whose columns are often few, as many are slower as faster (9177 x 18 x
    // 301 27 -> 35, 3060 x 23 x 313 12.5 -> 15.4, others 10 % faster), so those keep lines of rows.
    // WIDE: 64 x 64.  Two warps per scheduler, so the gathers of a later k tile are spread over the FMAs of this one (5329^3 40.5 -> 45.2
    // TFLOP/s without and 49.8 with that; without any gathers the FMAs reach 66), and sixteen columns leave at a time (3001 x 2001 x 601 in
    // clusters of 2 277 -> 205 us).
    static constexpr bool WIDE = !F64 && BN / WN == 64, GRID = !F64 && BN / WN >= 32;
    static constexpr int LDA = F64 || GRID ? BM + 4 : BM + 2, LDB = BN + 4;
    static constexpr int A_ELEMS = BK * LDA, STAGE_ELEMS = (BK * (LDA + LDB) + 3) / 4 * 4;
    // Tiles whose row tables are live at once: the one being multiplied, up to STAGES behind it in the ring, one being built
    static constexpr int TABLES = FLAT ? STAGES + 2 : 1, TABLE_ENTRIES = 2 * (BM + BN);
    static constexpr int KTAB = F64 && BM * BN > 1024 ? 128 : 256;   // contracted ranges up to this keep their k offsets in shared memory for good
    static constexpr int SMEM = STAGES * STAGE_ELEMS * static_cast<int>(sizeof(T)) + (TABLES * TABLE_ENTRIES + 2 * KTAB) * 8;
    static_assert(STAGES * BK <= KTAB, "k ring fits");
    static_assert(STAGES * STAGE_ELEMS >= KG * BM * BN, "the partial tiles fit the operand ring");
    static_assert(!FLAT || KG == 1, "the ring is never free for partial tiles");
    static_assert((BK * LDA) % 4 == 0, "B tile alignment");
    static_assert(THREADS % BK == 0 && (THREADS % BM == 0) && (THREADS % BN == 0), "gather mapping");
    static_assert(F64 || GRID || BN / WN == 16, "float warp tile is 16 columns wide");
    static_assert(!GRID || (BM / WM % 32 == 0 && !FLAT && KG == 1), "float warp tile of lanes 8 x 4");
    static_assert(!WIDE || (BM / WM == 64 && BM == BN && THREADS == BM && !FLAT && KG == 1), "wide warp tiles");
    static constexpr int K_HALF = KTAB / BK / 2;   // WIDE: contracted ranges past KTAB have their k offsets in a ring of two halves
    static_assert(!WIDE || (K_HALF * BK == THREADS && K_HALF >= STAGES), "one k offset per thread and half");
};

// Gathers a ROWS x BK operand tile into [k][row] shared memory.  along_k = false: a thread serves one row (`row_ptr`) for
// several k; true: one k for several rows, whose offsets come from shared memory.  k past the range is filled with zeros;
// rows past the tensor hold some other row (their results are never stored).
template <typename T, int ROWS, int LD, int BK, int THREADS>
__device__ __forceinline__ void gather_tile(uint32_t dst, const T* __restrict__ X, int row, const T* row_ptr, const long long* row_off,
                                            const long long* koff, int k_left, bool along_k, int tid)
{
    constexpr int B = sizeof(T);
    if (!along_k) {
        constexpr int STEP = THREADS / ROWS;
        int kl = tid / ROWS;
        uint32_t d = dst + static_cast<uint32_t>(kl * LD + row) * B;
#pragma unroll
        for (int i = 0; i < BK / STEP; ++i) {
            cp_async<B>(d, row_ptr + koff[kl], kl < k_left);
            kl += STEP;
            d += STEP * LD * B;
        }
    } else {
        constexpr int STEP = THREADS / BK;
        const int kl = tid % BK;
        int r = tid / BK;
        const T* base = X + koff[kl];
        const bool ok = kl < k_left;
        uint32_t d = dst + static_cast<uint32_t>(kl * LD + r) * B;
#pragma unroll
        for (int i = 0; i < ROWS / STEP; ++i) {
            cp_async<B>(d, base + row_off[r], ok);
            r += STEP;
            d += STEP * B;
        }
    }
}

// Element i of the BK that a thread gathers of such a tile, by itself, for a block of as many threads as the tile has rows.
template <typename T, int LD, int BK, int THREADS>
struct TileGather {
    const T* from;
    uint32_t off, off_step;   // where in shared memory the offset of the next element is
    uint32_t dst, dst_step;
    int valid;
    __device__ __forceinline__ void begin(uint32_t tile, const T* X, int row, const T* row_ptr, const long long* row_off, const long long* koff,
                                          int k_left, bool along_k, int tid)
    {
        const int kl = tid % BK, r = tid / BK;
        from = along_k ? X + koff[kl] : row_ptr;
        off = smem_addr(along_k ? row_off + r : koff);
        off_step = (along_k ? THREADS / BK : 1) * 8;
        dst = tile + static_cast<uint32_t>(along_k ? kl * LD + r : row) * sizeof(T);
        dst_step = (along_k ? THREADS / BK : LD) * sizeof(T);
        valid = !along_k ? k_left : kl < k_left ? BK : 0;
    }
    __device__ __forceinline__ void element(int i)
    {
        long long at;
        asm volatile("ld.shared.b64 %0, [%1];" : "=l"(at) : "r"(off));
        cp_async<sizeof(T)>(dst, from + at, i < valid);
        off += off_step;
        dst += dst_step;
    }
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, Cfg::MINB) gather_contract_kernel(const __grid_constant__ GatherParams p)
{
    using T = typename Cfg::type;
    constexpr int BM = Cfg::BM, BN = Cfg::BN, BK = Cfg::BK, STAGES = Cfg::STAGES, THREADS = Cfg::THREADS, LDA = Cfg::LDA, LDB = Cfg::LDB;
    constexpr int TILE_M = BM / Cfg::WM, TILE_N = BN / Cfg::WN;
    constexpr bool F64 = Cfg::F64;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* ring = reinterpret_cast<T*>(smem_raw);
    // per tile: A offsets [BM], B offsets [BN], C offsets of rows [BM] and columns [BN] (-1 past the tensor)
    long long* tables = reinterpret_cast<long long*>(smem_raw + static_cast<size_t>(STAGES) * Cfg::STAGE_ELEMS * sizeof(T));
    long long* k_a = tables + Cfg::TABLES * Cfg::TABLE_ENTRIES;   // A and B offsets of each k: the whole range, or a ring of k tiles
    long long* k_b = k_a + Cfg::KTAB;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t S = static_cast<uint32_t>(p.cluster);
    const uint32_t rank = S > 1 ? blockIdx.x % S : 0u, first_tile = S > 1 ? blockIdx.x / S : blockIdx.x;
    const uint32_t tile_step = S > 1 ? gridDim.x / S : gridDim.x, total_tiles = p.tiles_m * p.tiles_n;
    const uint32_t my_tiles = Cfg::FLAT ? (total_tiles - first_tile + tile_step - 1) / tile_step : 1u;   // (no block is without a tile)
    const long long k_begin = static_cast<long long>(rank) * p.k_per_cta;
    const long long k_end = k_begin + p.k_per_cta < p.K ? k_begin + p.k_per_cta : p.K;
    const int nk = k_end > k_begin ? static_cast<int>((k_end - k_begin + BK - 1) / BK) : 0;
    const bool k_whole = static_cast<long long>(nk) * BK <= Cfg::KTAB;

    // Row, column and C offsets of the block's tile number t, into its table slot.
    auto build = [&](uint32_t t) {
        const uint32_t tile = first_tile + t * tile_step;
        // groups of raster_group tile rows are swept column by column, so that blocks that run together share operand panels in L2
        const uint32_t g = static_cast<uint32_t>(p.raster_group), per_group = g * p.tiles_n;
        const uint32_t group = tile / per_group, first = group * g;
        const uint32_t rows = p.tiles_m - first < g ? p.tiles_m - first : g;
        const uint32_t local = tile - group * per_group;
        const uint32_t tn = local / rows, tm = first + local - tn * rows;
        long long* tab = tables + (t % Cfg::TABLES) * Cfg::TABLE_ENTRIES;
        for (int r = tid; r < BM + BN; r += THREADS) {
            const bool is_m = r < BM;
            const long long i = is_m ? static_cast<long long>(tm) * BM + r : static_cast<long long>(tn) * BN + (r - BM);
            const long long total = is_m ? p.M : p.N;
            long long x, y;
            const bool inside = radix_offsets(is_m ? p.m : p.n, i < total ? i : total - 1, &x, &y);
            tab[r] = x;
            tab[BM + BN + r] = i < total && inside ? y : -1;
        }
    };
    auto fill_k = [&](int kt, int at, int kl) {
        const long long k = k_begin + static_cast<long long>(kt) * BK + kl;
        long long x, y;
        radix_offsets(p.k, k < k_end ? k : 0, &x, &y);
        k_a[at + kl] = x;
        k_b[at + kl] = y;
    };

    // The step whose gathers are issued next (tile number, k tile, ring slot) and the tile that step + 1 starts, if it does.
    uint32_t is_tile = 0;
    int is_kt = 0, is_slot = 0;
    const T* __restrict__ A = static_cast<const T*>(p.A);
    const T* __restrict__ B = static_cast<const T*>(p.B);
    const bool a_k = p.a_along_k != 0, b_k = p.b_along_k != 0;
    // Rows cut in two modes lie in the tile as t0 indices of C's stride-1 mode times t1 of A's; the threads that gather run
    // along A's.
    int a_r = tid % BM;
    if (p.m.lim0) a_r = (a_r % static_cast<int>(p.m.t1)) * static_cast<int>(p.m.t0) + a_r / static_cast<int>(p.m.t1);
    const int b_r = tid % BN;
    const T *a_row = A, *b_row = B;
    const uint32_t ring_addr = smem_addr(ring);
    // WIDE: starts the gathers of the next k tile.  Past the last one nothing is read, its slots are filled with zeros.
    TileGather<T, LDA, BK, THREADS> next_a;
    TileGather<T, LDB, BK, THREADS> next_b;
    auto begin_issue = [&]() {
        const long long left = k_end - k_begin - static_cast<long long>(is_kt) * BK;
        const int k_left = left < 0 ? 0 : left < BK ? static_cast<int>(left) : BK, at = is_kt % (2 * Cfg::K_HALF) * BK;
        const uint32_t st = ring_addr + static_cast<uint32_t>(is_slot * Cfg::STAGE_ELEMS) * sizeof(T);
        next_a.begin(st, A, a_r, a_row, tables, k_a + at, k_left, a_k, tid);
        next_b.begin(st + Cfg::A_ELEMS * sizeof(T), B, b_r, b_row, tables + BM, k_b + at, k_left, b_k, tid);
        ++is_kt;
        if (++is_slot == STAGES) is_slot = 0;
    };
    auto issue = [&]() {
        if constexpr (Cfg::WIDE) {
            begin_issue();
#pragma unroll
            for (int i = 0; i < BK; ++i) {
                next_a.element(i);
                next_b.element(i);
            }
            cp_async_commit();
            return;
        }
        if (is_tile < my_tiles) {
            const long long* tab = tables + (is_tile % Cfg::TABLES) * Cfg::TABLE_ENTRIES;
            if (is_kt == 0) {
                a_row = A + tab[a_r];
                b_row = B + tab[BM + b_r];
            }
            const uint32_t st = ring_addr + static_cast<uint32_t>(is_slot * Cfg::STAGE_ELEMS) * sizeof(T);
            const long long left = k_end - k_begin - static_cast<long long>(is_kt) * BK;
            const int k_left = left < BK ? static_cast<int>(left) : BK, at = (k_whole ? is_kt : is_slot) * BK;
            gather_tile<T, BM, LDA, BK, THREADS>(st, A, a_r, a_row, tab, k_a + at, k_left, a_k, tid);
            gather_tile<T, BN, LDB, BK, THREADS>(st + Cfg::A_ELEMS * sizeof(T), B, b_r, b_row, tab + BM, k_b + at, k_left, b_k, tid);
            if (++is_kt == nk) {
                is_kt = 0;
                ++is_tile;
            }
            if (++is_slot == STAGES) is_slot = 0;
        }
        cp_async_commit();   // one group per step, empty past the end, so that the wait below counts uniformly
    };

    const int kg = warp / (Cfg::WM * Cfg::WN), wm = warp % Cfg::WM, wn = warp / Cfg::WM % Cfg::WN;
    constexpr int FM = F64 || Cfg::GRID ? TILE_M / 8 : TILE_M / 32, FN = F64 || Cfg::GRID ? TILE_N / 8 : TILE_N / 2;
    using Acc = typename std::conditional<F64, double[2], unsigned long long[1]>::type;
    Acc acc[FM][FN];
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN; ++j) {
            acc[i][j][0] = 0;
            if constexpr (F64) acc[i][j][1] = 0;
        }
    const int fr = lane >> 2, fk = lane & 3;
    T* __restrict__ C = static_cast<T*>(p.C);
    const T alpha = static_cast<T>(p.alpha), beta = static_cast<T>(p.beta);
    const bool scaled = p.scaled != 0, add = p.scaled != 0 && beta != T(0);

    // tables of the tiles that steps 0 .. STAGES - 1 belong to
    if (Cfg::FLAT && nk > 0) {
        for (uint32_t t = 0; t < my_tiles && t * static_cast<uint32_t>(nk) < STAGES; ++t) build(t);
    } else {
        build(0);   // (also for the empty range of a cluster split, which only takes part in the sum below)
    }
    if (Cfg::WIDE) {
        for (int t = tid / BK; t < 2 * Cfg::K_HALF; t += Cfg::K_HALF) fill_k(t, t * BK, tid % BK);
    } else if (k_whole) {
        for (int i = tid; i < nk * BK; i += THREADS) fill_k(i / BK, i / BK * BK, i % BK);
    } else if (tid < STAGES * BK) {
        fill_k(tid / BK, tid / BK * BK, tid % BK);
    }
    if (!p.release_late) chain_release();
    chain_wait();   // (everything above works on the parameters alone)
    __syncthreads();

    if (Cfg::WIDE) {
        a_row = A + tables[a_r];
        b_row = B + tables[BM + b_r];
    }
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) issue();
    const uint32_t steps = nk > 0 ? my_tiles * static_cast<uint32_t>(nk) : 0u;
    uint32_t tile = 0;
    int kt = 0, slot = 0;
    for (uint32_t q = 0; q < steps; ++q) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();   // step q has landed for everyone; the slot refilled below was read at step q - 1
        if constexpr (Cfg::WIDE) {
            // the k offsets of the half ring after next, once those that lie there have all been used
            if (is_kt % Cfg::K_HALF == 0) {
                const int t = is_kt + Cfg::K_HALF + tid / BK;
                fill_k(t, t % (2 * Cfg::K_HALF) * BK, tid % BK);
            }
            begin_issue();
        } else {
            issue();
        }
        // what step q + STAGES needs, one barrier ahead of its issue
        if (Cfg::FLAT && is_kt == 0 && is_tile < my_tiles) build(is_tile);
        if (!Cfg::WIDE && !k_whole && tid < BK) fill_k(is_kt, slot * BK, tid);
        if (add && kt == 0) {
            // the tile's old values into L2 while it is multiplied: the epilogue reads them a few at a time
            const long long* c_m = tables + (tile % Cfg::TABLES) * Cfg::TABLE_ENTRIES + BM + BN;
            constexpr int LINE = 128 / static_cast<int>(sizeof(T)), LOOKS = (BM + LINE - 1) / LINE;
            for (int i = tid; i < LOOKS * BN; i += THREADS) {
                const long long m = c_m[i % LOOKS * LINE], n = c_m[BM + i / LOOKS];
                if (m >= 0 && n >= 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(C + m + n));
            }
        }
        const T* As = ring + slot * Cfg::STAGE_ELEMS;
        const T* Bs = As + Cfg::A_ELEMS;
        if constexpr (F64) {
#pragma unroll
            for (int s = 0; s < BK / 4 / Cfg::KG; ++s) {
                double a[FM], b[FN];
                const int k = 4 * (s * Cfg::KG + kg) + fk;   // (ascending: one chain of FMAs per element, in the order of k)
#pragma unroll
                for (int i = 0; i < FM; ++i) a[i] = As[k * LDA + wm * TILE_M + i * 8 + fr];
#pragma unroll
                for (int j = 0; j < FN; ++j) b[j] = Bs[k * LDB + wn * TILE_N + j * 8 + fr];
#pragma unroll
                for (int i = 0; i < FM; ++i)
#pragma unroll
                    for (int j = 0; j < FN; ++j) dmma_m8n8k4(acc[i][j], a[i], b[j]);
            }
        } else {
            const long long left = k_end - k_begin - static_cast<long long>(kt) * BK;
            auto step = [&](int k) {
                unsigned long long a[FM], b[FN];
#pragma unroll
                for (int i = 0; i < FM; ++i) a[i] = dup2(As[k * LDA + wm * TILE_M + i * 32 + lane]);
#pragma unroll
                for (int j = 0; j < FN; j += 2) {
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(Bs + k * LDB + wn * TILE_N + 2 * j);
                    b[j] = v.x;
                    b[j + 1] = v.y;
                }
#pragma unroll
                for (int i = 0; i < FM; ++i)
#pragma unroll
                    for (int j = 0; j < FN; ++j) ffma2(acc[i][j][0], a[i], b[j]);
            };
            if constexpr (Cfg::GRID) {
#pragma unroll
                for (int k = 0; k < BK; ++k) {
                    float4 a4[FM / 4];
                    ulonglong2 b4[FN / 2];
#pragma unroll
                    for (int i = 0; i < FM / 4; ++i) a4[i] = *reinterpret_cast<const float4*>(As + k * LDA + wm * TILE_M + i * 32 + (lane & 7) * 4);
#pragma unroll
                    for (int j = 0; j < FN / 2; ++j) b4[j] = *reinterpret_cast<const ulonglong2*>(Bs + k * LDB + wn * TILE_N + j * 16 + (lane >> 3) * 4);
                    if constexpr (Cfg::WIDE) {
                        next_a.element(k);
                        next_b.element(k);
                    }
#pragma unroll
                    for (int i = 0; i < FM; ++i) {
                        const float4 v = a4[i / 4];
                        const unsigned long long a = dup2(i % 4 == 0 ? v.x : i % 4 == 1 ? v.y : i % 4 == 2 ? v.z : v.w);
#pragma unroll
                        for (int j = 0; j < FN; ++j) ffma2(acc[i][j][0], a, j & 1 ? b4[j / 2].y : b4[j / 2].x);
                    }
                }
                if constexpr (Cfg::WIDE) cp_async_commit();
            } else if (!Cfg::FLAT || left >= BK) {
#pragma unroll
                for (int k = 0; k < BK / Cfg::KG; ++k) step(k * Cfg::KG + kg);
            } else {
                for (int k = 0; k < static_cast<int>(left); ++k) step(k);
            }
        }
        if (++slot == STAGES) slot = 0;
        if (++kt < nk) continue;
        kt = 0;
        if (Cfg::GRID || (!Cfg::FLAT && (Cfg::KG > 1 || S > 1))) break;
        const long long* c_m = tables + (tile % Cfg::TABLES) * Cfg::TABLE_ENTRIES + BM + BN;
        const long long* c_n = c_m + BM;
        ++tile;

        if constexpr (F64) {
            long long cm[FM];
#pragma unroll
            for (int i = 0; i < FM; ++i) cm[i] = c_m[wm * TILE_M + i * 8 + fr];
            // two columns of fragments at a time: the old values of both are asked for before the first is used
#pragma unroll
            for (int j0 = 0; j0 < FN; j0 += 2) {
                long long cn[4];
                T old[4][FM];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    cn[u] = c_n[wn * TILE_N + (j0 + (u >> 1)) * 8 + 2 * fk + (u & 1)];
#pragma unroll
                    for (int i = 0; i < FM; ++i) old[u][i] = add && cn[u] >= 0 && cm[i] >= 0 ? C[cm[i] + cn[u]] : T(0);
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
#pragma unroll
                    for (int i = 0; i < FM; ++i) {
                        T v = acc[i][j0 + (u >> 1)][u & 1];
                        if (scaled) v = alpha * v + beta * old[u][i];
                        if (cn[u] >= 0 && cm[i] >= 0) __stcs(C + cm[i] + cn[u], v);
                        acc[i][j0 + (u >> 1)][u & 1] = 0;
                    }
                }
            }
        } else {
            long long cm[FM];
#pragma unroll
            for (int i = 0; i < FM; ++i) cm[i] = c_m[wm * TILE_M + i * 32 + lane];
#pragma unroll
            for (int j = 0; j < FN; ++j) {
                const long long cn0 = c_n[wn * TILE_N + 2 * j], cn1 = c_n[wn * TILE_N + 2 * j + 1];
                T old[FM][2];
#pragma unroll
                for (int i = 0; i < FM; ++i) {
                    old[i][0] = add && cn0 >= 0 && cm[i] >= 0 ? C[cm[i] + cn0] : T(0);
                    old[i][1] = add && cn1 >= 0 && cm[i] >= 0 ? C[cm[i] + cn1] : T(0);
                }
#pragma unroll
                for (int i = 0; i < FM; ++i) {
                    T v0 = lo2(acc[i][j][0]), v1 = hi2(acc[i][j][0]);
                    if (scaled) {
                        v0 = alpha * v0 + beta * old[i][0];
                        v1 = alpha * v1 + beta * old[i][1];
                    }
                    if (cm[i] >= 0 && cn0 >= 0) __stcs(C + cm[i] + cn0, v0);
                    if (cm[i] >= 0 && cn1 >= 0) __stcs(C + cm[i] + cn1, v1);
                    acc[i][j][0] = 0;
                }
            }
        }
    }
    cp_async_wait<0>();
    if (!Cfg::GRID && (Cfg::FLAT || (Cfg::KG == 1 && S == 1))) return;
    if (p.release_late) chain_release();   // (not inside the loop: a test there costs the FP64 main loop 3 to 8 %)

    // k groups and cluster split: partial tiles into this CTA's shared memory as [group][n][m]; CTA r then adds up columns
    // r, r + S, ... over all groups and CTAs, in that order.
    __syncthreads();   // everyone is done reading the operand ring
    T* part = ring;
    T* mine = part + kg * BM * BN;
    if constexpr (F64) {
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
            for (int j = 0; j < FN; ++j)
#pragma unroll
                for (int h = 0; h < 2; ++h) mine[(wn * TILE_N + j * 8 + 2 * fk + h) * BM + wm * TILE_M + i * 8 + fr] = acc[i][j][h];
    } else if constexpr (Cfg::GRID) {
#pragma unroll
        for (int i = 0; i < FM; i += 4)
#pragma unroll
            for (int j = 0; j < FN; ++j) {
                float* to = mine + (wn * TILE_N + (j >> 1) * 16 + (lane >> 3) * 4 + (j & 1) * 2) * BM + wm * TILE_M + i * 8 + (lane & 7) * 4;
                *reinterpret_cast<float4*>(to) = make_float4(lo2(acc[i][j][0]), lo2(acc[i + 1][j][0]), lo2(acc[i + 2][j][0]), lo2(acc[i + 3][j][0]));
                *reinterpret_cast<float4*>(to + BM) = make_float4(hi2(acc[i][j][0]), hi2(acc[i + 1][j][0]), hi2(acc[i + 2][j][0]), hi2(acc[i + 3][j][0]));
            }
    } else {
#pragma unroll
        for (int i = 0; i < FM; ++i)
#pragma unroll
            for (int j = 0; j < FN; ++j) {
                mine[(wn * TILE_N + 2 * j) * BM + wm * TILE_M + i * 32 + lane] = lo2(acc[i][j][0]);
                mine[(wn * TILE_N + 2 * j + 1) * BM + wm * TILE_M + i * 32 + lane] = hi2(acc[i][j][0]);
            }
    }
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    if (S > 1) cluster.sync();
    else __syncthreads();
    const long long* c_m = tables + BM + BN;
    const long long* c_n = c_m + BM;
    constexpr int COLS_STEP = THREADS / BM;   // columns the block handles at a time (threads run along m)
    const int m = tid % BM;
    const long long cm = c_m[m];
    if (Cfg::WIDE || (BM * BN > 1024 && S <= 4)) {
        // Several columns at a time, so that neither C's old values nor other SMs' shared memory is waited for one by one.  Before / after
        // in us, 64 x 64 tiles in clusters of 2 and 4: 1061 x 679 x 245 Float32 28.9 / 23.9, 34891 x 37 x 159 FP64 accumulating
        // 63.7 / 50.1.  In larger clusters a thread has a column or two to add up: 295 x 189 x 955 FP64, clusters of 16, 17.5 / 22.1.
        constexpr int AT_ONCE = Cfg::WIDE ? 16 : 4;
        for (uint32_t n0 = rank + S * static_cast<uint32_t>(tid / BM); n0 < static_cast<uint32_t>(BN); n0 += S * COLS_STEP * AT_ONCE) {
            long long cn[AT_ONCE];
            T old[AT_ONCE], v[AT_ONCE];
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                const uint32_t nl = n0 + S * COLS_STEP * u;
                cn[u] = nl < static_cast<uint32_t>(BN) && cm >= 0 ? c_n[nl] : -1;
                old[u] = add && cn[u] >= 0 ? C[cm + cn[u]] : T(0);
                v[u] = 0;
            }
            for (uint32_t s = 0; s < S; ++s) {
                const T* from = (S > 1 ? cluster.map_shared_rank(part, s) : part) + n0 * BM + m;
#pragma unroll
                for (int u = 0; u < AT_ONCE; ++u) {
                    if (Cfg::WIDE ? n0 + S * COLS_STEP * u >= static_cast<uint32_t>(BN) : cn[u] < 0) continue;   // (wide: rows that are not stored take part)
#pragma unroll
                    for (int g = 0; g < Cfg::KG; ++g) v[u] += from[S * COLS_STEP * u * BM + g * BM * BN];
                }
            }
#pragma unroll
            for (int u = 0; u < AT_ONCE; ++u) {
                if (scaled) v[u] = alpha * v[u] + (add ? beta * old[u] : T(0));
                if (cn[u] >= 0) __stcs(C + cm + cn[u], v[u]);
            }
        }
    } else {
        for (uint32_t nl = rank + S * static_cast<uint32_t>(tid / BM); nl < static_cast<uint32_t>(BN); nl += S * COLS_STEP) {
            const long long cn = c_n[nl];
            if (cm < 0 || cn < 0) continue;
            T v = 0;
            for (uint32_t s = 0; s < S; ++s) {
                const T* from = (S > 1 ? cluster.map_shared_rank(part, s) : part) + nl * BM + m;
#pragma unroll
                for (int g = 0; g < Cfg::KG; ++g) v += from[g * BM * BN];
            }
            if (scaled) v = alpha * v + (add ? beta * C[cm + cn] : T(0));
            __stcs(C + cm + cn, v);
        }
    }
    if (S > 1) cluster.sync();   // a CTA's shared memory stays until every other has read it
}

template <class Cfg>
cudaError_t launch(GatherParams p, int num_sms, cudaStream_t stream)
{
    const long long tiles_m = (p.M + Cfg::BM - 1) / Cfg::BM, tiles_n = (p.N + Cfg::BN - 1) / Cfg::BN;
    if (p.cluster < 1 || p.cluster > kMaxGatherCluster || tiles_m <= 0 || tiles_n <= 0 ||
        tiles_n > 0x7fffffffLL / p.cluster / tiles_m) return cudaErrorInvalidValue;
    p.tiles_m = static_cast<uint32_t>(tiles_m);
    p.tiles_n = static_cast<uint32_t>(tiles_n);
    // a raster group of 8 tile rows: about as many rows as columns of tiles run at a time
    p.raster_group = static_cast<int>(tiles_m < 8 ? tiles_m : 8);
    const long long per = (p.K + p.cluster - 1) / p.cluster;
    p.k_per_cta = (per + Cfg::BK - 1) / Cfg::BK * Cfg::BK;
    const long long tiles = tiles_m * tiles_n, resident = static_cast<long long>(num_sms) * Cfg::MINB;
    const long long grid = p.cluster > 1 ? tiles * p.cluster : !Cfg::FLAT || tiles < resident ? tiles : resident;
    // Back to back, the blocks of the next launch fill whatever slots the SMs have free.  Blocks without a cluster are kept to
    // their even share of an SM; clusters are not (with less room per SM fewer of them fit a GPC), but let the next kernel in
    // only when their main loop is done -- if they run in one round: of several rounds the last one releases it anyway.
    // At first / now / not chained at all: 7056 x 7 x 47 Float32, grid of 111: 19.5 / 7.2 / 10.2 us; 4199 x 17 x 40 FP64, 66
    // blocks: 19.2 / 6.8 / 10.3; 693 x 47 x 41 Float32, 44 blocks: 5.4 / 3.5 / 6.2; 96 x 128 x 432 FP64, clusters of 8: 12.5 /
    // 6.3 / 10.1; 176 x 169 x 399 Float32, clusters of 8: 11.6 / 10.1 / 12.3.
    p.release_late = p.cluster > 1 && grid <= resident ? 1 : 0;
    const int smem = p.cluster > 1 ? Cfg::SMEM : spread_smem(grid, num_sms, Cfg::MINB, Cfg::SMEM);
    return launch_chained(gather_contract_kernel<Cfg>, dim3(static_cast<unsigned>(grid)), dim3(Cfg::THREADS), static_cast<size_t>(smem), stream,
                          static_cast<unsigned>(p.cluster), p);
}

using F64Square = GatherCfg<double, 64, 64, 2, 2, 1, false, 4, 3>;
using F64SquareFlat = GatherCfg<double, 64, 64, 2, 2, 1, true, 3, 3>;
using F64Tall = GatherCfg<double, 128, 32, 4, 1, 1, false, 4, 2>;
using F64TallFlat = GatherCfg<double, 128, 32, 4, 1, 1, true, 3, 2>;
using F64Small = GatherCfg<double, 32, 32, 1, 1, 4, false, 4, 4>;
using F64SmallFlat = GatherCfg<double, 32, 32, 2, 2, 1, true, 4, 4>;
using F32Big = GatherCfg<float, 128, 128, 1, 8, 1, false, 4, 2>;
using F32Wide = GatherCfg<float, 128, 128, 2, 2, 1, false, 4, 2>;
using F32BigFlat = GatherCfg<float, 128, 128, 1, 8, 1, true, 4, 2>;
using F32Square = GatherCfg<float, 64, 64, 2, 2, 1, false, 4, 4>;
using F32SquareShort = GatherCfg<float, 64, 64, 1, 4, 1, false, 4, 4>;
using F32SquareFlat = GatherCfg<float, 64, 64, 1, 4, 1, true, 4, 4>;
using F32Tall = GatherCfg<float, 128, 32, 2, 2, 1, false, 4, 4>;
using F32TallFlat = GatherCfg<float, 128, 32, 2, 2, 1, true, 4, 3>;
using F32Small = GatherCfg<float, 32, 32, 1, 2, 4, false, 4, 4>;

}  // namespace

cudaError_t gather_configure()
{
    cudaError_t e = cudaSuccess;
    auto set = [&](auto* kernel, int smem) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem > kMaxSpreadSmem ? smem : kMaxSpreadSmem);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    };
    set(gather_contract_kernel<F64Square>, F64Square::SMEM);
    set(gather_contract_kernel<F64SquareFlat>, F64SquareFlat::SMEM);
    set(gather_contract_kernel<F64Tall>, F64Tall::SMEM);
    set(gather_contract_kernel<F64TallFlat>, F64TallFlat::SMEM);
    set(gather_contract_kernel<F64Small>, F64Small::SMEM);
    set(gather_contract_kernel<F64SmallFlat>, F64SmallFlat::SMEM);
    set(gather_contract_kernel<F32Big>, F32Big::SMEM);
    set(gather_contract_kernel<F32Wide>, F32Wide::SMEM);
    set(gather_contract_kernel<F32BigFlat>, F32BigFlat::SMEM);
    set(gather_contract_kernel<F32Square>, F32Square::SMEM);
    set(gather_contract_kernel<F32SquareShort>, F32SquareShort::SMEM);
    set(gather_contract_kernel<F32SquareFlat>, F32SquareFlat::SMEM);
    set(gather_contract_kernel<F32Tall>, F32Tall::SMEM);
    set(gather_contract_kernel<F32TallFlat>, F32TallFlat::SMEM);
    set(gather_contract_kernel<F32Small>, F32Small::SMEM);
    return e;
}

cudaError_t launch_gather_contract(const GatherParams& p, int scalar_type, int tile, int num_sms, cudaStream_t stream)
{
    if (p.flat && p.cluster != 1) return cudaErrorInvalidValue;
    if (scalar_type == 1) {
        if (tile == GATHER_SQUARE) return p.flat ? launch<F64SquareFlat>(p, num_sms, stream) : launch<F64Square>(p, num_sms, stream);
        if (tile == GATHER_TALL) return p.flat ? launch<F64TallFlat>(p, num_sms, stream) : launch<F64Tall>(p, num_sms, stream);
        if (tile == GATHER_SMALL) return p.flat ? launch<F64SmallFlat>(p, num_sms, stream) : launch<F64Small>(p, num_sms, stream);
    } else {
        if (tile == GATHER_BIG && p.form == GATHER_FORM_WIDE) return launch<F32Wide>(p, num_sms, stream);
        if (tile == GATHER_BIG) return p.flat ? launch<F32BigFlat>(p, num_sms, stream) : launch<F32Big>(p, num_sms, stream);
        if (tile == GATHER_SQUARE && p.form == GATHER_FORM_SHORT) return launch<F32SquareShort>(p, num_sms, stream);
        if (tile == GATHER_SQUARE) return p.flat ? launch<F32SquareFlat>(p, num_sms, stream) : launch<F32Square>(p, num_sms, stream);
        if (tile == GATHER_TALL) return p.flat ? launch<F32TallFlat>(p, num_sms, stream) : launch<F32Tall>(p, num_sms, stream);
        if (tile == GATHER_SMALL && !p.flat) return launch<F32Small>(p, num_sms, stream);
    }
    return cudaErrorInvalidValue;
}

}  // namespace tcontb
