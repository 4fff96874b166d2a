// kernels.hpp -- host-callable launchers of the sm_100a kernels (implemented in the .cu files).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <utility>

#include "planner.hpp"

namespace tcontb {

// Every kernel of a run is launched with this: its blocks may be scheduled, and set themselves up, while the kernel in front
// of it in the stream drains; they wait (chain_wait in chain.cuh) before they touch global memory.
//
// Blocks that are scheduled while the kernel in front still holds some SMs fill the free ones to the brim, and a grid that
// does not fill the GPU then runs on half of it.  spread_smem is the dynamic shared memory with which an SM holds no more
// blocks of such a grid than an even share (228 KB an SM, 1 KB of it reserved per block).
constexpr int kSmemPerSm = 228 * 1024;
constexpr int kMaxSpreadSmem = kSmemPerSm / 2 - 1024 + 128;   // one block per SM
inline int spread_smem(long long blocks, int num_sms, int resident, int smem)
{
    const long long per_sm = (blocks + num_sms - 1) / num_sms;
    if (per_sm >= resident) return smem;
    const int least = (kSmemPerSm / static_cast<int>(per_sm + 1) - 1024 + 128) / 128 * 128;
    return smem > least ? smem : least;
}
template <typename... KernelArgs, typename... Args>
cudaError_t launch_chained(void (*kernel)(KernelArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, unsigned cluster, Args&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

// ---- generic SIMT contraction (simt_contract.cu) -----------------------------------------
// GEMM view with offset tables: C[offCm[m] + offCn[n]] = sum_k A[offAm[m] + offAk[k]] * B[offBn[n] + offBk[k]].
struct SimtParams {
    const void* A;
    const void* B;
    void* C;
    int64_t M, N, K;
    const int64_t* offAm;
    const int64_t* offAk;
    const int64_t* offBn;
    const int64_t* offBk;
    const int64_t* offCm;
    const int64_t* offCn;
    int a_along_k, b_along_k;  // 0: threads run along the rows, 1: along k
};
cudaError_t launch_simt_contract(const SimtParams& p, int scalar_type, cudaStream_t stream);

// Division by a number known before the launch, by multiplication (Granlund and Montgomery, 1994): n / d = (umulhi(n, mul) + n)
// >> shr for n < 2^31, with shr = ceil(log2 d) and mul = floor(2^32 (2^shr - d) / d) + 1.  Five instructions where the
// hardware-less integer division takes thirty.
struct FastDiv {
    uint32_t d, mul, shr;
};
inline FastDiv make_fast_div(int64_t d)
{
    FastDiv f;
    f.d = static_cast<uint32_t>(d);
    f.shr = 0;
    while ((uint64_t(1) << f.shr) < f.d) ++f.shr;
    f.mul = static_cast<uint32_t>((((uint64_t(1) << f.shr) - f.d) << 32) / f.d + 1);
    return f;
}

// ---- any descriptor, gathered operands (gather_contract.cu) -----------------------------------
// A group of modes (rows, columns or contracted indices) of the GEMM view: flat index -> element offsets in the group's
// two tensors.  rows: x = A, y = C; columns: x = B, y = C; contracted: x = A, y = B.
constexpr int kMaxDigits = kMaxModes + 2;
struct RadixGroup {
    int n;     // modes (digits), fastest first, at least one
    int wide;  // flat indices of 2^31 and more: 64-bit division
    FastDiv ext[kMaxDigits];
    long long sx[kMaxDigits], sy[kMaxDigits];
    // Two modes cut in two digits each (rows whose stride-1 mode differs between A and C): digit 0 and t0 x digit 2 are one
    // index, which must stay below lim0, digit 1 and t1 x digit 3 the other (lim1).  lim0 = 0: no mode is cut.
    uint32_t t0, t1, lim0, lim1;
};
struct GatherParams {
    const void* A;
    const void* B;
    void* C;
    long long M, N, K;
    RadixGroup m, n, k;
    int a_along_k, b_along_k;  // 0: neighbouring threads gather neighbouring rows, 1: neighbouring k
    int cluster;               // CTAs that share a tile, each a range of k (1: no split)
    int flat;                  // 1: persistent blocks, one ring of stages across their tiles (cluster 1 only)
    int form;                  // GATHER_FORM_*
    int scaled;                // 0: C = A B; 1: C = alpha A B + beta C (C read only when beta is not zero)
    double alpha, beta;
    int release_late;          // the rest is filled in by the launcher: when the next kernel's blocks may be scheduled
    long long k_per_cta;
    uint32_t tiles_m, tiles_n;
    int raster_group;
};
cudaError_t gather_configure();  // once per device before the first launch
cudaError_t launch_gather_contract(const GatherParams& p, int scalar_type, int tile, int num_sms, cudaStream_t stream);

// ---- tensor permutation (transpose.cu) ------------------------------------------------------
struct TransposeParams {
    int rank;                      // after merging, <= kMaxModes
    int64_t ext[kMaxModes];        // source extents
    int64_t src_stride[kMaxModes]; // element strides of source mode i in the source
    int64_t dst_stride[kMaxModes]; // element strides of source mode i in the destination
    int64_t elements;
};
// Builds merged params for dst mode i = src mode perm[i]; returns false for a bad permutation.
// `src_stride` (optional): element strides of the source modes when the source is a view into a larger tensor.
// `dst_extent` (optional): extents of the destination modes, padding included.
bool make_transpose_params(int rank, const int64_t* src_extent, const int* perm, TransposeParams* out, const int64_t* src_stride = nullptr,
                           const int64_t* dst_extent = nullptr);
cudaError_t launch_transpose(const void* src, void* dst, const TransposeParams& p, int elem_bytes, cudaStream_t stream);

// ---- TF32 tcgen05 contraction (umma_tf32.cu) -------------------------------------------------
constexpr int kMaxOwners = 8;  // GPUs of one box

struct UmmaOperandDev {
    int major, slab_w, slabs_per_tile, n_row_digits, slab_bytes;
    int slabs_per_op, digit0_scale, oob_coord;
    int chunk_digit;  // which row digit is the chunk of the slab mode (scaled by digit0_scale, out-of-range past the tensor)
    int k0_scale;  // TMA coordinate of k digit 0 = k iteration * this
    int row_digit_dim[kMaxTmaRank];
    FastDiv row_digit_ext[kMaxTmaRank];
    long long row_digit_cstride[kMaxTmaRank];
    long long row_elem_cstride;
    int slab_mode_ext;
    long long total_slabs;
    int k_digit_dim[3];
    int slab_shift;                 // log2 of slab_w
    int split_inner;                // operand-level row fusion: see UmmaOperand (0 = none)
    FastDiv split_div;
    long long split_outer_cstride;
};
struct UmmaParams {
    UmmaOperandDev a, b;
    int BN, BK, stages, n_k_digits;
    int pair;  // 1: two-CTA clusters, 256 x BN tiles (cta_group::2); 0: one CTA per 128 x BN tile
    int producers;  // tcgen05 kernel: 2 = two producer warps taking turns stage by stage (needs an even number of stages)
    int k_digit_ext[3];
    int full_chunks;  // FP64 kernel: chunks of the chunked mode (k digit 0) below this one hold more than eight k (k chunk of 8: none)
    int k_iters;
    // Split-K: every tile is computed k_splits times over consecutive ranges of k_iters_per_split
    // iterations; split s writes its partial tile at C + s * split_stride (a workspace laid out like
    // C, summed afterwards by launch_splitk_reduce).  k_splits = 1: the kernel writes C itself.
    int k_splits, k_iters_per_split;
    long long split_stride;
    long long tiles_m, tiles_n;
    int raster_group;
    // divisors of the raster (filled in by fill_raster_divs): tiles of a whole group of tile rows, rows of a whole group and of the last one, splits
    FastDiv div_group, div_rows, div_last_rows, div_splits;
    float* C;       // tcgen05 TF32 kernel
    double* C64;    // TMA-fed FP64 kernel
    int scaled;            // 1: the epilogue stores alpha A B + beta C (C read only when beta is not zero); not with k_splits > 1 or owners
    double alpha, beta;
    int* status;  // device status word: set non-zero when a bounded wait gives up
    long long* prof;  // optional per-CTA cycle counters [grid][8] (TCONT_UMMA_PROF=1), else null
    // Test hooks of the bounded-wait exit: a shorter wait limit (0 = the default 2 s), and the index of one k iteration
    // per CTA whose stage the producer leaves unfilled and unannounced (-1 = none), so that the wait on it runs out with
    // nothing in flight for that stage.  FP64 kernel: the tile of a block with this iteration and those behind it are not
    // filled, and the producers raise the block's abort flag after the limit, which ends its waits as one that ran out does.
    unsigned long long wait_limit_ns;
    int test_skip_iter;
    // Contracted-mode split over several GPUs (tcgen05 kernel): this GPU's partial C is cut into `owners`
    // contiguous ranges along C's slowest mode, `tn_per_owner` tile columns each, and range o is stored straight
    // into the memory of the GPU that owns it, over NVLink: element i of the full C (i inside range o) goes to
    // owner_base[o][i].  owners = 0 or 1: everything goes to C.  `tn_rotate` shifts the order in which a GPU
    // visits the tile columns, so that the GPUs of a job write to different owners at any one time.
    int store_across_slabs;  // FP64 kernel: see UmmaSpec
    int piece;               // FP64 kernel: see UmmaSpec
    int slim;                // FP64 kernel: see UmmaSpec
    int groups;              // FP64 kernel: consumer groups of a block, see UmmaSpec
    int old_staged;          // FP64 kernel, three groups (set by the launcher): old values of C are copied to shared memory while a tile is computed
    // tcgen05 kernel.  1: the next kernel's blocks may be scheduled when this one's copies are issued, 0: at once.  Late where
    // every block stores many tiles of few k iterations: 806400 x 112 x 48 behind its permutation, 43 tiles a block: let in at
    // once 200 us, late 184, not chained 187.  Short kernels lose by it (4096 x 3072 x 32, 3 tiles: 16.9, late 17.3).  The FP64
    // kernel always releases at once: a choice in front of its main loop costs that loop 1.4 % (5184^3: 9518 and 9643 us),
    // which is more than output-bound kernels gain (81920 x 1152 x 16: 244, late 234).
    int release_late;
    // tcgen05 kernel, pace keeping: the CTAs (pairs) of a launch walk their panels along k at about the same
    // pace, so that a panel one of them fetched is still in L2 when the others of its tile row or column ask for
    // it.  pace[0] counts the producers that have ended, pace[1 + g] those that have started their block g of
    // 2^pace_shift k iterations; a producer starts block g only when all have started block g - pace_lead
    // (bounded wait; after one time-out it stops looking).  Zeroed before every launch.  nullptr = off.
    unsigned int* pace;
    int pace_shift, pace_lead;
    int owners, tn_per_owner, tn_rotate;
    float* owner_base[kMaxOwners];
};
// tmapA / tmapB are 128-byte CUtensorMap objects passed by value as kernel parameters.
cudaError_t launch_umma_tf32(const UmmaParams& p, const void* tmapA, const void* tmapB, int smem_bytes, int num_sms,
                             cudaStream_t stream);
// Opt-in maximum of dynamic shared memory per block on sm_100 (227 KB); set once per function and device.
constexpr int kMaxDynamicSmemBytes = 227 * 1024;
cudaError_t umma_tf32_configure();

// ---- TF32 with tiles across A's and C's stride-1 modes (across_tf32.cu) ------------------------
struct AcrossParams {
    // A unit's index: rows (chunks of y, chunks of x, other row modes o0, o1) and columns (chunks of n, other column modes p0, p1) of
    // tiles.  rows_first: the rows run faster, and x slowest among them; else the columns do, and x follows y.  `inner` = how many
    // of the faster kind there are.
    int rows_first;
    FastDiv inner, n_chunks, p0, y_chunks, x_chunks, o0, o1;
    int row_others, column_others;   // how many of the other modes there are
    int k_ext, k1_ext;               // extents of the chunked contracted mode and of the next one
    uint32_t units;
    int BN, BK, stages, k_iters;
    int b_major;            // 1: B's stride-1 mode is the column mode, 0: the chunked contracted mode
    int n_ext, x_ext;       // extents of the column mode and of A's stride-1 mode
    int release_late;       // see UmmaParams
    unsigned long long wait_limit_ns;   // see UmmaParams
    int test_skip_iter;
    int* status;
};
cudaError_t across_tf32_configure();  // once per device before the first launch
int across_tf32_smem(int stages, int BN, int BK);
cudaError_t launch_across_tf32(const AcrossParams& p, const void* tmapA, const void* tmapB, const void* tmapC, int num_sms, cudaStream_t stream);

// ---- TMA-fed FP64 tensor-path contraction (dmma_tma_f64.cu), same parameter block ------------
cudaError_t launch_dmma_tma(const UmmaParams& p, const void* tmapA, const void* tmapB, int num_sms, cudaStream_t stream);
cudaError_t dmma_tma_configure(const UmmaParams& p);

// ---- split-K: C[e] = sum over s of partial[s * stride + e], s ascending (splitk_reduce.cu) ----
// With alpha != 1 or beta != 0: C[e] = alpha * sum + beta * C[e] (C is read only when beta != 0).
cudaError_t splitk_reduce_configure();  // once per device before the first launch
cudaError_t launch_splitk_reduce(const void* partial, void* C, long long elements, int splits, long long stride, int elt_bytes,
                                 cudaStream_t stream, double alpha = 1.0, double beta = 0.0);
// One partial, tensors beyond L2: scheduled when the kernel in front has ended (see the .cu file).
cudaError_t launch_scale_pass(const double* product, double* C, long long elements, cudaStream_t stream, double alpha, double beta);

// ---- error-compensated Float32 (splitk_reduce.cu): lo = x - truncate_to_tf32(x), exact in fp32 ----
cudaError_t launch_tf32_residual(const float* x, float* lo, long long elements, cudaStream_t stream);

}  // namespace tcontb
