// Tensor-core kernel of the quantized Blocked-ELL projection for 32x32 blocks:
//     Y[cells, N] = alpha * deq(X_bell)[cells, genes] * W[genes, N] + beta * Y,   N in {128, 256}.
//
// Reference counterpart: quantized_blocked_ell_spmm_fwd_kernel_ (scalar, one thread per output
// element, src/compute/sparse/project/kernels/quantized_blocked_ell_spmm_fwd_kernel_.cuh:1-39) and
// the cuSPARSE f16 Blocked-ELL route (src/compute/sparse/project/project.cu:258-298).
//
// Formulation.  A block row is 32 cells and ell_cols/32 present blocks, each naming 32 genes.  A
// block row therefore is a dense contraction over K = 32 * blocks genes, but with only 32 rows --
// too few for the M side of a tcgen05 MMA.  The product is computed transposed:
//     D^T[N, 32 cells] += W^T[N, 32 genes of the block] * deq(X)^T[32 genes, 32 cells]
// i.e. M = 128 output columns per MMA (two MMAs side by side for N = 256), N_mma = 32 cells,
// K = 16 genes per instruction, fp32 accumulators in TMEM (lane = output column, TMEM column =
// cell).  Both operands are K-major in shared memory in the no-swizzle core-matrix layout
// (8 rows x 16 bytes per core matrix): that needs W^T, so a small kernel first writes, into the
// caller's workspace, W^T per gene block of 32 (genes padded with zeros) already in that operand
// layout; a block's N x 32 slice is then one contiguous 16 KB range.
//
// Operands are fp16 (eleven significant bits against bf16's eight), each stored times a power of two that brings
// its largest magnitude into [2^14, 2^15) so that fp16's exponent range cannot overflow; the factors (found on the
// device at every launch: largest |W|, and the bound of the decoded magnitudes from scales and offsets) are divided
// out of the result.  The decode runs on pairs: a byte permute (code -> fp16 1024 + code), a subtraction, a fused
// multiply-add with the pair's {scale, offset} from a table of fp16 pairs written beside W^T at launch.
//
// What bounds it: every block's slice of W^T comes from L2, N x 64 bytes per 32 x 32 codes (2.05 GB for 250k cells x 8,192 genes,
// 16 blocks wide, N = 256, against 0.38 GB of codes and Y), and bulk copies reach 14 TB/s of L2 -> shared memory at best.  The
// tensor pipe needs 40 cycles per 128 x 32 x 16 MMA, half of a block's time.  One CTA per SM walks block rows:
//   3 warps    one elected thread of each copies every third pair of neighbouring blocks' slices into the stages of a ring (216 KB);
//   16 warps   decode, in four groups that take the pairs of a block row in turn, into the same stages; their codes and
//              {scale, offset} pairs are read straight into registers a block row ahead, so nothing waits for DRAM and no
//              shared memory holds codes;
//   H warps    issue the MMAs, one per 128 output columns: one wait and one commit per pair of blocks;
//   warps 0-3  epilogue: tcgen05.ld the accumulators (double buffered, handed back before the last columns' stores), apply
//              alpha / beta, store Y rows coalesced.
// A form with two CTAs per SM, each with two stages of two blocks, whose decoding warps also started the copies, ran a stage's
// copy, MMAs and release one after the other (3,800 cycles per 36 KB): 222 us for that matrix, now 160 (N = 128: 185 -> 126); with
// a ring of single blocks and a commit per block the issuing threads were the bound (218 us; 331 before they were elected,
// see elect_one).
// Empty blocks (index 0xffffffff) are skipped; genes >= cols and cells past the last row decode to 0.  Every barrier wait is
// bounded; on a time-out a status word is set, every role ends, the copies and MMAs in flight are waited for, and the kernel
// frees its TMEM.
#include "kernels.cuh"
#include "operand_scaling.cuh"
#include "sm100_primitives.cuh"

#include <cuda_bf16.h>

namespace cb200 {

std::uint64_t qbell_tcgen05_workspace_bytes(std::int64_t cols, std::int64_t n) {
    const std::int64_t kpad = (cols + 31) / 32 * 32;
    return static_cast<std::uint64_t>(n * kpad * 2 + 256 + kpad * 4); // status block | W^T (fp16) | {scale, offset} pairs
}

namespace {

constexpr int kMaxWidth = 16;         // blocks per block row: the pairs whose codes a decode group keeps in registers
constexpr int kGroups = 4;            // decode groups of four warps
constexpr int kGroupPairs = kMaxWidth / 2 / kGroups;
static_assert(kGroupPairs * kGroups * 2 == kMaxWidth, "every pair has its group and place");
constexpr int kLoaders = 3;           // a copy with its wait and expect-tx holds its thread for hundreds of cycles, whatever its size
constexpr int kBTileBytes = 32 * 64;  // 32 cells x 32 genes fp16
constexpr int kEpilogueWarps = 4;
constexpr int kDecodeWarps = 4 * kGroups;
__host__ __device__ constexpr int a_tile_bytes(int h) { return h * 128 * 64; } // 128 h output columns x 32 genes fp16
__host__ __device__ constexpr int stage_bytes(int h) { return 2 * (a_tile_bytes(h) + kBTileBytes); } // a pair of blocks: [A][A][B][B]
__host__ __device__ constexpr int stages_of(int h) { return h == 2 ? 6 : 9; } // what shared memory holds; a loader's pairs keep to its stages
__host__ __device__ constexpr int threads_of(int h) { return 32 * (kEpilogueWarps + kDecodeWarps + h + kLoaders); }

struct tc_params {
    std::int64_t rows, cols;
    int width; // blocks per block row
    std::int64_t row_stride;
    const std::uint32_t *block_col_idx;
    const std::uint8_t *packed;
    const float *scales;
    const float *offsets;
    const __half *wt;        // [kpad/32 gene blocks][n x 32 slice of W^T in operand layout], fp16 times a power of two
    const uint2 *pairs;      // per pair of genes {scale pair, offset pair} as fp16, times the decoded operand's power of two;
                             // row-offset policy: the offset pair holds 1 for a gene of the matrix, 0 for padding
    const unsigned *w_absmax;    // largest |W| of this launch as float bits
    const unsigned *value_bound; // [2] bounds of the decoded magnitudes as float bits
    std::int64_t kpad;
    float *y;
    std::int64_t y_ld;
    std::int64_t block_row_begin, block_row_end; // block rows of this launch
    std::int64_t row_begin, row_end;             // cell rows of this launch
    int n;
    int policy;
    float alpha, beta;
    const float *bias;
    int epilogue;
    int *status;
    int poll_limit; // test hook: polls the MMA warps' waits for operands make
};

// K-major, no swizzle: core matrices of 8 rows x 16 bytes; LBO (between the two core matrices a
// K = 16 instruction reads) = 128 B, SBO (between groups of 8 rows) = 512 B.
__device__ __forceinline__ std::uint64_t smem_desc(std::uint32_t addr) {
    std::uint64_t d = 0;
    d |= static_cast<std::uint64_t>((addr & 0x3ffffu) >> 4);
    d |= static_cast<std::uint64_t>(128u >> 4) << 16;
    d |= static_cast<std::uint64_t>(512u >> 4) << 32;
    d |= static_cast<std::uint64_t>(1) << 46; // descriptor version of this architecture
    return d;
}
// kind::f16 instruction descriptor: D fp32, A and B fp16 (format 0), both K-major, N = 32, M = 128.
constexpr std::uint32_t kInstrDesc = (1u << 4) | ((32u >> 3) << 17) | ((128u >> 4) << 24);

// descriptors as {low, high} words: the high one is the same for every tile
__device__ __forceinline__ void mma_f16(std::uint32_t tmem_d, std::uint32_t desc_a, std::uint32_t desc_b, std::uint32_t desc_high, std::uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\tsetp.ne.b32 p, %4, 0;\n\tmov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
        :
        : "r"(tmem_d), "r"(desc_a), "r"(desc_b), "r"(kInstrDesc), "r"(accumulate), "r"(desc_high)
        : "memory");
}
// W [genes][n] (leading dimension ld) -> per gene block of 32, the n x 32 slice of W^T already in
// the shared-memory operand layout (core matrices of 8 output columns x 8 genes, 128 bytes each:
// byte offset of (column m, gene e) = (m/8)*512 + (e/8)*128 + (m%8)*16 + (e%8)*2), zero for
// genes >= cols, as fp16(w * ws), ws = operand_scale(largest |w|) (eleven significant bits instead of bf16's
// eight; the exponent range is kept by the power of two).  A block's slice is one contiguous n*64-byte range, so
// the main kernel fetches it with a single bulk copy.  The block's 16 gene pairs of {scale pair, offset pair}
// (fp16, times vs = operand_scale(bound of the decoded magnitudes)) are written beside it.
__global__ void __launch_bounds__(256) pack_w_kernel(const __nv_bfloat16 *w, std::int64_t ld, std::int64_t cols, int n, __half *packed_wt,
                                                     const float *scales, const float *offsets, int row_policy, const unsigned *w_absmax,
                                                     const unsigned *value_bound, uint2 *pairs) {
    wait_for_previous_launch();
    let_next_launch_start();
    const std::int64_t block = blockIdx.x;                     // gene block
    const float ws = operand_scale(__uint_as_float(*w_absmax));
    __half *dst = packed_wt + block * static_cast<std::int64_t>(n) * 32;
    // a thread makes one 16-byte piece: a column's values of eight consecutive genes; consecutive threads take consecutive
    // columns, so that their loads of a gene's row and their pieces are contiguous
    for (int item = threadIdx.x; item < n * 4; item += blockDim.x) {
        const int m = item % n, e8 = item / n;
        std::uint32_t packed[4];
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            float v[2];
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const std::int64_t gene = block * 32 + e8 * 8 + j + k;
                v[k] = gene < cols ? __bfloat162float(w[gene * ld + m]) : 0.0f;
            }
            const __half2 h = __floats2half2_rn(v[0] * ws, v[1] * ws);
            packed[j >> 1] = *reinterpret_cast<const std::uint32_t *>(&h);
        }
        *reinterpret_cast<uint4 *>(reinterpret_cast<unsigned char *>(dst) + (m >> 3) * 512 + e8 * 128 + (m & 7) * 16) =
            make_uint4(packed[0], packed[1], packed[2], packed[3]);
    }
    if (threadIdx.x < 16) {
        const float vs = operand_scale(__uint_as_float(value_bound[0]) + __uint_as_float(value_bound[1]));
        float sc[2], of[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const std::int64_t g = block * 32 + threadIdx.x * 2 + i;
            sc[i] = g < cols ? (scales != nullptr ? scales[g] : 1.0f) * vs : 0.0f;
            if (row_policy) of[i] = g < cols ? 1.0f : 0.0f;
            else of[i] = g < cols && offsets != nullptr ? offsets[g] * vs : 0.0f;
        }
        const __half2 s2 = __floats2half2_rn(sc[0], sc[1]), o2 = __floats2half2_rn(of[0], of[1]);
        pairs[block * 16 + threadIdx.x] = make_uint2(*reinterpret_cast<const unsigned *>(&s2), *reinterpret_cast<const unsigned *>(&o2));
    }
}

// The present blocks of a block row, and its pairs of neighbouring slots with a present block (bit 2 j of `pairs`: slots
// 2 j and 2 j + 1).  A block's place in the W ring and a pair's in the decode ring are their numbers in the CTA's walk.
struct block_row {
    std::uint32_t column; // of the block in this lane's slot
    unsigned blocks, pairs;
};
__device__ __forceinline__ std::uint32_t load_column(const tc_params &p, std::int64_t br, int lane) {
    return br < p.block_row_end && lane < p.width ? __ldg(p.block_col_idx + br * p.width + lane) : 0xffffffffu;
}
__device__ __forceinline__ block_row make_block_row(std::uint32_t column) {
    block_row r;
    r.column = column;
    r.blocks = __ballot_sync(0xffffffffu, column != 0xffffffffu);
    r.pairs = (r.blocks | (r.blocks >> 1)) & 0x55555555u;
    return r;
}
// the same answer in every lane: a warp that gives up leaves its loops as one
__device__ __forceinline__ bool warp_wait(std::uint64_t *bar, int parity, volatile int *abort_flag, int limit = kPollLimit) {
    return __any_sync(0xffffffffu, bar_wait(smem_addr(bar), static_cast<std::uint32_t>(parity & 1), abort_flag, limit)) != 0;
}
__device__ __forceinline__ bool warp_wait_sleeping(std::uint64_t *bar, int parity, volatile int *abort_flag, unsigned ns) {
    return __any_sync(0xffffffffu, bar_wait_sleeping(smem_addr(bar), static_cast<std::uint32_t>(parity & 1), abort_flag, ns)) != 0;
}

// TEST_HOOK: what cb200_test_arm_wait_timeout selects.  Decode group 0 hands nothing over, so that the MMA warps' waits run out
// (after p.poll_limit polls) with copies in flight whose barriers lack arrivals; the rest is common code.
template<int BITS, int H /* N / 128 */, bool TEST_HOOK>
__global__ void __launch_bounds__(threads_of(H), 1) qbell_tcgen05_kernel(const tc_params p) {
    constexpr int kATileBytes = a_tile_bytes(H), kStageBytes = stage_bytes(H), kStages = stages_of(H);
    static_assert(kStages % kLoaders == 0, "a loader's pairs keep to its stages");
    constexpr int kTmemCols = 2 * H * 32; // two accumulator buffers
    extern __shared__ __align__(1024) unsigned char smem[];
    // [kStages][A][A][B][B] | barriers | tmem base | flags | what an abort drains
    std::uint64_t *bars = reinterpret_cast<std::uint64_t *>(smem + kStages * kStageBytes);
    std::uint64_t *full = bars;                      // [kStages] loader (with the copies' bytes) and the warps of a decode group -> MMA
    std::uint64_t *empty = full + kStages;           // [kStages] MMA commits -> loader and decode group
    std::uint64_t *acc_full = empty + kStages;       // [2]       MMA commits -> epilogue
    std::uint64_t *acc_empty = acc_full + 2;         // [2]       epilogue -> MMA (one arrival per warp)
    std::uint64_t *mma_drain = acc_empty + 2;        // [H]       an MMA warp's own, used once, after an abort
    std::uint32_t *tmem_slot = reinterpret_cast<std::uint32_t *>(mma_drain + H);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *row_has_blocks = reinterpret_cast<volatile int *>(tmem_slot + 2); // [2] per accumulator buffer
    volatile int *issued = reinterpret_cast<volatile int *>(tmem_slot + 4); // [kStages] pair last copied into the stage, x kGroups + its decode group; -1
    volatile int *handed_over = issued + kStages;                          // [kDecodeWarps] last pair the warp handed over, once it has ended

    const int tid = threadIdx.x, warp = warp_of_block(), lane = tid & 31;
    const std::uint32_t smem0 = smem_addr(smem);

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) {
            bar_init(smem_addr(full + s), 1 + 4);
            bar_init(smem_addr(empty + s), H);
            issued[s] = -1;
        }
        for (int h = 0; h < H; ++h) bar_init(smem_addr(mma_drain + h), 1);
        for (int b = 0; b < 2; ++b) {
            bar_init(smem_addr(acc_full + b), H);
            bar_init(smem_addr(acc_empty + b), kEpilogueWarps);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const std::uint32_t tmem_base = *tmem_slot;
    wait_for_previous_launch();

    const std::int64_t first = p.block_row_begin + blockIdx.x, step = gridDim.x;
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;

    if (warp < kEpilogueWarps) {
        // ================= epilogue: TMEM lane = output column, TMEM column = cell =================
        // both operands were stored times powers of two (fp16 range): the result is divided by them again
        const float alpha = p.alpha / (operand_scale(__uint_as_float(__ldg(p.w_absmax))) *
                                       operand_scale(__uint_as_float(__ldg(p.value_bound)) + __uint_as_float(__ldg(p.value_bound + 1))));
        const bool composed = p.epilogue != CB200_EPILOGUE_NONE;
        int use = 0; // block rows of this CTA
        for (std::int64_t br = first; br < p.block_row_end; br += step, ++use) {
            const int buf = use & 1;
            if (warp_wait_sleeping(acc_full + buf, use >> 1, abort_flag, 100u)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const bool any = row_has_blocks[buf] != 0;
            const std::int64_t row0 = br * 32;
            const bool plain = row0 >= p.row_begin && row0 + 32 <= p.row_end && p.beta == 0.0f && !composed;
#pragma unroll 1
            for (int h = 0; h < H; ++h) {
                float v[32];
                if (any) {
                    tmem_ld32(tmem_base + (static_cast<std::uint32_t>(warp * 32) << 16) + buf * (H * 32) + h * 32, v);
                } else {
#pragma unroll
                    for (int i = 0; i < 32; ++i) v[i] = 0.0f;
                }
                if (h == H - 1) { // the accumulators are in registers
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) bar_arrive(smem_addr(acc_empty + buf));
                }
                const int col = h * 128 + warp * 32 + lane;
                // this thread writes one output column of 32 rows: its bias is loaded once
                const float bias = composed && epilogue_has_bias(p.epilogue) ? __ldg(p.bias + col) : 0.0f;
                float *out = p.y + row0 * p.y_ld + col;
                if (plain) {
#pragma unroll
                    for (int c = 0; c < 32; ++c, out += p.y_ld) *out = alpha * v[c];
                } else {
#pragma unroll
                    for (int c = 0; c < 32; ++c, out += p.y_ld) {
                        const std::int64_t row = row0 + c;
                        if (row >= p.row_begin && row < p.row_end) {
                            float r = alpha * v[c];
                            if (p.beta != 0.0f) r = fmaf(p.beta, *out, r);
                            if (composed) r = apply_epilogue(r, bias, p.epilogue);
                            *out = r;
                        }
                    }
                }
            }
        }
    } else if (warp < kEpilogueWarps + kDecodeWarps) {
        // ================= decode: group g takes the pairs g, g + kGroups, ... of every block row; a lane decodes eight genes
        // of one cell of each of the pair's blocks.  The four lanes of a cell read a 32-byte sector; eight lanes of one
        // chunk store 128 contiguous bytes of the operand tile =================
        const int group = (warp - kEpilogueWarps) >> 2, cell = ((warp - kEpilogueWarps) & 3) * 8 + (lane & 7), chunk = lane >> 3;
        const float vs = operand_scale(__uint_as_float(__ldg(p.value_bound)) + __uint_as_float(__ldg(p.value_bound + 1)));
        const __half2 magic = __half2half2(__ushort_as_half(static_cast<unsigned short>(0x6400u))); // 1024: fp16(0x6400 | code) = 1024 + code
        uint2 codes[kGroupPairs][2];   // of the block row to come, and its blocks'
        uint4 meta[kGroupPairs][2][2]; // {scale pair, offset pair} of the chunk's four gene pairs
        const auto fetch = [&](std::int64_t br, std::uint32_t row_column, int r) {
            const std::int64_t row = br * 32 + cell;
            const bool valid = br < p.block_row_end && row >= p.row_begin && row < p.row_end;
            const std::uint8_t *from = p.packed + (valid ? row * p.row_stride : 0);
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                const int slot = (group + r * kGroups) * 2 + t;
                const std::uint32_t bc = __shfl_sync(0xffffffffu, row_column, slot);
                codes[r][t] = make_uint2(0u, 0u);
                if (bc == 0xffffffffu) continue;
                if (valid) {
                    if constexpr (BITS == 8) codes[r][t] = __ldg(reinterpret_cast<const uint2 *>(from + slot * 32 + chunk * 8));
                    else codes[r][t].x = __ldg(reinterpret_cast<const unsigned *>(from + slot * 16 + chunk * 4));
                }
                const uint4 *pairs = reinterpret_cast<const uint4 *>(p.pairs + static_cast<std::int64_t>(bc) * 16 + chunk * 4);
                meta[r][t][0] = __ldg(pairs);
                meta[r][t][1] = __ldg(pairs + 1);
            }
        };
        std::uint32_t column = load_column(p, first, lane), next_column = load_column(p, first + step, lane);
#pragma unroll
        for (int r = 0; r < kGroupPairs; ++r) fetch(first, column, r);
        int item0 = 0; // pairs of the CTA before this block row
        int last = -1; // pair last handed over
        bool dead = false;
        for (std::int64_t br = first; br < p.block_row_end && !dead; br += step) {
            const block_row blocks = make_block_row(column);
            column = next_column;
            next_column = load_column(p, br + 2 * step, lane);
            const std::int64_t row = br * 32 + cell;
            const bool cell_valid = row >= p.row_begin && row < p.row_end;
            // row-offset policy: the cell's offset, times the operand's power of two, for both genes of a pair
            const __half2 row_offset2 = __float2half2_rn((row_policy && p.offsets != nullptr && cell_valid) ? __ldg(p.offsets + row) * vs : 0.0f);
#pragma unroll
            for (int r = 0; r < kGroupPairs; ++r) {
                const int j = group + r * kGroups;
                if (((blocks.pairs >> (2 * j)) & 1u) != 0u) {
                    const int item = item0 + __popc(blocks.pairs & ((1u << (2 * j)) - 1u)), stage = item % kStages;
                    if (warp_wait_sleeping(empty + stage, item / kStages + 1, abort_flag, 40u)) { dead = true; break; }
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (((blocks.blocks >> (2 * j + t)) & 1u) == 0u) continue;
                        // per pair of codes a byte permute (code -> fp16 1024 + code), a subtraction (exact), a fused
                        // multiply-add with the pair's {scale, offset}; genes past the matrix have scale and offset 0
                        std::uint32_t out[4] = {0u, 0u, 0u, 0u};
                        if (cell_valid) {
                            const std::uint32_t lo = codes[r][t].x, hi = codes[r][t].y;
                            std::uint32_t raw[4];
                            if constexpr (BITS == 8) {
                                raw[0] = __byte_perm(lo, 0x64646464u, 0x4140u);
                                raw[1] = __byte_perm(lo, 0x64646464u, 0x4342u);
                                raw[2] = __byte_perm(hi, 0x64646464u, 0x4140u);
                                raw[3] = __byte_perm(hi, 0x64646464u, 0x4342u);
                            } else {
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    const std::uint32_t two = lo >> (8 * e); // the byte that holds the pair's two 4-bit codes
                                    raw[e] = 0x64006400u | (two & 0xfu) | ((two & 0xf0u) << 12);
                                }
                            }
                            const std::uint32_t sc[4] = {meta[r][t][0].x, meta[r][t][0].z, meta[r][t][1].x, meta[r][t][1].z};
                            const std::uint32_t of[4] = {meta[r][t][0].y, meta[r][t][0].w, meta[r][t][1].y, meta[r][t][1].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const __half2 code2 = __hsub2(*reinterpret_cast<const __half2 *>(&raw[e]), magic);
                                __half2 o2 = *reinterpret_cast<const __half2 *>(&of[e]);
                                if (row_policy) o2 = __hmul2(o2, row_offset2); // the pair's {1 | 0} times the cell's offset
                                const __half2 v = __hfma2(code2, *reinterpret_cast<const __half2 *>(&sc[e]), o2);
                                out[e] = *reinterpret_cast<const std::uint32_t *>(&v);
                            }
                        }
                        const std::uint32_t dst = smem0 + stage * kStageBytes + 2 * kATileBytes + t * kBTileBytes + (cell >> 3) * 512 + chunk * 128 + (cell & 7) * 16;
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(out[0]), "r"(out[1]), "r"(out[2]), "r"(out[3]) : "memory");
                    }
                    fence_async_proxy(); // written with ordinary stores, read by the MMAs
                    __syncwarp();
                    if (TEST_HOOK && group == 0) continue;
                    if (lane == 0) bar_arrive(smem_addr(full + stage));
                    last = item;
                }
            }
#pragma unroll
            for (int r = 0; r < kGroupPairs; ++r) fetch(br + step, column, r);
            item0 += __popc(blocks.pairs);
        }
        if (lane == 0) handed_over[warp - kEpilogueWarps] = last;
    } else if (warp < kEpilogueWarps + kDecodeWarps + H) {
        // ================= MMA issuers: warp h issues the MMAs of output columns [128 h, 128 h + 128) =================
        const int h = warp - kEpilogueWarps - kDecodeWarps;
        const std::uint64_t desc0 = smem_desc(smem0);
        const std::uint32_t lo0 = static_cast<std::uint32_t>(desc0), hi = static_cast<std::uint32_t>(desc0 >> 32);
        int use = 0, stage = 0, phase = 0;
        bool dead = false;
        std::uint32_t column = load_column(p, first, lane);
        for (std::int64_t br = first; br < p.block_row_end && !dead; br += step, ++use) {
            const int buf = use & 1;
            const block_row blocks = make_block_row(column);
            column = load_column(p, br + step, lane);
            if (warp_wait(acc_empty + buf, (use >> 1) + 1, abort_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const std::uint32_t d = tmem_base + buf * (H * 32) + h * 32;
            std::uint32_t accumulate = 0; // the block row's first MMA overwrites the accumulators
            for (unsigned todo = blocks.pairs; todo != 0u; todo &= todo - 1u) {
                const unsigned present = blocks.blocks >> (__ffs(static_cast<int>(todo)) - 1);
                dead = warp_wait(full + stage, phase, abort_flag, TEST_HOOK ? p.poll_limit : kPollLimit);
                if (dead) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const std::uint32_t a = lo0 + ((stage * kStageBytes + h * 8192) >> 4), b = lo0 + ((stage * kStageBytes + 2 * kATileBytes) >> 4);
                    if ((present & 1u) != 0u) {
                        mma_f16(d, a, b, hi, accumulate);
                        mma_f16(d, a + 16, b + 16, hi, 1u);
                    }
                    if ((present & 2u) != 0u) {
                        mma_f16(d, a + (kATileBytes >> 4), b + (kBTileBytes >> 4), hi, accumulate | (present & 1u));
                        mma_f16(d, a + (kATileBytes >> 4) + 16, b + (kBTileBytes >> 4) + 16, hi, 1u);
                    }
                    mma_commit(smem_addr(empty + stage));
                }
                accumulate = 1;
                if (++stage == kStages) { stage = 0; phase ^= 1; }
            }
            if (!dead && elect_one()) {
                if (h == 0) row_has_blocks[buf] = blocks.blocks != 0u ? 1 : 0;
                mma_commit(smem_addr(acc_full + buf)); // accumulators complete (or nothing was issued)
            }
        }
    } else {
        // ================= loaders: a block's slice of W^T is one contiguous copy, already in operand layout; loader l takes the
        // pairs whose number in the CTA's walk is l modulo kLoaders =================
        const int loader = warp - kEpilogueWarps - kDecodeWarps - H;
        int number = 0, stage = loader, phase = 1;
        bool dead = false; // the elected lane: a wait was given up
        std::uint32_t column = load_column(p, first, lane);
        for (std::int64_t br = first; br < p.block_row_end; br += step) {
            const block_row blocks = make_block_row(column);
            column = load_column(p, br + step, lane);
            for (unsigned todo = blocks.pairs; todo != 0u; todo &= todo - 1u, ++number) {
                if (number % kLoaders != loader) continue;
                const int even = __ffs(static_cast<int>(todo)) - 1;
                std::uint32_t bc[2];
#pragma unroll
                for (int t = 0; t < 2; ++t) bc[t] = __shfl_sync(0xffffffffu, blocks.column, even + t);
                if (elect_one() && !dead) {
                    dead = bar_wait(smem_addr(empty + stage), static_cast<std::uint32_t>(phase), abort_flag);
                    if (!dead) { // no new copies once a wait of the CTA has run out
                        issued[stage] = number * kGroups + (even >> 1) % kGroups;
                        bar_arrive_expect_tx(smem_addr(full + stage), ((bc[0] != 0xffffffffu) + (bc[1] != 0xffffffffu)) * kATileBytes);
#pragma unroll
                        for (int t = 0; t < 2; ++t)
                            if (bc[t] != 0xffffffffu)
                                bulk_copy_g2s(smem0 + stage * kStageBytes + t * kATileBytes, p.wt + static_cast<std::int64_t>(bc[t]) * (H * 128 * 32), kATileBytes,
                                              smem_addr(full + stage));
                    }
                }
                stage += kLoaders;
                if (stage >= kStages) { stage = loader; phase ^= 1; }
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag != 0) {
        // Every role has ended.  The copies and MMAs still in flight finish before the CTA gives up its shared and tensor memory.
        // A stage's barrier may lack arrivals of the decode group that owns its pair: the loader makes up for them.
        if (warp >= kEpilogueWarps + kDecodeWarps + H) {
            if (elect_one()) {
                for (int stage = warp - kEpilogueWarps - kDecodeWarps - H; stage < kStages; stage += kLoaders) {
                    if (issued[stage] < 0) continue;
                    const int item = issued[stage] / kGroups, group = issued[stage] % kGroups;
                    for (int w = 0; w < 4; ++w)
                        if (handed_over[group * 4 + w] < item) bar_arrive(smem_addr(full + stage));
                    bar_wait_drain(smem_addr(full + stage), static_cast<std::uint32_t>((item / kStages) & 1));
                }
            }
        } else if (warp >= kEpilogueWarps + kDecodeWarps) {
            if (elect_one()) {
                mma_commit(smem_addr(mma_drain + (warp - kEpilogueWarps - kDecodeWarps)));
                bar_wait_drain(smem_addr(mma_drain + (warp - kEpilogueWarps - kDecodeWarps)), 0u);
            }
        }
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
    if (tid == 0 && *abort_flag != 0 && p.status != nullptr) atomicExch(p.status, 1);
}

template<int BITS, int H, bool TEST_HOOK = false>
cb200_status launch(const tc_params &p, int sm_count, cudaStream_t stream) {
    constexpr std::size_t smem = stages_of(H) * stage_bytes(H) + (2 * stages_of(H) + 4 + H) * sizeof(std::uint64_t) + (4 + stages_of(H) + kDecodeWarps) * sizeof(int);
    static_assert(smem <= 232448, "shared memory budget");
    CB200_CUDA_OK(cudaFuncSetAttribute(qbell_tcgen05_kernel<BITS, H, TEST_HOOK>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    const std::int64_t block_rows = p.block_row_end - p.block_row_begin;
    const unsigned grid = static_cast<unsigned>(std::min<std::int64_t>(block_rows, sm_count));
    CB200_CUDA_OK(launch_kernel(true, qbell_tcgen05_kernel<BITS, H, TEST_HOOK>, grid, threads_of(H), smem, stream, p));
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

} // namespace

cb200_status launch_qbell_tcgen05(const qbell_view &x, const dense_args &d, std::int64_t row_begin,
                                  std::int64_t row_end, void *workspace, std::uint64_t workspace_bytes, int sm_count,
                                  cudaStream_t stream, bool *taken) {
    *taken = false;
    if (x.block_size != 32 || (d.n != 128 && d.n != 256) || d.dense_dtype != CB200_DTYPE_BF16) return CB200_STATUS_SUCCESS;
    if (x.bits != 8 && x.bits != 4) return CB200_STATUS_SUCCESS;
    if (x.ell_cols <= 0 || x.ell_cols % 32 != 0 || x.ell_cols / 32 > kMaxWidth) return CB200_STATUS_SUCCESS;
    // the decode warps read up to 8 bytes at a time
    if (x.row_stride_bytes % 16 != 0 || reinterpret_cast<std::uintptr_t>(x.packed) % 16u != 0u) return CB200_STATUS_SUCCESS;
    if (reinterpret_cast<std::uintptr_t>(x.scales) % 16u != 0u || reinterpret_cast<std::uintptr_t>(x.offsets) % 16u != 0u) return CB200_STATUS_SUCCESS;
    if (workspace == nullptr || workspace_bytes < qbell_tcgen05_workspace_bytes(x.cols, d.n)) return CB200_STATUS_SUCCESS;
    if (reinterpret_cast<std::uintptr_t>(workspace) % 256u != 0u) return CB200_STATUS_SUCCESS;
    if (row_end <= row_begin) return CB200_STATUS_SUCCESS;

    const std::int64_t kpad = (x.cols + 31) / 32 * 32;
    int *status = static_cast<int *>(workspace);
    unsigned *w_absmax = reinterpret_cast<unsigned *>(workspace) + 1;    // float bits of the largest |W|
    unsigned *value_bound = reinterpret_cast<unsigned *>(workspace) + 2; // [2], [3]: bounds of the decoded magnitudes
    __half *wt = reinterpret_cast<__half *>(static_cast<unsigned char *>(workspace) + 256);
    uint2 *pairs = reinterpret_cast<uint2 *>(static_cast<unsigned char *>(workspace) + 256 + d.n * kpad * 2);
    const bool row_policy = x.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    CB200_CUDA_OK(cudaMemsetAsync(status, 0, 4 * sizeof(int), stream));
    const std::int64_t elements = x.cols * d.n;
    const unsigned w_blocks = static_cast<unsigned>(std::min<std::int64_t>((elements + 1023) / 1024, 4 * static_cast<std::int64_t>(sm_count)));
    const std::int64_t span = std::max<std::int64_t>(x.cols, row_policy ? x.rows : 0);
    operand_bounds_kernel<<<w_blocks + static_cast<unsigned>((span + 255) / 256), 256, 0, stream>>>(
        static_cast<const __nv_bfloat16 *>(d.dense), d.dense_ld, x.cols, static_cast<int>(d.n), w_blocks, x.scales,
        row_policy ? nullptr : x.offsets, row_policy ? x.offsets : nullptr, x.rows, static_cast<float>((1 << x.bits) - 1), w_absmax, value_bound);
    CB200_CUDA_OK(launch_kernel(true, pack_w_kernel, dim3(static_cast<unsigned>(kpad / 32)), 256, 0, stream, static_cast<const __nv_bfloat16 *>(d.dense),
                                d.dense_ld, x.cols, static_cast<int>(d.n), wt, x.scales, x.offsets, row_policy ? 1 : 0, w_absmax, value_bound, pairs));
    count_launch(2);
    CB200_CUDA_OK(cudaGetLastError());
    tc_params p{};
    p.rows = x.rows; p.cols = x.cols; p.width = x.ell_cols / 32; p.row_stride = x.row_stride_bytes;
    p.block_col_idx = x.block_col_idx; p.packed = x.packed; p.scales = x.scales; p.offsets = x.offsets;
    p.wt = wt; p.pairs = pairs; p.w_absmax = w_absmax; p.value_bound = value_bound; p.kpad = kpad; p.y = d.out; p.y_ld = d.out_ld;
    p.block_row_begin = row_begin / 32; p.block_row_end = (row_end + 31) / 32;
    p.row_begin = row_begin; p.row_end = row_end;
    p.n = static_cast<int>(d.n); p.policy = x.policy; p.alpha = d.alpha; p.beta = d.beta; p.bias = d.bias; p.epilogue = d.epilogue; p.status = status;
    *taken = true;
    if (x.bits == 8 && d.n == 256 && test_poll_limit() != 0) {
        p.poll_limit = test_poll_limit();
        return launch<8, 2, true>(p, sm_count, stream);
    }
    if (x.bits == 8) return d.n == 256 ? launch<8, 2>(p, sm_count, stream) : launch<8, 1>(p, sm_count, stream);
    return d.n == 256 ? launch<4, 2>(p, sm_count, stream) : launch<4, 1>(p, sm_count, stream);
}

} // namespace cb200
