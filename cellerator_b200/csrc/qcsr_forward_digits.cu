// Forward projection with exact integer sums on the tensor cores:
//     Y[cells, N] = act(alpha * deq(X)[cells, genes] * W[genes, N] + beta * Y + bias),   zero-points per gene.
//
// Reference counterpart: the decode to floats and csr_spmm_fwd_kernel_ (src/compute/sparse/project/kernels/csr_spmm_fwd_kernel_.cuh:1-22),
// one thread per (row, output column).
//
// Formulation.  A row of Y is  sum of code * (scale W[gene]) + sum of (offset W[gene])  over its entries.  Both operands on W's side are
// written in fixed point with one step per column, as four signed digits of base 256 each; the matrix's side is a code (less
// 128, to be signed) and a constant per entry.  The 8-bit integer MMAs add the products exactly, in any order, so a row has the
// same bits however the genes are cut and whatever rows stand beside it.  For entry {c, 127} of a gene with step d:
//     qc = round(scale W / d),   qi = round((offset W / d + 128 qc) / 127):   (c - 128) qc + 127 qi = c qc + offset W / d + rounding,
// the rounding of qc counts c times, that of qi 127 times, each at most half a step of 2^-30 of the column's largest operand.
// Against 64 bits (2-norm, 20,000 x 2,000 and 4,099 x 33,538): 4.3e-8 and 4.6e-8, where fp32 FMAs leave 1.1e-7 and 1.3e-7.
//
// A column whose operands are small beside the largest (kMostSpread), or an operand that is not finite, does not fit: the
// device notices while it lays W out, this kernel then does nothing, and the gather kernel behind it takes all rows.  The rows of pieces
// in which a cell holds a gene twice are summed here, entry by entry.
//
// Data.  The entries come as words {code, place in the tile}, in pieces of 16 or 32 cells and inside them by window of 128 genes
// (digit_words_kernel); a prepared operation keeps them, a call that sees its matrix once makes them in its workspace.  (Reading the
// CSR arrays here instead, a lane finding its entry's row by search or a few lanes per row, takes more instructions of the shared-memory
// pipe -- shuffles, two loads and a store per 32 entries at best -- than an SM can issue: 4,000 to 16,000 cycles a tile against 2,048 of MMAs.)
//
// Structure of a CTA (640 threads, one per SM): a tile is 256 cells x 128 genes, 2 bytes a place {code, 127}: K-major, 128-byte
// swizzle, 64 KB.  Two groups of eight warps zero and fill alternate tiles, a warp each brings them their words, one warp issues the MMAs
// (two halves of the cells, K steps of 16 genes, N = 4 digits x the columns of W), one feeds the ring of W.  The tiles, group after
// group of cells and in each window after window, are dealt to the CTAs in equal shares; a group that a CTA has to itself is written
// to Y from tensor memory, the sums of the others go through the workspace as 64-bit integers and sum_parts_kernel adds them.
//
// What bounds it: at 33,538 genes and N = 64 the tensor pipe, sixteen 128 x 256 x 32 MMAs of 128 cycles in the 2,300 cycles of a tile;
// at 17 % density and N = 32 the scatter (5,600 words a tile, 3,300 cycles with two chunks of 2,048 waited for; chunks of 4,096 there).
// One call that makes its words, gathered rows of W -> this: 4,099 x 33,538, N = 50 bf16, 117 -> 107 us (words 39, W 13, this kernel
// 45, sums 6, in places beside each other); 20,000 x 2,000, N = 32, 85 -> 76; 8,192 x 33,538, N = 128, 455 -> 250; 3,000 x 8,000, N =
// 128, 112 -> 64.
#include "dependent_launch.cuh"
#include "kernels.cuh"
#include "sm100_primitives.cuh"

#include <algorithm>

namespace cb200 {
namespace {

constexpr int kWin = 128;
constexpr int kRows = 256;
constexpr int kSlices = 4;
constexpr int kMostGroupPieces = kRows / 16; // pieces of 16 or 32 cells, whose words lie together
constexpr int kScatterWarps = 16;
constexpr int kGroupThreads = kScatterWarps * 16;
constexpr int kThreads = (kScatterWarps + 4) * 32;
// words a scatter group gets at a time: what shared memory holds beside the ring of W
__host__ __device__ constexpr int chunk_entries(int nb) { return nb == 64 ? 2048 : 4096; }
constexpr std::uint32_t kPadding = 0x80000000u; // a word that holds no entry
constexpr int kHalfBytes = kRows * 128;      // 64 genes of every row
constexpr int kTileBytes = 2 * kHalfBytes;
constexpr int kWPieces = 4;                  // W comes in pieces of 32 genes
constexpr int kMaxCtas = 256;
constexpr int kMaxColumns = 256;
// A column is written in fixed point if its numbers are on average (of the binary exponents of those that are not zero, which a few
// large ones do not move) not more than 2^6 below the largest: half a step is then at most 2^-24 of the average number, what fp32
// rounds a product at, while a normal distribution leaves 2^-27.
constexpr unsigned kMostSpread = 6;
// |code| <= 128, 127 and digits of at most 128: 2^15 an entry, 65,536 entries of a row until a sum could leave 32 bits
constexpr std::int64_t kMostGenes = 61440;

__host__ __device__ constexpr int mma_columns(int nb) { return nb * kSlices; }
__host__ __device__ constexpr int w_piece_bytes(int nb) { return 64 * mma_columns(nb); }
__host__ __device__ constexpr int ring_pieces(int nb) { return nb == 64 ? 5 : 8; }

constexpr int kParts = 96;
constexpr std::uint64_t kStepsAt = 256, kPartMaxAt = kStepsAt + kMaxColumns * 8, kPartSumAt = kPartMaxAt + kParts * kMaxColumns * 4,
                        kRecordsAt = kPartSumAt + kParts * kMaxColumns * 16;
static_assert(kRecordsAt % 256 == 0, "W's records are copied 16 bytes at a time");

// ---- W in digits -----------------------------------------------------------------------------------------------------------

struct meta_source {
    const float *scales, *offsets;
    float bias; // 128 for 8-bit codes, 0 for 4-bit ones
    __device__ __forceinline__ float2 of(std::int64_t gene) const {
        return make_float2(scales != nullptr ? __ldg(scales + gene) : 1.0f, offsets != nullptr ? __ldg(offsets + gene) : 0.0f);
    }
    // the larger of the two operands of a gene, for |W| = 1
    __device__ __forceinline__ float reach(float2 so) const { // (as bits a NaN is the larger)
        return __uint_as_float(max(__float_as_uint(so.x) & 0x7fffffffu, __float_as_uint((fabsf(so.y) + bias * fabsf(so.x)) * (1.0f / 127.0f)) & 0x7fffffffu));
    }
};

// Largest operand of each column (as bits; an infinity or a NaN is the largest), and the operands' binary exponents' sum and number where
// one is not zero, in parts.
template<typename WT>
__global__ void __launch_bounds__(1024) w_range_kernel(const WT *w, std::int64_t ld, int n, int padded, std::int64_t genes, meta_source meta,
                                                       unsigned *part_max, ulonglong2 *part_sum, int *status) {
    __shared__ unsigned most_of[1024];
    __shared__ unsigned exponents_of[1024], count_of[1024];
    let_next_launch_start();
    if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    const int c = threadIdx.x % padded, lanes = 1024 / padded;
    unsigned most = 0u, exponents = 0u, count = 0u;
    if (c < n) {
        const std::int64_t step = static_cast<std::int64_t>(gridDim.x) * lanes;
        const auto take = [&](float v, float reach) {
            const unsigned bits = __float_as_uint(fabsf(v) * reach) & 0x7fffffffu;
            most = max(most, bits);
            exponents += bits >> 23;
            count += bits != 0u ? 1u : 0u;
        };
        std::int64_t g = static_cast<std::int64_t>(blockIdx.x) * lanes + threadIdx.x / padded;
        for (; g + 3 * step < genes; g += 4 * step) {
            float v[4], reach[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[k] = load1(w + (g + k * step) * ld + c);
                reach[k] = meta.reach(meta.of(g + k * step));
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) take(v[k], reach[k]);
        }
        for (; g < genes; g += step) take(load1(w + g * ld + c), meta.reach(meta.of(g)));
    }
    most_of[threadIdx.x] = most;
    exponents_of[threadIdx.x] = exponents;
    count_of[threadIdx.x] = count;
    __syncthreads();
    if (threadIdx.x < static_cast<unsigned>(padded)) {
        unsigned long long sum = exponents, number = count;
        for (int k = 1; k < lanes; ++k) {
            most = max(most, most_of[threadIdx.x + k * padded]);
            sum += exponents_of[threadIdx.x + k * padded];
            number += count_of[threadIdx.x + k * padded];
        }
        part_max[blockIdx.x * kMaxColumns + threadIdx.x] = most;
        part_sum[blockIdx.x * kMaxColumns + threadIdx.x] = make_ulonglong2(sum, number);
    }
    // beside digit_words_kernel in a call that makes its words: what waits for this kernel waits for that one too
    wait_for_previous_launch();
}

constexpr int kPackThreads = 1024; // one block per SM: each adds the parts up for itself

// W -> per (block of NB columns, window of 128 genes) a record of four pieces of 32 genes, each the 4 NB x 64 digits in the no-swizzle K-major operand layout (byte of (column k NB + c: digit k of column c, the
// highest first; K = 2 gene + {0: the code's operand, 1: the constant's}) = column / 8 * 512 + K / 16 * 128 + column % 8 * 16 +
// K % 16).  Zeroes past the last gene and column.
template<typename WT, int NB>
__global__ void __launch_bounds__(kPackThreads) pack_w_digits_kernel(const WT *w, std::int64_t ld, int n, int padded, std::int64_t genes, int windows, meta_source meta,
                                                                     const unsigned *part_max, const ulonglong2 *part_sum, double *steps, unsigned char *records, int *wide) {
    __shared__ unsigned most_of[kPackThreads];
    __shared__ ulonglong2 sum_of[kPackThreads];
    __shared__ double factor[kMaxColumns];
    const int tid = threadIdx.x, block = static_cast<int>(blockIdx.x), blocks = static_cast<int>(gridDim.x);
    wait_for_previous_launch();
    let_next_launch_start();
    {
        const int c = tid % padded, lanes = kPackThreads / padded;
        unsigned most = 0u;
        ulonglong2 sum = make_ulonglong2(0u, 0u);
        for (int k0 = tid / padded; k0 < kParts; k0 += 3 * lanes) { // lanes 4, 8, 16, 32
            unsigned m[3];
            ulonglong2 q[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                m[k] = __ldcg(part_max + (k0 + k * lanes) * kMaxColumns + c);
                q[k] = __ldcg(part_sum + (k0 + k * lanes) * kMaxColumns + c);
            }
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                most = max(most, m[k]);
                sum.x += q[k].x;
                sum.y += q[k].y;
            }
        }
        most_of[tid] = most;
        sum_of[tid] = sum;
        __syncthreads();
        int too_wide = 0;
        if (tid < padded) {
            for (int k = 1; k < lanes; ++k) {
                most = max(most, most_of[tid + k * padded]);
                sum.x += sum_of[tid + k * padded].x;
                sum.y += sum_of[tid + k * padded].y;
            }
            double f = 0.0, step = 0.0;
            if (most >= 0x7f800000u) {
                too_wide = 1;
            } else if (most != 0u) {
                // largest = m 2^e, m in [0.5, 1); the largest number of four balanced digits is 0.996 * 2^31
                const int e = most >= 0x800000u ? static_cast<int>(most >> 23) - 126 : 32 - __clz(most) - 149;
                const int k = 8 * kSlices - 1 - e - ((most & 0x7fffffu) > 8100000u || most < 0x800000u ? 1 : 0);
                f = __longlong_as_double(static_cast<long long>(1023 + k) << 52);
                step = __longlong_as_double(static_cast<long long>(1023 - k) << 52);
                too_wide = (most >> 23) * sum.y > sum.x + kMostSpread * sum.y ? 1 : 0;
            }
            factor[tid] = f;
            if (block == 0) steps[tid] = step;
        }
        too_wide = __syncthreads_or(too_wide);
        if (block == 0 && tid == 0) *wide = too_wide;
        if (too_wide != 0) return;
    }
    constexpr int NC = mma_columns(NB), kItems = NB * 4; // of a piece: eight genes of a column
    const int items = (n + NB - 1) / NB * windows * kWPieces * kItems;
    for (int i = block * kPackThreads + tid; i < items; i += blocks * kPackThreads) {
        const int b = i / kItems, item = i % kItems, c0 = b / (windows * kWPieces) * NB, c = item % NB, g8 = item / NB;
        const std::int64_t gene0 = static_cast<std::int64_t>(b % (windows * kWPieces)) * 32 + g8 * 8;
        unsigned char *rec = records + static_cast<std::size_t>(b) * (64 * NC);
        const bool real = c0 + c < n;
        const double f = real ? factor[c0 + c] : 0.0;
        std::uint32_t digit[kSlices][4];
#pragma unroll
        for (int k = 0; k < kSlices; ++k)
#pragma unroll
            for (int j = 0; j < 4; ++j) digit[k][j] = 0u;
        float v[8];
        float2 so[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            v[j] = real && gene0 + j < genes ? load1(w + (gene0 + j) * ld + c0 + c) : 0.0f;
            so[j] = gene0 + j < genes ? meta.of(gene0 + j) : make_float2(0.0f, 0.0f);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const double scaled = static_cast<double>(v[j]) * f;
            int qc = __double2int_rn(static_cast<double>(so[j].x) * scaled);
            int qi = __double2int_rn(fma(static_cast<double>(so[j].y), scaled, static_cast<double>(meta.bias) * static_cast<double>(qc)) * (1.0 / 127.0));
#pragma unroll
            for (int k = kSlices - 1; k >= 0; --k) {
                digit[k][j >> 1] |= ((static_cast<std::uint32_t>(qc) & 0xffu) | (static_cast<std::uint32_t>(qi) & 0xffu) << 8) << ((j & 1) * 16);
                qc = (qc - static_cast<int>(static_cast<signed char>(qc & 0xff))) >> 8;
                qi = (qi - static_cast<int>(static_cast<signed char>(qi & 0xff))) >> 8;
            }
        }
#pragma unroll
        for (int k = 0; k < kSlices; ++k) {
            const int column = k * NB + c;
            *reinterpret_cast<uint4 *>(rec + (column >> 3) * 512 + g8 * 128 + (column & 7) * 16) = make_uint4(digit[k][0], digit[k][1], digit[k][2], digit[k][3]);
        }
    }
}

// ---- the sums --------------------------------------------------------------------------------------------------------------

struct fwd_digit_params {
    const std::uint32_t *words;
    const std::uint32_t *bounds;
    const std::int64_t *bases;
    std::int64_t pieces;
    int group_pieces, piece_rows;
    const std::int64_t *row_ptr, *packed_row_ptr; // for rows that are done entry by entry, these and ...
    const std::int32_t *col_idx;
    const std::uint8_t *packed;
    meta_source meta;
    const void *w;
    std::int64_t w_ld;
    int w_bf16;
    const unsigned char *records;
    const double *steps;
    const int *wide;
    long long *slots;     // [2 CTA + (0: its first group, 1: its last)][NB][row]
    float *out;
    std::int64_t out_ld;
    std::int64_t row_begin, row_end, cols;
    std::int64_t first_row; // of the first group
    int first_group;        // of the launch, among those of the words
    int groups, windows, column_blocks, n, bits;
    float alpha, beta;
    const float *bias;
    int epilogue, out_vector;
    int *status;
    int poll_limit;       // test hook (cb200_test_arm_wait_timeout): the loader of W issues no copies and gives up after so many polls; 0: none
};

// Tiles (column block, group, window), numbered in this order, are dealt to the CTAs in equal contiguous shares.
__host__ __device__ __forceinline__ std::int64_t share_begin(std::int64_t total, int cta, int ctas) { return total * cta / ctas; }

// K-major operand, no swizzle (a piece of W): core matrices of 8 columns x 16 bytes; the next 16 bytes of K 128 bytes on, the next
// 8 columns 512.
__device__ __forceinline__ std::uint64_t smem_desc_w(std::uint32_t addr) {
    std::uint64_t d = 0;
    d |= static_cast<std::uint64_t>((addr & 0x3ffffu) >> 4);
    d |= static_cast<std::uint64_t>(128u >> 4) << 16;
    d |= static_cast<std::uint64_t>(512u >> 4) << 32;
    d |= static_cast<std::uint64_t>(1) << 46; // descriptor version of this architecture
    return d;
}

// One output element from its exact sum.
__device__ __forceinline__ float sum_to_output(long long sum, double step, const fwd_digit_params &p) { return p.alpha * static_cast<float>(static_cast<double>(sum) * step); }

// Eight consecutive columns of a row.
__device__ __forceinline__ void write_columns(const fwd_digit_params &p, std::int64_t row, int c0, float (&v)[8]) {
    float *dst = p.out + row * p.out_ld + c0;
    if (p.out_vector != 0 && c0 + 8 <= p.n) {
        if (p.beta != 0.0f) {
            const float4 a = *reinterpret_cast<const float4 *>(dst), b = *reinterpret_cast<const float4 *>(dst + 4);
            v[0] = fmaf(p.beta, a.x, v[0]); v[1] = fmaf(p.beta, a.y, v[1]); v[2] = fmaf(p.beta, a.z, v[2]); v[3] = fmaf(p.beta, a.w, v[3]);
            v[4] = fmaf(p.beta, b.x, v[4]); v[5] = fmaf(p.beta, b.y, v[5]); v[6] = fmaf(p.beta, b.z, v[6]); v[7] = fmaf(p.beta, b.w, v[7]);
        }
        if (p.epilogue != CB200_EPILOGUE_NONE) {
#pragma unroll
            for (int c = 0; c < 8; ++c) v[c] = finish_output(v[c], p.bias, c0 + c, p.epilogue);
        }
        *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
        *reinterpret_cast<float4 *>(dst + 4) = make_float4(v[4], v[5], v[6], v[7]);
        return;
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        if (c0 + c >= p.n) break;
        if (p.beta != 0.0f) v[c] = fmaf(p.beta, dst[c], v[c]);
        dst[c] = finish_output(v[c], p.bias, c0 + c, p.epilogue);
    }
}

// Whether the cells of the piece that holds cell r of a group are done entry by entry.
__device__ __forceinline__ bool cell_is_odd(const fwd_digit_params &p, int group, int r) {
    const std::int64_t at = static_cast<std::int64_t>(p.first_group + group) * p.group_pieces + r / p.piece_rows;
    return at < p.pieces && (__ldcg(p.bases + at) & kDigitWordsTwice) != 0;
}
__device__ __forceinline__ void put_sum(const fwd_digit_params &p, std::int64_t row, int c, double sum) {
    float v = p.alpha * static_cast<float>(sum);
    float *dst = p.out + row * p.out_ld + c;
    if (p.beta != 0.0f) v = fmaf(p.beta, *dst, v);
    *dst = finish_output(v, p.bias, c, p.epilogue);
}
// A warp's columns [c0, c0 + nb) of a row, entry by entry: 32 of them decoded at a time, two columns of 64 to a lane; fp32 FMAs over
// 32 entries, whose sums are added in double precision.
__device__ __noinline__ void row_by_entries(const fwd_digit_params &p, std::int64_t row, int c0, int nb, int lane) {
    const std::int64_t begin = __ldg(p.row_ptr + row), length = __ldg(p.row_ptr + row + 1) - begin;
    const std::uint8_t *codes = p.packed + (p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row) : begin);
    const int end = min(c0 + nb, p.n), ca = min(c0 + lane, end - 1), cb = min(c0 + 32 + lane, end - 1); // (lanes past the last column read it again)
    double sum_a = 0.0, sum_b = 0.0;
    for (std::int64_t e0 = 0; e0 < length; e0 += 32) {
        const std::int64_t i = e0 + lane;
        int gene = i < length ? __ldg(p.col_idx + begin + i) : -1;
        const std::uint32_t valid_of = __ballot_sync(0xffffffffu, gene >= 0 && gene < p.cols); // others, and those past the end, add nothing
        float value = 0.0f;
        if ((valid_of >> lane & 1u) != 0u) {
            unsigned code = __ldg(codes + (p.bits == 8 ? i : i >> 1));
            if (p.bits == 4) code = (i & 1) != 0 ? code >> 4 : code & 0xfu;
            const float2 so = p.meta.of(gene);
            value = fmaf(static_cast<float>(code), so.x, so.y);
        }
        float a = 0.0f, b = 0.0f;
        for (std::uint32_t left = valid_of; left != 0u; left &= left - 1u) {
            const int j = __ffs(left) - 1;
            const std::int64_t at = __shfl_sync(0xffffffffu, gene, j) * p.w_ld;
            const float v = __shfl_sync(0xffffffffu, value, j);
            a = fmaf(v, p.w_bf16 != 0 ? load1(static_cast<const __nv_bfloat16 *>(p.w) + at + ca) : load1(static_cast<const float *>(p.w) + at + ca), a);
            b = fmaf(v, p.w_bf16 != 0 ? load1(static_cast<const __nv_bfloat16 *>(p.w) + at + cb) : load1(static_cast<const float *>(p.w) + at + cb), b);
        }
        sum_a += static_cast<double>(a);
        sum_b += static_cast<double>(b);
    }
    if (c0 + lane < end) put_sum(p, row, c0 + lane, sum_a);
    if (c0 + 32 + lane < end) put_sum(p, row, c0 + 32 + lane, sum_b);
}

template<int NB>
__global__ void __launch_bounds__(kThreads, 1) qcsr_fwd_digits_kernel(const __grid_constant__ fwd_digit_params p) {
    constexpr int NC = mma_columns(NB), WPIECE = w_piece_bytes(NB), kPieces = ring_pieces(NB), kChunkEntries = chunk_entries(NB), kChunkBytes = kChunkEntries * 4;
    constexpr int kTmem = 2 * NC;
    constexpr std::uint32_t IDESC = instr_desc_i8(NC);
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *chunk_base = smem + 2 * kTileBytes + kPieces * WPIECE;
    std::uint64_t *a_full = reinterpret_cast<std::uint64_t *>(chunk_base + 2 * kChunkBytes); // [2] scatter warps -> MMA
    std::uint64_t *a_empty = a_full + 2;        // [2] MMA commit -> scatter warps
    std::uint64_t *c_full = a_empty + 2;        // [2] copy engine -> scatter warps (a chunk stage per scatter group)
    std::uint64_t *c_empty = c_full + 2;        // [2] scatter warps -> loader
    std::uint64_t *acc_full = c_empty + 2;      // MMA commit -> scatter warps
    std::uint64_t *acc_empty = acc_full + 1;    // scatter warps -> MMA
    std::uint64_t *mma_drain = acc_empty + 1;   // the MMA warp's own, used once, after an abort
    std::uint64_t *w_full = mma_drain + 1;      // [kPieces]
    std::uint64_t *w_empty = w_full + kPieces;  // [kPieces]
    volatile int *chunk_meta = reinterpret_cast<volatile int *>(w_empty + kPieces); // [2]
    std::uint32_t *tmem_slot = reinterpret_cast<std::uint32_t *>(const_cast<int *>(chunk_meta) + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *fills = reinterpret_cast<volatile int *>(tmem_slot + 2); // [3] of the ring of W and of the groups' chunk stages, once the loaders have ended
    unsigned char *scratch_slot = reinterpret_cast<unsigned char *>(tmem_slot + 5); // where padding words go

    const int tid = threadIdx.x, warp = warp_of_block(), lane = tid & 31;
    const std::uint32_t smem0 = smem_addr(smem), wring0 = smem0 + 2 * kTileBytes, chunk0 = wring0 + kPieces * WPIECE;
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            bar_init(smem_addr(a_full + b), kScatterWarps / 2);
            bar_init(smem_addr(a_empty + b), 1);
            bar_init(smem_addr(c_full + b), 1);
            bar_init(smem_addr(c_empty + b), kScatterWarps / 2);
        }
        for (int s = 0; s < kPieces; ++s) {
            bar_init(smem_addr(w_full + s), 1);
            bar_init(smem_addr(w_empty + s), 1);
        }
        bar_init(smem_addr(acc_full), 1);
        bar_init(smem_addr(acc_empty), kScatterWarps);
        bar_init(smem_addr(mma_drain), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(kTmem) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const std::uint32_t tmem_base = *tmem_slot;
    wait_for_previous_launch();

    const int ctas = static_cast<int>(gridDim.x);
    const std::int64_t total = static_cast<std::int64_t>(p.column_blocks) * p.groups * p.windows;
    const std::int64_t t0 = share_begin(total, blockIdx.x, ctas);
    const std::int64_t t1 = __ldcg(p.wide) != 0 ? t0 : share_begin(total, blockIdx.x + 1, ctas); // too wide: the gather kernel's work

    if (warp < kScatterWarps) {
        // ================= zero, scatter, read back =================
        const int grp = warp / (kScatterWarps / 2), gtid = tid - grp * kGroupThreads;
        unsigned char *tile = smem + grp * kTileBytes;
        const std::uint32_t chunk_full = smem_addr(c_full + grp), chunk_empty = smem_addr(c_empty + grp);
        const uint4 *chunk = reinterpret_cast<const uint4 *>(chunk_base + grp * kChunkBytes);
        const auto scatter = [&](std::uint32_t e) {
            unsigned char *dst = static_cast<int>(e) >= 0 ? tile + ((e >> 8) & 0x7fffu) * 2u : scratch_slot;
            *reinterpret_cast<unsigned short *>(dst) = static_cast<unsigned short>((e & 0xffu) | 0x7f00u);
        };
        // The sums of a run, [w0, w1) of a line, once its MMAs have ended.  TMEM lane = row of the half; a warp reads the lane quarter its
        // number allows: NB / 2 columns of one half.
        int run = 0;
        const auto put_together = [&](std::int64_t line, bool whole) {
            const int group = static_cast<int>(line % p.groups), c0 = static_cast<int>(line / p.groups) * NB;
            const std::int64_t first_row = p.first_row + static_cast<std::int64_t>(group) * kRows;
            const std::int64_t slot = 2 * static_cast<std::int64_t>(blockIdx.x) + (line != t0 / p.windows ? 1 : 0);
            bar_wait(smem_addr(acc_full), static_cast<std::uint32_t>(run & 1), abort_flag);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int quarter = warp & 3, half = (warp >> 2) & 1, part = (warp >> 3) * (NB / 2), r = half * 128 + quarter * 32 + lane;
            const bool write = whole && first_row + r >= p.row_begin && first_row + r < p.row_end && !cell_is_odd(p, group, r);
#pragma unroll 1
            for (int h = 0; h < NB / 2; h += 8) {
                long long sum[8];
#pragma unroll
                for (int k = 0; k < kSlices; ++k) {
                    int d[8];
                    tmem_ld8(tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16) + half * NC + k * NB + part + h, d);
#pragma unroll
                    for (int c = 0; c < 8; ++c) sum[c] = k == 0 ? d[c] : sum[c] * 256 + d[c];
                }
                if (*abort_flag != 0) continue;
                if (!whole) {
                    long long *dst = p.slots + (slot * NB + part + h) * kRows + r; // column after column: a store is 256 bytes in one place
#pragma unroll
                    for (int c = 0; c < 8; ++c) dst[c * kRows] = sum[c];
                } else if (write && c0 + part + h < p.n) {
                    float v[8];
#pragma unroll
                    for (int c = 0; c < 8; ++c) v[c] = sum_to_output(sum[c], __ldg(p.steps + c0 + part + h + c), p);
                    write_columns(p, first_row + r, c0 + part + h, v);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(smem_addr(acc_empty));
            ++run;
            if (whole && cell_is_odd(p, group, warp * 16)) // a warp does sixteen cells
                for (int k = 0; k < 16; ++k) {
                    const std::int64_t row = first_row + warp * 16 + k;
                    if (row >= p.row_begin && row < p.row_end) row_by_entries(p, row, c0, NB, lane);
                }
        };
        // A run's sums are read once the group has filled a tile of a later run, so that the MMAs of that have a tile to start with.
        std::uint32_t q = 0, qc = 0; // this group's tiles and chunks
        std::int64_t drained = t0;   // first tile of the run to be read next
        const auto end_of = [&](std::int64_t t) { return min((t / p.windows + 1) * p.windows, t1); };
        const auto drain = [&]() {
            const std::int64_t end = end_of(drained);
            put_together(drained / p.windows, drained % p.windows == 0 && end - drained == p.windows);
            drained = end;
        };
        std::int64_t drained_end = t0 < t1 ? end_of(t0) : t1;
        for (std::int64_t t = t0 + grp; t < t1; t += 2, ++q) {
            // the tile's first chunk goes into registers while the MMAs still read the group's previous tile
            bar_wait(chunk_full, qc & 1u, abort_flag);
            const int meta = chunk_meta[grp];
            const int n_entries = *abort_flag != 0 ? 0 : meta >> 1;
            bool last = (meta & 1) != 0 || *abort_flag != 0;
            uint4 held[kChunkEntries / (kGroupThreads * 4)];
            std::uint32_t all = 0;
#pragma unroll
            for (int k = 0; k < kChunkEntries / (kGroupThreads * 4); ++k) {
                const int i = (k * kGroupThreads + gtid) * 4;
                held[k] = i < n_entries ? chunk[i >> 2] : make_uint4(kPadding, kPadding, kPadding, kPadding);
                all |= held[k].x | held[k].y | held[k].z | held[k].w;
            }
            arrive_when_loaded(chunk_empty, all, lane, static_cast<std::uint32_t>(p.windows) >> 31);
            ++qc;
            bar_wait(smem_addr(a_empty + grp), (q & 1u) ^ 1u, abort_flag);
#pragma unroll
            for (int k = 0; k < kTileBytes / (kGroupThreads * 8); ++k) // 8-byte stores: fewer wavefronts of the LSU data pipe per byte than 16-byte ones
                *reinterpret_cast<uint2 *>(tile + k * (kGroupThreads * 8) + gtid * 8) = make_uint2(0u, 0u);
            if (grp == 0) asm volatile("bar.sync 2, %0;" ::"n"(kGroupThreads) : "memory");
            else asm volatile("bar.sync 3, %0;" ::"n"(kGroupThreads) : "memory");
#pragma unroll
            for (int k = 0; k < kChunkEntries / (kGroupThreads * 4); ++k) {
                scatter(held[k].x); scatter(held[k].y); scatter(held[k].z); scatter(held[k].w);
            }
            int guard = 0;
            while (!last && ++guard < (1 << 20)) {
                bar_wait(chunk_full, qc & 1u, abort_flag);
                const int more = chunk_meta[grp];
                const int n_more = *abort_flag != 0 ? 0 : more >> 1;
                last = (more & 1) != 0 || *abort_flag != 0;
                for (int i = gtid * 4; i < n_more; i += kGroupThreads * 4) {
                    const uint4 e = chunk[i >> 2];
                    scatter(e.x); scatter(e.y); scatter(e.z); scatter(e.w);
                }
                __syncwarp();
                if (lane == 0) bar_arrive(chunk_empty);
                ++qc;
            }
            fence_async_proxy(); // ordinary stores, read by the MMA through the async proxy
            __syncwarp();
            if (lane == 0) bar_arrive(smem_addr(a_full + grp));
            while (drained_end <= t) {
                drain();
                drained_end = end_of(drained);
            }
        }
        while (drained < t1) drain();
    } else if (warp == kScatterWarps) {
        // ================= MMA issuer: one thread, which does the waiting too =================
        if (elect_one()) {
            std::uint32_t q = 0, phase = 0;
            int s = 0, run = 0;
            for (std::int64_t t = t0; t < t1; ++run) {
                const std::int64_t te = min((t / p.windows + 1) * p.windows, t1);
                bar_wait(smem_addr(acc_empty), static_cast<std::uint32_t>((run & 1) ^ 1), abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (bool first = true; t < te; ++t, ++q, first = false) {
                    const std::uint32_t b = q & 1u;
                    bar_wait(smem_addr(a_full + b), (q >> 1) & 1u, abort_flag);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                    for (int piece = 0; piece < kWPieces; ++piece) {
                        bar_wait(smem_addr(w_full + s), phase, abort_flag);
                        const std::uint32_t a = smem0 + b * kTileBytes + (piece >> 1) * kHalfBytes + (piece & 1) * 64, w_piece = wring0 + s * WPIECE;
#pragma unroll
                        for (int kk = 0; kk < 2; ++kk) {
                            mma_i8(tmem_base, smem_desc_sw128(a + kk * 32), smem_desc_w(w_piece + kk * 256), IDESC, !first || piece > 0 || kk > 0);
                            mma_i8(tmem_base + NC, smem_desc_sw128(a + kHalfBytes / 2 + kk * 32), smem_desc_w(w_piece + kk * 256), IDESC, !first || piece > 0 || kk > 0);
                        }
                        mma_commit(smem_addr(w_empty + s));
                        if (++s == kPieces) { s = 0; phase ^= 1u; }
                    }
                    mma_commit(smem_addr(a_empty + b));
                }
                mma_commit(smem_addr(acc_full));
            }
        }
    } else if (warp == kScatterWarps + 2) {
        // ================= the ring of W =================
        if (elect_one()) {
            int s = 0, issued = 0, window = static_cast<int>(t0 % p.windows);
            std::uint32_t ph = 1;
            std::int64_t line = t0 / p.windows;
            const unsigned char *block = p.records + line / p.groups * p.windows * (kWPieces * static_cast<std::int64_t>(WPIECE)); // of the column block
            bool dead = p.poll_limit != 0 && bar_wait(smem_addr(w_full), 0u, abort_flag, p.poll_limit);
            for (std::int64_t t = t0; t < t1 && !dead; ++t) {
                const unsigned char *src = block + static_cast<std::int64_t>(window) * (kWPieces * WPIECE);
                if (++window == p.windows) {
                    window = 0;
                    ++line;
                    block = p.records + line / p.groups * p.windows * (kWPieces * static_cast<std::int64_t>(WPIECE));
                }
                for (int piece = 0; piece < kWPieces; ++piece, src += WPIECE) {
                    dead = bar_wait(smem_addr(w_empty + s), ph, abort_flag);
                    if (dead) break; // no new copies once a wait of the CTA has run out
                    ++issued;
                    bar_arrive_expect_tx(smem_addr(w_full + s), WPIECE);
                    bulk_copy_g2s(wring0 + s * WPIECE, src, WPIECE, smem_addr(w_full + s));
                    if (++s == kPieces) { s = 0; ph ^= 1u; }
                }
            }
            fills[0] = issued;
        }
    } else {
        // ================= the words: a warp per scatter group; a tile's lie in the group's eight or sixteen pieces, a lane each =================
        const int ring = warp == kScatterWarps + 1 ? 0 : 1;
        const std::uint32_t full = smem_addr(c_full + ring), empty = smem_addr(c_empty + ring), dst = chunk0 + ring * kChunkBytes;
        std::int64_t t = t0 + ring;
        int window = static_cast<int>(t % p.windows), group = static_cast<int>(t / p.windows % p.groups);
        // the bounds of the next tile's words are on their way while this one's are copied
        std::uint32_t lo = 0, hi = 0;
        std::int64_t base = 0;
        const auto fetch = [&]() {
            lo = hi = 0u;
            const std::int64_t piece = static_cast<std::int64_t>(p.first_group + group) * p.group_pieces + lane;
            if (t < t1 && lane < p.group_pieces && piece < p.pieces) {
                const std::uint32_t *bound = p.bounds + piece * (p.windows + 1) + window;
                lo = __ldcg(bound);
                hi = __ldcg(bound + 1);
                base = __ldcg(p.bases + piece) & (kDigitWordsTwice - 1);
            }
        };
        fetch();
        int done = 0; // chunks issued
        bool dead = false;
        while (t < t1 && !dead) {
            const int words = static_cast<int>(hi - lo);
            const std::uint32_t *src = p.words + base + lo;
            t += 2;
            for (window += 2; window >= p.windows; window -= p.windows)
                if (++group == p.groups) group = 0;
            fetch();
            int upto = words;
#pragma unroll
            for (int d = 1; d < kMostGroupPieces; d <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += below;
            }
            const int begin = upto - words, total_words = __shfl_sync(0xffffffffu, upto, kMostGroupPieces - 1);
            int c0 = 0;
            do {
                const int n = min(kChunkEntries, total_words - c0);
                dead = __any_sync(0xffffffffu, bar_wait(empty, static_cast<std::uint32_t>((done & 1) ^ 1), abort_flag));
                if (dead) break; // no new copies once a wait of the CTA has run out
                if (lane == 0) {
                    chunk_meta[ring] = (n << 1) | (c0 + n >= total_words ? 1 : 0);
                    if (n > 0) bar_arrive_expect_tx(full, static_cast<std::uint32_t>(n) * 4u);
                    else bar_arrive(full); // a tile without entries still hands over one (empty) chunk
                }
                __syncwarp();
                const int first = max(begin, c0), end = min(begin + words, c0 + n);
                if (first < end)
                    bulk_copy_g2s(dst + (first - c0) * 4, src + (first - begin), static_cast<std::uint32_t>(end - first) * 4u, full);
                __syncwarp();
                ++done;
                c0 += n;
            } while (c0 < total_words);
        }
        if (lane == 0) fills[1 + ring] = done;
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag != 0) { // every role has ended: what is in flight finishes before the CTA gives up its shared and tensor memory
        if (warp == kScatterWarps) {
            if (elect_one()) drain_mmas(smem_addr(mma_drain));
        } else if (warp == kScatterWarps + 2) {
            if (elect_one()) drain_fills(smem_addr(w_full), kPieces, fills[0]);
        } else if (warp > kScatterWarps && lane == 0) {
            const int ring = warp == kScatterWarps + 1 ? 0 : 1;
            drain_fills(smem_addr(c_full + ring), 1, fills[1 + ring]);
        }
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmem) : "memory");
    }
    if (tid == 0 && *abort_flag != 0) atomicExch(p.status, 1);
}

template<int NB> constexpr std::size_t fwd_digits_smem_bytes() {
    return 2 * kTileBytes + ring_pieces(NB) * w_piece_bytes(NB) + 2 * chunk_entries(NB) * 4 + (11 + 2 * ring_pieces(NB)) * sizeof(std::uint64_t) + 32;
}

// The lines (column block, group) that lie in the shares of several CTAs, counted on the host: 64-bit divisions in every block of
// sum_parts_kernel cost it 1.9 M instructions.
constexpr int kSumColumns = 16; // of a block of sum_parts_kernel
struct cut_lines {
    int count;
    struct { int line; unsigned char first, last; bool second_slot; } at[kMaxCtas]; // the first and the last CTA; the first's slot for it
};

// Y of those lines.  Block (j, y, z): rows [32 y, 32 y + 32) and kSumColumns columns of the j-th; a warp for each eighth of the columns and a
// lane per row, whose sums change places in shared memory to be written a row's columns side by side.  Bound by the latency of the slots'
// loads, wave after wave of blocks: sixteen columns instead of eight take the whole call of 8,000 x 4,000, N = 64 from 66.2 to 63.6 us, of
// 8,192 x 33,538 from 172.5 to 169.9, of 20,000 x 2,000, N = 32 from 75.1 to 74.9 and of 4,099 x 33,538, N = 50 from 107.5 to 107.7; 32
// columns 64.7, 171.1, 77.6 and 109.0.
template<int NB>
__global__ void __launch_bounds__(256) sum_parts_kernel(const __grid_constant__ fwd_digit_params p, const __grid_constant__ cut_lines cuts) {
    constexpr int kColumns = kSumColumns;
    __shared__ float turned[32][kColumns + 1];
    const int line = cuts.at[blockIdx.x].line, b0 = cuts.at[blockIdx.x].first, b1 = cuts.at[blockIdx.x].last;
    const int group = line % p.groups, c0 = line / p.groups * NB, r0 = blockIdx.y * 32, column = blockIdx.z * kColumns;
    const std::int64_t first_row = p.first_row + static_cast<std::int64_t>(group) * kRows + r0;
    if (first_row >= p.row_end || first_row + 32 <= p.row_begin || c0 + column >= p.n) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    wait_for_previous_launch();
    const int wide = __ldcg(p.wide);
    const bool odd = cell_is_odd(p, group, r0 + lane);
    bool odd_row[kColumns / 8];
#pragma unroll
    for (int k = 0; k < kColumns / 8; ++k) odd_row[k] = cell_is_odd(p, group, r0 + tid / kColumns + k * (256 / kColumns));
    // only the group's first CTA can have another group before it: its slot may be the second of its two, the others' is the first
    const long long *src = p.slots + static_cast<std::int64_t>(column + warp) * kRows + r0 + lane;
    constexpr std::int64_t kSlot = static_cast<std::int64_t>(NB) * kRows;
    const std::int64_t first_slot = (2 * b0 + (cuts.at[blockIdx.x].second_slot ? 1 : 0)) * kSlot;
    double step[kColumns / 8];
    long long sum[kColumns / 8];
#pragma unroll
    for (int k = 0; k < kColumns / 8; ++k) {
        step[k] = __ldcg(p.steps + c0 + column + warp + 8 * k);
        sum[k] = __ldcg(src + first_slot + 8 * k * kRows);
    }
#pragma unroll 4
    for (int b = b0 + 1; b <= b1; ++b)
#pragma unroll
        for (int k = 0; k < kColumns / 8; ++k) sum[k] += __ldcg(src + 2 * b * kSlot + 8 * k * kRows);
    if (wide != 0) return;
#pragma unroll
    for (int k = 0; k < kColumns / 8; ++k) turned[lane][warp + 8 * k] = sum_to_output(sum[k], step[k], p);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kColumns / 8; ++k) {
        const int r = tid / kColumns + k * (256 / kColumns), c = c0 + column + tid % kColumns;
        const std::int64_t row = first_row + r;
        if (row >= p.row_begin && row < p.row_end && c < p.n && !odd_row[k]) {
            float *dst = p.out + row * p.out_ld + c;
            float v = turned[r][tid % kColumns];
            if (p.beta != 0.0f) v = fmaf(p.beta, *dst, v);
            *dst = finish_output(v, p.bias, c, p.epilogue);
        }
    }
    std::uint32_t left = blockIdx.z == 0 ? __ballot_sync(0xffffffffu, odd) : 0u;
    for (; left != 0u; left &= left - 1u) {
        const int k = __ffs(left) - 1;
        if (k % 8 == warp && first_row + k >= p.row_begin && first_row + k < p.row_end) row_by_entries(p, first_row + k, c0, NB, lane);
    }
}

int column_block(std::int64_t n) { return n <= 32 ? 32 : 64; }
int padded_columns(std::int64_t n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : 256; }
std::uint64_t record_bytes(std::int64_t cols, std::int64_t n) {
    const int nb = column_block(n);
    return device_arena::rounded(static_cast<std::uint64_t>((n + nb - 1) / nb * ((cols + kWin - 1) / kWin)) * kWPieces * static_cast<std::uint64_t>(w_piece_bytes(nb)));
}
std::uint64_t slot_bytes(std::int64_t n) { return static_cast<std::uint64_t>(2 * kMaxCtas) * kRows * static_cast<std::uint64_t>(column_block(n)) * 8u; }

template<typename WT, int NB>
cb200_status launch_all(const fwd_digit_params &p, unsigned *part_max, ulonglong2 *part_sum, double *steps, unsigned char *records, int *wide, bool early, int sm_count, cudaStream_t stream) {
    constexpr std::size_t smem = fwd_digits_smem_bytes<NB>();
    static_assert(smem <= 232448, "shared memory budget");
    const int padded = padded_columns(p.n);
    const WT *w = static_cast<const WT *>(p.w);
    CB200_CUDA_OK(launch_kernel(early, w_range_kernel<WT>, dim3(kParts), 1024, 0, stream, w, p.w_ld, p.n, padded, p.cols, p.meta, part_max, part_sum, early ? nullptr : p.status));
    const int pack_blocks = std::min((p.column_blocks * p.windows * kWPieces * NB * 4 + kPackThreads - 1) / kPackThreads, sm_count);
    CB200_CUDA_OK(launch_kernel(true, pack_w_digits_kernel<WT, NB>, dim3(static_cast<unsigned>(pack_blocks)), kPackThreads, 0, stream, w, p.w_ld, p.n, padded, p.cols, p.windows,
                                p.meta, part_max, part_sum, steps, records, wide));
    const std::int64_t total = static_cast<std::int64_t>(p.column_blocks) * p.groups * p.windows;
    const int ctas = static_cast<int>(std::min<std::int64_t>(total, sm_count));
    CB200_CUDA_OK(cudaFuncSetAttribute(qcsr_fwd_digits_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    CB200_CUDA_OK(launch_kernel(true, qcsr_fwd_digits_kernel<NB>, dim3(static_cast<unsigned>(ctas)), kThreads, smem, stream, p));
    cut_lines cuts{};
    for (int b = 0; b + 1 < ctas; ++b) { // the border behind CTA b
        const std::int64_t border = share_begin(total, b + 1, ctas), line = border / p.windows;
        if (border % p.windows == 0 || (cuts.count > 0 && cuts.at[cuts.count - 1].line == line)) {
            if (border % p.windows != 0) cuts.at[cuts.count - 1].last = static_cast<unsigned char>(b + 1);
            continue;
        }
        auto &cut = cuts.at[cuts.count++];
        cut.line = static_cast<int>(line);
        cut.first = static_cast<unsigned char>(b);
        cut.last = static_cast<unsigned char>(b + 1);
        cut.second_slot = share_begin(total, b, ctas) / p.windows != line;
    }
    if (cuts.count > 0) {
        CB200_CUDA_OK(launch_kernel(true, sum_parts_kernel<NB>, dim3(static_cast<unsigned>(cuts.count), kRows / 32, NB / kSumColumns), 256, 0, stream, p, cuts));
        count_launch();
    }
    count_launch(3);
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

} // namespace

bool qcsr_forward_digits_shape_ok(std::int64_t rows, std::int64_t cols, std::int64_t n, int bits, int policy) {
    return (bits == 8 || bits == 4) && policy == CB200_DECODE_PER_GENE_AFFINE && n > 0 && n <= kMaxColumns && rows > 0 && rows <= 0x7fffffff && cols > 0 && cols <= kMostGenes;
}
std::uint64_t qcsr_forward_digits_workspace_bytes(std::int64_t cols, std::int64_t n) { return kRecordsAt + record_bytes(cols, n) + slot_bytes(n); }

cb200_status launch_qcsr_forward_digits(const qcsr_view &x, const dense_args &d, std::int64_t row_begin, std::int64_t row_end, void *workspace,
                                        std::uint64_t workspace_bytes, const digit_layout *layout, int sm_count, cudaStream_t stream, const int **wide_word) {
    *wide_word = nullptr;
    const std::uint64_t own = qcsr_forward_digits_workspace_bytes(x.cols, d.n);
    if (!qcsr_forward_digits_shape_ok(x.rows, x.cols, d.n, x.bits, x.policy) || workspace == nullptr || reinterpret_cast<std::uintptr_t>(workspace) % 256u != 0u ||
        workspace_bytes < own + (layout == nullptr ? qcsr_digit_words_bytes_bound(x.rows, x.cols, x.nnz) : 0u) || sm_count > kMaxCtas ||
        (x.bits == 4 && x.packed_row_ptr == nullptr))
        return CB200_STATUS_SUCCESS;
    if (layout != nullptr && (x.row_ptr != layout->src_row_ptr || x.col_idx != layout->src_col_idx || x.packed != layout->src_packed))
        return fail(CB200_STATUS_STALE_STRUCTURE, "the launch's matrix is not the one the entry words were built from");
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    const int nb = column_block(d.n);
    fwd_digit_params p{};
    p.row_ptr = x.row_ptr; p.packed_row_ptr = x.packed_row_ptr; p.col_idx = x.col_idx; p.packed = x.packed;
    p.meta = meta_source{x.scales, x.offsets, x.bits == 8 ? 128.0f : 0.0f};
    p.w = d.dense; p.w_ld = d.dense_ld; p.w_bf16 = d.dense_dtype == CB200_DTYPE_BF16 ? 1 : 0;
    double *steps = reinterpret_cast<double *>(ws + kStepsAt);
    unsigned char *records = ws + kRecordsAt;
    int *wide = reinterpret_cast<int *>(ws) + 1;
    p.records = records; p.steps = steps; p.wide = wide;
    p.slots = reinterpret_cast<long long *>(records + record_bytes(x.cols, d.n));
    digit_layout words;
    std::int64_t words_row = 0, words_rows = x.rows; // the words' first row, and how many
    if (layout != nullptr) {
        words = *layout;
    } else {
        words = digit_words_at(ws + own, x);
        words_row = row_begin;
        words_rows = row_end - row_begin;
        const cb200_status st = launch_digit_words(x, row_begin, row_end, true, words.words, words.bounds, words.bases, reinterpret_cast<int *>(ws), stream);
        if (st != CB200_STATUS_SUCCESS) return st;
    }
    p.words = words.words; p.bounds = words.bounds; p.bases = words.bases;
    p.piece_rows = qcsr_digit_piece_rows(x.rows);
    p.group_pieces = kRows / p.piece_rows;
    p.pieces = (words_rows + p.piece_rows - 1) / p.piece_rows;
    p.out = d.out; p.out_ld = d.out_ld;
    p.row_begin = row_begin; p.row_end = row_end; p.cols = x.cols;
    p.first_group = static_cast<int>((row_begin - words_row) / kRows);
    p.first_row = words_row + static_cast<std::int64_t>(p.first_group) * kRows;
    p.groups = static_cast<int>((row_end - p.first_row + kRows - 1) / kRows);
    p.windows = static_cast<int>((x.cols + kWin - 1) / kWin);
    p.column_blocks = static_cast<int>((d.n + nb - 1) / nb);
    p.n = static_cast<int>(d.n); p.bits = x.bits;
    p.alpha = d.alpha; p.beta = d.beta; p.bias = d.bias; p.epilogue = d.epilogue;
    p.out_vector = reinterpret_cast<std::uintptr_t>(d.out) % 16u == 0u && d.out_ld % 4 == 0 ? 1 : 0;
    p.status = reinterpret_cast<int *>(ws);
    p.poll_limit = test_poll_limit();
    unsigned *part_max = reinterpret_cast<unsigned *>(ws + kPartMaxAt);
    ulonglong2 *part_sum = reinterpret_cast<ulonglong2 *>(ws + kPartSumAt);
    *wide_word = wide;
    if (d.dense_dtype == CB200_DTYPE_BF16)
        return nb == 64 ? launch_all<__nv_bfloat16, 64>(p, part_max, part_sum, steps, records, wide, layout == nullptr, sm_count, stream)
                        : launch_all<__nv_bfloat16, 32>(p, part_max, part_sum, steps, records, wide, layout == nullptr, sm_count, stream);
    return nb == 64 ? launch_all<float, 64>(p, part_max, part_sum, steps, records, wide, layout == nullptr, sm_count, stream)
                    : launch_all<float, 32>(p, part_max, part_sum, steps, records, wide, layout == nullptr, sm_count, stream);
}

} // namespace cb200
