// Gene-side transpose with exact integer sums on the tensor cores:
//     G'[genes, N] = alpha * deq(X)^T[genes, cells] * G[cells, N] + beta * G',   zero-points per gene.
//
// Reference counterpart: csr_spmm_bwd_rhs_kernel_ (src/compute/sparse/ops/kernels/base_sparse/csr_spmm_bwd_rhs_kernel_.cuh:1-22),
// one atomicAdd per (stored entry, output column).
//
// Formulation.  The stored value of (cell, gene) is scale * code + offset with scale and offset of the gene, so
//     G'[gene] = scale * (sum over cells of code * G[cell]) + offset * (sum over the gene's cells of G[cell]).
// Both sums have whole numbers on the matrix's side: the codes, and ones.  A column of G is written in fixed point, to 8 S - 1 bits below
// its largest magnitude, as S signed digits of base 256 (S = 4: rounded at 2^-31 of the largest; S = 3: at 2^-23).  Codes
// (less 128, to be signed) and digits are what the tensor cores' 8-bit integer MMAs multiply, and these add in 32 bits without
// rounding: every product and every sum up to the end of a run is exact, whatever their order.  The only errors are the rounding
// of G to its fixed point and a handful of fp32 roundings at the end: of each run, and of the sum of a set's runs, of which there are as many as
// CTAs share the set.  A request that has to be repeatable (EXACT) adds the runs up as whole numbers instead, 64 bits in L2, and rounds once:
// its bits follow from the operands and the row range alone, not from the number of SMs nor from the workspace, whose lack
// only cuts the launch into slices of groups and chunks of windows (100,003 x 33,538, N = 64: 1,099 us, with rounded runs 1,093).  Against
// 64 bits (2-norm, normal G, genes of the 33,538-gene matrices): S = 4 4e-8, where fp32 FMAs leave 1.2e-7 (8,191 cells) to 4.8e-7 (100,003
// cells, in a fixed order); S = 3 3e-7, where products put together from three bf16 products and summed by the fp32 MMAs leave 6.2e-6.
//
// Where G spreads too far for that (most_spread), the launch takes as many digits again, those behind the first ones, in a second pass over
// the tiles: 62 bits (S = 4) or 46; where three digits are asked for, four in one pass come first.  A G that spreads further still is taken entry
// by entry, in double precision and in a fixed order (beside_tiles).  Infinities and NaNs are zeroes in the digits; the last kernel finds the
// entries of their cells and what they make of these genes' sums.  The device decides; nothing is read back.
//
// Data.  The entries lie in pieces of 32 cells; inside a piece they are ordered by window of 128 genes, one word per entry
// {code, place in the operand tile}, cell after cell (digit_words_kernel: a CTA per piece counts the entries of each cell and window in
// shared memory, adds them up, and places the words; no atomics between CTAs, the same words on every run).
// A prepared operation keeps the words; a call that sees its matrix once makes them in its workspace.
//
// Structure of the main kernel (640 threads, one CTA per SM): warps 0-15 in two groups of eight on alternate tiles zero a tile
// of 256 cells x 128 genes (32 KB of codes, 32 KB of ones, K-major with the 128-byte swizzle) and scatter its words; warp 16
// issues the MMAs (M = genes, K = cells, N = S digits x the columns of G); warp 18 feeds the ring of G; warps 17 and 19 the
// words, each to one of the groups.  The two sums of a window take 2 S N columns of tensor memory, all 512 at S = 4, N = 64, and stay there while
// the CTA walks the groups of its run.  Every wait is bounded (sm100_primitives.cuh); if one runs out, the status word is set and the last kernel
// adds the entries up by itself, ten to fifty times slower: the callers of a call without a handle cannot ask for the status.
//
// What bounds it: at S = 4, N = 64 the tensor pipe, sixteen 128 x 256 x 32 MMAs of 128 cycles in the 2,410 cycles of a tile; at S = 3
// the scatter groups' chain (release, zeroes, two one-byte stores a word, fence, hand-over), 2,125 cycles against 1,536 of MMAs; over a
// second of launches the power cap (1.6 GHz).  One B200, start of this kernel's life -> now: 125,000 x 33,538, N = 64, S = 3 1,645 (bf16
// products) -> 1,170 us; 100,003 cells, S = 4 2,879 (rows of G gathered gene by gene) -> 1,096; 8,191 cells, S = 4 with the words made in
// the call 313 (sorted in shared memory) -> 175.  With one row of G at 1e6: 1,511 -> 2,090, 2,641 -> 1,970, 313 -> 258; Student-t numbers with
// three degrees of freedom (four digits in one pass instead of three in two, 2,014 us): 125,000 cells, S = 3 1,204.
#include "dependent_launch.cuh"
#include "kernels.cuh"
#include "sm100_primitives.cuh"

#include <algorithm>
#include <math_constants.h>

namespace cb200 {

namespace {

// Thirty-two cells to a piece, or sixteen where those would leave SMs without a CTA to lay them out (4,099 x 33,538: 49 us and 38; 8,191
// rows, two CTAs to most SMs: 65 and 70).
int piece_rows_of(std::int64_t rows) { return rows >= 32 * 148 ? 32 : 16; }

constexpr int kWin = 128;                       // genes per window
constexpr int kRows = 256;                      // cells per group
constexpr int kPieceRows = 32;                  // most cells whose words one CTA lays out
constexpr int kBuildThreads = 768;
constexpr int kBuildWarps = kBuildThreads / 32;
constexpr std::uint32_t kPadding = 0x80000000u; // a word that holds no entry
constexpr std::uint32_t kAgain = 0xc0000000u;   // added to a word whose place in the tile another entry has: a gene that its cell holds already

constexpr int kMostGroupPieces = kRows / 16;
constexpr int kProducerWarps = 16;
constexpr int kProducerThreads = kProducerWarps * 32;
constexpr int kGroupThreads = kProducerThreads / 2;
constexpr int kThreads = kProducerThreads + 4 * 32;
constexpr int kPlaneBytes = kWin * kRows;       // 32 KB: [cell half][gene][128 cells], a byte each
constexpr int kTileBytes = 2 * kPlaneBytes;     // codes, then ones
constexpr int kGPieceRows = 64;                 // G comes in pieces of 64 cells, four per group
constexpr int kGPieces = kRows / kGPieceRows;
constexpr int kChunkEntries = 2048;
constexpr int kChunkBytes = kChunkEntries * 4;
constexpr int kMaxCtas = 256;
// |code - 128| <= 128 and |digit| <= 128: 2^31 / 2^14 cells until a sum could leave 32 bits
constexpr std::int64_t kRunGroups = (1 << 17) / kRows - 1;

// digits x columns of one MMA, windows whose sums fit in tensor memory, pieces in the ring of G
__host__ __device__ constexpr int mma_columns(int nb, int slices) { return nb * slices; }
__host__ __device__ constexpr int set_windows(int nb, int slices) { return 512 / (2 * mma_columns(nb, slices)); }
__host__ __device__ constexpr int g_piece_bytes(int nb, int slices) { return kGPieceRows * mma_columns(nb, slices); }
__host__ __device__ constexpr int ring_pieces(int nb, int slices) { return mma_columns(nb, slices) >= 256 ? 5 : mma_columns(nb, slices) >= 192 ? 6 : 8; }

// workspace: status block {status, mode, ...}, steps of the columns, what is known of G's columns in parts (largest magnitudes; sums of
// 1 / sqrt(magnitude) and numbers; smallest row maxima), G in digits, sums of the runs or totals, and for a call that sees its matrix
// once the words
constexpr int kParts = 48;
constexpr int kMaxColumns = 256;
constexpr int kBlockColumns = 16; // columns whose largest number stands for a cell's
// How far G may spread, in binary orders, for a launch of `slices` digits and `passes`: the numbers are rounded at half a step, 2^-(8 slices - 1) to
// 2^-(8 slices) of their column's largest, which has to stay below what the products of the kernel this one replaces were rounded
// at: 2^-24 (fp32; a base of 4 digits) or 2.8e-6, root mean square, of a product put together from bf16 pieces (a base of 3).
//
// The spread is the larger of two numbers.  (1) A cell's largest number of sixteen neighbouring columns, against the largest of these columns:
// the smallest of them over all cells and columns.  A gene that only such cells hold has its result in these columns to the precision of
// fp32 products.  An average over a column does not see them where they are few: 10 % of the cells at 2^-20 move the average exponent by 2.
// (2) For a column by itself, where a cell's others are large: the square of the mean of sqrt(largest / number), halved; numbers at 2^-s of the
// largest raise it from 2^(2 log2 of their share + s) on.  Normal numbers have 3 and 3 (100,000 cells).  20,000 cells, a gene held by 800 cells at 2^-k alone,
// error against 64 bits of 32-bit FMAs or hi / lo products -> this (one pass whatever the spread): k = 7, S = 4 2.5e-8 -> 1e-9 (6e-9);
// k = 20, S = 4 3e-8 -> 1e-9 (4e-5); k = 4, S = 3 2.3e-7 -> 2e-9 (2e-7); k = 20, S = 3 2.3e-7 -> 1e-8 (1e-2).
__host__ __device__ constexpr int most_spread(int base, int slices, int passes) {
    return 8 * slices - (base == 4 ? 24 : 19) + (passes == 2 ? 8 * slices - 1 : 0);
}
// The launch's mode, a word in the workspace that its first kernels write: digits, passes over the tiles, or entry by entry; whether there are
// words with kAgain; whether G holds infinities or NaNs.
constexpr int kByEntry = 1 << 8, kRepeats = 1 << 9, kNonFinite = 1 << 10;
__host__ __device__ constexpr int mode_of(int slices, int passes) { return slices << 4 | passes; }
__host__ __device__ constexpr int slices_of(int mode) { return mode >> 4 & 15; }
__host__ __device__ constexpr int passes_of(int mode) { return mode & 15; }
constexpr int kMostSlices = 4;

constexpr std::uint64_t kStepsAt = 256, kPartMaxAt = kStepsAt + 2 * kMaxColumns * 8, kPartSumAt = kPartMaxAt + kParts * kMaxColumns * 4,
                        kPartLeastAt = kPartSumAt + kParts * kMaxColumns * 16, kRecordsAt = kPartLeastAt + kParts * (kMaxColumns / kBlockColumns) * 4;
static_assert(kParts % 48 == 0, "six at a time on up to eight lanes");
static_assert(kRecordsAt % 256 == 0, "G's records are copied 16 bytes at a time");

// A call that sees its matrix once and holds more entries adds them in shared memory (qcsr_transpose_tiled.cu), in 32 MB of workspace:
// the words of this many take 200 MB.
constexpr std::int64_t kMostOnceEntries = 50'000'000, kLeastOnceEntries = 2'000'000;

// ---- the words -----------------------------------------------------------------------------------------------------------

struct words_params {
    const std::int64_t *row_ptr;
    const std::int64_t *packed_row_ptr;
    const std::int32_t *col_idx;
    const std::uint8_t *packed;
    std::int64_t row_begin, row_end, cols;
    int windows, code_bias, piece_rows;
    std::uint32_t *words;
    std::uint32_t *bounds; // [pieces][windows + 1], from the piece's base
    std::int64_t *bases;   // [pieces]; kTwice: a cell of the piece holds a gene more than once
    int *status;           // cleared, where given
    int *outside;          // CHECK: set if a gene lies outside the matrix; such entries have no word
};
constexpr std::int64_t kTwice = kDigitWordsTwice;

// A CTA's cells are one stretch of the CSR arrays, which its warps take 256 entries at a time whatever cells they belong to (rows
// are of very different lengths: a warp per row took 240 us for 8,191 x 33,538 with 14.7 M entries, this takes 59).  Where genes ascend,
// an entry starts a window if the one before it lies in another; from those starts follow the sizes, the places of the windows and
// so the place of every entry, without an atomic, which the second pass computes from a look-up per entry.  A CTA that finds a gene
// outside the matrix or not above the one before it counts and places entry by entry with atomics instead, and marks the genes that a cell
// holds already (kAgain): a tile has one place for them, and finish_kernel adds the others.
//
// What bounds it: the latency of the genes' loads (eight in flight per warp, 48 warps per SM) and issue, half of the slots.
// CHECK: genes outside the matrix are reported (at prepare; in a call the test cost registers, 68 us instead of 66 for 8,191 cells).
template<int BITS, bool CHECK>
__global__ void __launch_bounds__(kBuildThreads, 2) digit_words_kernel(const words_params p) {
    extern __shared__ std::uint32_t place_of[]; // [kPieceRows][pitch]; see below.  Behind it [chunks][kPieceRows + 1] and [windows]
    __shared__ std::int64_t codes_of[kPieceRows]; // where the codes of a cell begin
    __shared__ int cell_start[kPieceRows + 1];    // from the CTA's first entry
    __shared__ std::uint32_t cell_bits[kPieceRows]; // of the words of a cell
    __shared__ std::uint32_t warp_sums[kBuildWarps];
    __shared__ std::uint32_t carry;
    __shared__ int irregular;
    constexpr std::uint32_t kNone = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_of_block(), pitch = p.windows | 1; // an odd pitch: a lane per cell reads without conflicts
    const std::int64_t row0 = p.row_begin + static_cast<std::int64_t>(blockIdx.x) * p.piece_rows;
    const int cells = static_cast<int>(min(static_cast<std::int64_t>(p.piece_rows), p.row_end - row0));
    let_next_launch_start();
    if (p.status != nullptr && blockIdx.x == 0 && tid == 0) *p.status = 0;
    const std::int64_t first = __ldg(p.row_ptr + row0);
    if (tid <= cells) {
        const std::int64_t at = __ldg(p.row_ptr + row0 + tid);
        cell_start[tid] = static_cast<int>(at - first);
        if (tid < cells) {
            const std::uint32_t cell = (blockIdx.x * p.piece_rows + tid) & (kRows - 1);
            codes_of[tid] = p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row0 + tid) : at;
            const std::uint32_t place = (cell >> 7) * (kPlaneBytes / 2) + ((cell & 127u) >> 4 << 4) + (cell & 15u); // plane half, 16-byte piece, byte
            cell_bits[tid] = place << 8 | static_cast<std::uint32_t>(p.code_bias);
        }
    }
    for (int i = tid; i < kPieceRows * pitch; i += kBuildThreads) place_of[i] = kNone;
    if (tid == 0) {
        carry = 0u;
        irregular = 0;
    }
    __syncthreads();
    const std::int32_t *genes = p.col_idx + first;
    const std::int64_t base = ((first - __ldg(p.row_ptr + p.row_begin) + 3) & ~static_cast<std::int64_t>(3)) + static_cast<std::int64_t>(blockIdx.x) * (4 * p.windows + 4);
    std::uint32_t *out = p.words + base;

    // A lane takes four neighbouring entries at a time, at places of the whole matrix that are multiples of four, so that they are one
    // load; a warp 128 kSteps of them.  e: the first of the four, from the CTA's first entry.
    const int end = cell_start[cells], skew = static_cast<int>(first & 3);
    const bool wide_loads = (reinterpret_cast<std::uintptr_t>(p.col_idx) & 15u) == 0u;
    const auto four_genes = [&](int e) {
        if (wide_loads && e + 3 < end) return __ldg(reinterpret_cast<const int4 *>(genes + e)); // (entries before the first are the cell's before)
        const auto at = [&](int k) { return e + k >= 0 && e + k < end ? __ldg(genes + e + k) : 0; };
        return make_int4(at(0), at(1), at(2), at(3));
    };
    struct { int r, begin, next; } in; // the cell of the lane's entry, and where it begins and ends
    const auto find = [&](int e) { // last cell that begins at or before e and is not empty
        int lo = 0, hi = cells - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (cell_start[mid] <= e) lo = mid;
            else hi = mid - 1;
        }
        in = {lo, cell_start[lo], cell_start[lo + 1]};
    };
    const auto advance = [&](int e) {
        while (e >= in.next) in = {in.r + 1, in.next, cell_start[in.r + 2]};
    };

    // ---- the first entry of each (cell, window): place_of[cell][window] = its place among the cell's ----
    {
        constexpr int kSteps = 4;
        bool odd = false;
        for (int e0 = warp * (128 * kSteps) - skew; e0 < end; e0 += kBuildThreads * 4 * kSteps) {
            int4 four[kSteps];
#pragma unroll
            for (int u = 0; u < kSteps; ++u) four[u] = four_genes(min(e0 + u * 128 + lane * 4, end));
            int before = e0 > 0 ? __ldg(genes + e0 - 1) : 0; // of the warp's first entry
            find(max(e0 + lane * 4, 0));
#pragma unroll
            for (int u = 0; u < kSteps; ++u) {
                const int e = e0 + u * 128 + lane * 4;
                int last = __shfl_up_sync(0xffffffffu, four[u].w, 1);
                if (lane == 0) last = before;
                before = __shfl_sync(0xffffffffu, four[u].w, 31);
                const int gene[4] = {four[u].x, four[u].y, four[u].z, four[u].w};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (e + j >= 0 && e + j < end) {
                        advance(e + j);
                        if (e + j == in.begin) last = -1;
                        if (static_cast<unsigned>(gene[j]) >= static_cast<unsigned>(p.cols) || last >= gene[j]) odd = true;
                        else if (static_cast<unsigned>(last ^ gene[j]) >= kWin) place_of[in.r * pitch + (gene[j] >> 7)] = static_cast<std::uint32_t>(e + j - in.begin);
                    }
                    last = gene[j];
                }
            }
        }
        if (odd) irregular = 1;
    }
    __syncthreads();
    const bool ordered = irregular == 0;
    const auto each_entry = [&](auto &&f) { // f(cell, gene, place among the cell's)
        for (int r = warp; r < cells; r += kBuildWarps)
            for (int e = cell_start[r] + lane; e < cell_start[r + 1]; e += 32) {
                const int gene = __ldg(genes + e);
                if (static_cast<unsigned>(gene) < static_cast<unsigned>(p.cols)) f(r, gene, e - cell_start[r]);
                else if constexpr (CHECK) *p.outside = 1;
            }
    };
    const auto word_of = [&](std::uint32_t bits, int gene, std::uint32_t code) {
        // {code less the bias, place in the tile << 8}; the place: [plane half][gene][piece ^ gene % 8][byte]
        return bits ^ (static_cast<std::uint32_t>(gene & (kWin - 1)) << 15 | static_cast<std::uint32_t>(gene & 7) << 12) ^ code;
    };
    const auto code_at = [&](int r, int i) -> std::uint32_t {
        if constexpr (BITS == 8) return __ldg(p.packed + codes_of[r] + i);
        const std::uint32_t byte = __ldg(p.packed + codes_of[r] + (i >> 1));
        return (i & 1) != 0 ? byte >> 4 : byte & 0xfu;
    };
    const int chunks = (p.windows + 31) / 32;
    std::uint32_t *first_in = place_of + kPieceRows * pitch; // [chunk][cell]: the first entry of 32 windows
    std::uint32_t *start_of = first_in + chunks * (kPieceRows + 1);
    if (ordered) {
        // windows a cell has no entry in start where the next one does: inside 32 windows here, beyond them below
        const int shift = p.piece_rows == 32 ? 5 : 4;
#pragma unroll 2
        for (int item = warp; item < chunks << shift; item += kBuildWarps) {
            const int r = item & (p.piece_rows - 1), chunk = item >> shift, w = chunk * 32 + lane; // (rows past the last hold kNone)
            std::uint32_t v = w < p.windows ? place_of[r * pitch + w] : kNone;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) v = min(v, __shfl_down_sync(0xffffffffu, v, d)); // the lanes past the end give their own
            if (w < p.windows) place_of[r * pitch + w] = v;
            if (lane == 0) first_in[chunk * (kPieceRows + 1) + r] = v;
        }
    } else {
        for (int i = tid; i < kPieceRows * pitch; i += kBuildThreads) place_of[i] = 0u;
        __syncthreads();
        each_entry([&](int r, int gene, int) { atomicAdd(place_of + r * pitch + (gene >> 7), 1u); });
    }
    __syncthreads();
    // The places: window after window, inside a window cell after cell; a window's words are padded to a multiple of four.  A lane per
    // cell and a run of windows per warp, from the last to the first: place_of[cell][window] becomes, where genes ascend, what to add to
    // an entry's place in its cell, and otherwise the next free place, both from the window's first.
    const int share = (p.windows + kBuildWarps - 1) / kBuildWarps, w_first = warp * share, w_last = min(p.windows, w_first + share) - 1;
    {
        const bool mine = lane < cells;
        const std::uint32_t length = mine ? static_cast<std::uint32_t>(cell_start[lane + 1] - cell_start[lane]) : 0u;
        const auto beyond = [&](int chunk) { // the first entry behind the 32 windows of a chunk
            std::uint32_t v = length;
            for (int k = chunk + 1; k < chunks; ++k) v = min(v, first_in[k * (kPieceRows + 1) + lane]);
            return v;
        };
        std::uint32_t follow = length, up = length;
        if (ordered && w_first <= w_last && mine) {
            follow = beyond(w_last >> 5);
            if (w_last + 1 < p.windows) up = min(place_of[lane * pitch + w_last + 1], (w_last + 1) % 32 == 0 ? beyond((w_last + 1) >> 5) : follow);
        }
        __syncthreads(); // the window above the warp's has been read
#pragma unroll 4
        for (int w = w_last; w >= w_first; --w) {
            std::uint32_t v = mine ? place_of[lane * pitch + w] : 0u, entries = v;
            if (ordered) {
                if (w % 32 == 31 && mine) follow = w + 1 < p.windows ? up : length; // into the chunk before: what follows it is the window above
                v = mine ? min(v, follow) : 0u;
                entries = mine ? up - v : 0u;
                up = v;
            }
            std::uint32_t upto = entries;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const std::uint32_t below = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += below;
            }
            if (mine) place_of[lane * pitch + w] = upto - entries - (ordered ? v : 0u);
            if (lane == 31) start_of[w] = upto;
        }
    }
    __syncthreads();
    for (int w0 = 0; w0 < p.windows; w0 += kBuildThreads) {
        const int w = w0 + tid;
        const std::uint32_t total = w < p.windows ? start_of[w] : 0u, padded = (total + 3u) & ~3u;
        std::uint32_t upto = padded;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const std::uint32_t below = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= d) upto += below;
        }
        if (lane == 31) warp_sums[warp] = upto;
        __syncthreads();
        std::uint32_t before = lane < warp ? warp_sums[lane] : 0u;
        before = __reduce_add_sync(0xffffffffu, before);
        const std::uint32_t start = carry + before + upto - padded;
        __syncthreads();
        if (tid == kBuildThreads - 1) carry = start + padded;
        if (w < p.windows) {
            p.bounds[static_cast<std::int64_t>(blockIdx.x) * (p.windows + 1) + w] = start;
            start_of[w] = start;
            for (std::uint32_t k = total; k < padded; ++k) out[start + k] = kPadding;
        }
        __syncthreads();
    }
    for (int w = w_first; w <= w_last; ++w)
        if (lane < cells) place_of[lane * pitch + w] += start_of[w];
    __syncthreads();
    if (tid == 0) {
        p.bounds[static_cast<std::int64_t>(blockIdx.x) * (p.windows + 1) + p.windows] = carry;
        p.bases[blockIdx.x] = base;
    }
    if (!ordered) {
        __shared__ std::uint32_t seen_of[kBuildWarps][kWin]; // a window's (gene, cell)
        each_entry([&](int r, int gene, int i) { out[atomicAdd(place_of + r * pitch + (gene >> 7), 1u)] = word_of(cell_bits[r], gene, code_at(r, i)); });
        __syncthreads();
        std::uint32_t *seen = seen_of[warp];
        bool twice = false;
        const std::uint32_t *bounds = p.bounds + static_cast<std::int64_t>(blockIdx.x) * (p.windows + 1);
        for (int w = warp; w < p.windows; w += kBuildWarps) {
            for (int i = lane; i < kWin; i += 32) seen[i] = 0u;
            __syncwarp();
            for (std::uint32_t i = bounds[w] + lane; i < bounds[w + 1]; i += 32) {
                const std::uint32_t e = out[i];
                if (static_cast<int>(e) < 0) continue;
                const std::uint32_t place = e >> 8;
                const std::uint32_t gl = (place >> 7) & (kWin - 1), cell = (((place >> 4 ^ gl) & 7u) << 4 | (place & 15u)) & (kPieceRows - 1);
                if ((atomicOr(seen + gl, 1u << cell) >> cell & 1u) != 0u) {
                    twice = true;
                    out[i] = e | kAgain;
                }
            }
            __syncwarp();
        }
        if (__syncthreads_or(twice ? 1 : 0) != 0 && tid == 0) p.bases[blockIdx.x] = base | kTwice;
        return;
    }
    // Here a warp takes 256 entries of one cell: neighbouring entries of a window go to neighbouring words, so a store of 32 of them touches
    // six or seven places (four entries to a lane, as above, spread a store over four times as many: 54 us against 38).
    constexpr int kSteps = 8;
    const int my_begin = cell_start[min(lane, cells)], my_length = lane < cells ? cell_start[lane + 1] - my_begin : 0;
    const int my_pieces = (my_length + 32 * kSteps - 1) / (32 * kSteps);
    int my_first = my_pieces;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, my_first, d);
        if (lane >= d) my_first += below;
    }
    const int items = __shfl_sync(0xffffffffu, my_first, 31);
    my_first -= my_pieces;
    for (int item = warp; item < items; item += kBuildWarps) {
        const int r = 31 - __clz(__ballot_sync(0xffffffffu, my_first <= item));
        const int begin = __shfl_sync(0xffffffffu, my_begin, r), at = (item - __shfl_sync(0xffffffffu, my_first, r)) * (32 * kSteps);
        const int left = __shfl_sync(0xffffffffu, my_length, r) - at; // of the cell, from here on
        const std::int32_t *from = genes + begin + at + lane;
        const std::uint8_t *codes = p.packed + codes_of[r] + (BITS == 8 ? at + lane : (at + lane) >> 1); // (`at` is even)
        const std::uint32_t *mine = place_of + r * pitch;
        const std::uint32_t bits = cell_bits[r];
        std::uint32_t *dst = out + at + lane; // place_of is what to add to an entry's place in its cell: it can be negative
        int gene[kSteps];
        std::uint32_t code[kSteps];
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            const bool valid = u * 32 + lane < left;
            gene[u] = valid ? __ldg(from + u * 32) : 0;
            code[u] = valid ? __ldg(codes + (BITS == 8 ? u * 32 : u * 16)) : 0u;
        }
#pragma unroll
        for (int u = 0; u < kSteps; ++u) {
            if (u * 32 + lane >= left) break;
            std::uint32_t c = code[u];
            if constexpr (BITS == 4) c = (lane & 1) != 0 ? c >> 4 : c & 0xfu;
            dst[static_cast<std::int32_t>(mine[gene[u] >> 7]) + u * 32] = word_of(bits, gene[u], c);
        }
    }
}

// ---- G in digits -----------------------------------------------------------------------------------------------------------

// Of each column the largest finite magnitude (as bits; the top bit: there is an infinity or a NaN too) and, over the finite numbers that are not zero, the sum of 1 /
// sqrt(magnitude) and their number; of each sixteen columns (the last sixteen for a rest of them) the smallest row maximum that is not
// zero, as bits; in kParts parts.  HBM or L2.
__global__ void __launch_bounds__(1024) column_range_kernel(const float *g, std::int64_t ld, int n, int padded, std::int64_t row_begin, std::int64_t row_end,
                                                            unsigned *part_max, double2 *part_sum, unsigned *part_least, int *status) {
    __shared__ unsigned most_of[1024], least_of[1024], count_of[1024];
    __shared__ float inverse_of[1024];
    let_next_launch_start();
    if (status != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *status = 0;
    const int c = threadIdx.x % padded, lanes = 1024 / padded;
    // behind the last column of its sixteen a lane has one of the sixteen before
    const int from = c < n ? c : c / kBlockColumns * kBlockColumns < n && c >= kBlockColumns ? c - kBlockColumns : -1;
    unsigned most = 0u, count = 0u, least = 0xffffffffu, odd = 0u;
    float inverse = 0.0f;
    const std::int64_t step = static_cast<std::int64_t>(gridDim.x) * lanes;
    std::int64_t r = row_begin + static_cast<std::int64_t>(blockIdx.x) * lanes + threadIdx.x / padded; // the same in a warp
    const float *at = g + r * ld + from;
    const auto take = [&](float v) {
        unsigned bits = __float_as_uint(v) & 0x7fffffffu;
        if (bits >= 0x7f800000u) {
            odd |= c < n ? 0x80000000u : 0u;
            bits = 0u;
        }
        if (c < n) {
            most = max(most, bits);
            if (bits != 0u) {
                inverse += rsqrtf(fabsf(v));
                ++count;
            }
        }
        return bits;
    };
    float v[8]; // the next eight rows are on their way while eight are looked at
    const auto load = [&]() {
#pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = from >= 0 ? __ldg(at + k * step * ld) : 0.0f;
    };
    bool eight = r + 7 * step < row_end;
    if (eight) load();
    while (eight) {
        unsigned m[8];
        float now[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) now[k] = v[k];
        r += 8 * step;
        at += 8 * step * ld;
        eight = r + 7 * step < row_end;
        if (eight) load();
#pragma unroll
        for (int k = 0; k < 8; ++k) m[k] = take(now[k]);
        // eight rows over sixteen lanes: half of the rows stay with half of the lanes, three times, and two lanes have a row's halves
#pragma unroll
        for (int d = 4; d > 0; d >>= 1) {
            const bool upper = (threadIdx.x & d) != 0u;
#pragma unroll
            for (int k = 0; k < d; ++k) {
                const unsigned mine = upper ? m[k + d] : m[k], theirs = upper ? m[k] : m[k + d];
                m[k] = max(mine, __shfl_xor_sync(0xffffffffu, theirs, d));
            }
        }
        m[0] = max(m[0], __shfl_xor_sync(0xffffffffu, m[0], 8));
        if (m[0] != 0u) least = min(least, m[0]);
    }
    for (; r < row_end; r += step, at += step * ld) {
        unsigned m = take(from >= 0 ? __ldg(at) : 0.0f);
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
        if (m != 0u) least = min(least, m);
    }
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) least = min(least, __shfl_xor_sync(0xffffffffu, least, d));
    most_of[threadIdx.x] = most | odd;
    least_of[threadIdx.x] = least;
    count_of[threadIdx.x] = count;
    inverse_of[threadIdx.x] = inverse;
    __syncthreads();
    if (threadIdx.x < static_cast<unsigned>(padded)) {
        double sum = static_cast<double>(inverse), number = static_cast<double>(count);
        for (int k = 1; k < lanes; ++k) {
            odd |= most_of[threadIdx.x + k * padded] & 0x80000000u;
            most = max(most, most_of[threadIdx.x + k * padded] & 0x7fffffffu);
            least = min(least, least_of[threadIdx.x + k * padded]);
            sum += static_cast<double>(inverse_of[threadIdx.x + k * padded]);
            number += static_cast<double>(count_of[threadIdx.x + k * padded]);
        }
        part_max[blockIdx.x * kMaxColumns + threadIdx.x] = most | odd;
        part_sum[blockIdx.x * kMaxColumns + threadIdx.x] = make_double2(sum, number);
        if (threadIdx.x % kBlockColumns == 0u) part_least[(blockIdx.x * kMaxColumns + threadIdx.x) / kBlockColumns] = least;
    }
    // beside digit_words_kernel in a call that makes its words: what waits for this kernel waits for that one too
    wait_for_previous_launch();
}

// G -> per (pass, block of NB columns, group of 256 cells) a record of four pieces of 64 cells, each the S NB x 64 digits in the no-swizzle
// K-major operand layout (byte of (column k NB + c: digit k of column c, the highest first; cell r) = column / 8 * 512 + r / 16 *
// 128 + column % 8 * 16 + r % 16).  Cells outside [row_begin, row_end) and columns from n on are zero.
struct pack_params {
    const float *g;
    std::int64_t ld, first_row, row_begin, row_end, groups; // first_row: of the groups; row_begin, row_end: of the launch
    int n, padded;
    const unsigned *part_max;
    const double2 *part_sum;
    const unsigned *part_least;
    double *steps;
    unsigned char *records;
    const std::int64_t *bases;
    std::int64_t word_pieces;
    int *mode;
    uint4 *totals;            // the totals to clear, 16 bytes each, of one pass
    std::int64_t total_items;
    unsigned short *odd_rows; // [16 cells][32 columns]: which of the cells have an infinity or a NaN there; written if there is one at all
};
// the second pass takes up what the first rounds off, at most half a step
__host__ __device__ constexpr double second_step(int slices) { return 1.0 / static_cast<double>(1ull << (8 * slices - 1)); }

__host__ __device__ constexpr int odd_chunks(int n) { return n <= 32 ? 1 : (n + 63) / 64 * 2; } // of 32 columns, in blocks of NB

// factor: 2^k, what a column is multiplied by
template<int NB, int SLICES>
__device__ __forceinline__ void pack_records(const pack_params &p, int mode, const double *factor) {
    constexpr int NC = mma_columns(NB, SLICES);
    const int tid = threadIdx.x, passes = passes_of(mode);
    const std::int64_t pieces = static_cast<std::int64_t>((p.n + NB - 1) / NB) * p.groups * kGPieces;
    for (std::int64_t b = blockIdx.x; b < passes * pieces; b += gridDim.x) {
        const bool second = b >= pieces;
        const int c0 = static_cast<int>((second ? b - pieces : b) / (p.groups * kGPieces)) * NB;
        const std::int64_t row0 = p.first_row + b % (p.groups * kGPieces) * kGPieceRows;
        unsigned char *rec = p.records + b * (kGPieceRows * NC);
        for (int item = tid; item < NB * (kGPieceRows / 16); item += 256) {
            const int c = item % NB, r16 = item / NB;
            const double f = c0 + c < p.n ? factor[c0 + c] : 0.0;
            float v[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const std::int64_t row = row0 + r16 * 16 + j;
                v[j] = row >= p.row_begin && row < p.row_end && c0 + c < p.n ? __ldg(p.g + row * p.ld + c0 + c) : 0.0f;
            }
            if ((mode & kNonFinite) != 0) { // (a warp has 32 columns of sixteen cells)
                unsigned odd = 0u;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    if (isfinite(v[j])) continue;
                    odd |= 1u << j;
                    v[j] = 0.0f;
                }
                odd = __reduce_or_sync(0xffffffffu, odd);
                if (!second && (tid & 31) == 0)
                    p.odd_rows[(b % (p.groups * kGPieces) * (kGPieceRows / 16) + r16) * odd_chunks(p.n) + (c0 + c) / 32] = static_cast<unsigned short>(odd);
            }
            std::uint32_t digit[SLICES][4];
#pragma unroll
            for (int k = 0; k < SLICES; ++k)
#pragma unroll
                for (int w = 0; w < 4; ++w) digit[k][w] = 0u;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const double scaled = static_cast<double>(v[j]) * f;
                int q = __double2int_rn(scaled);
                if (second) q = __double2int_rn((scaled - static_cast<double>(q)) * (1.0 / second_step(SLICES)));
#pragma unroll
                for (int k = SLICES - 1; k >= 0; --k) {
                    digit[k][j >> 2] |= (static_cast<std::uint32_t>(q) & 0xffu) << ((j & 3) * 8);
                    q = (q - static_cast<int>(static_cast<signed char>(q & 0xff))) >> 8;
                }
            }
#pragma unroll
            for (int k = 0; k < SLICES; ++k) {
                const int column = k * NB + c;
                *reinterpret_cast<uint4 *>(rec + (column >> 3) * 512 + r16 * 128 + (column & 7) * 16) =
                    make_uint4(digit[k][0], digit[k][1], digit[k][2], digit[k][3]);
            }
        }
    }
}

// Every block adds the parts up for itself and so knows how the launch goes on; the first one writes the mode and the columns' steps.
template<int NB, int BASE>
__global__ void __launch_bounds__(256) pack_digits_kernel(const pack_params p) {
    __shared__ unsigned most_of[kMaxColumns], least_of[kMaxColumns / kBlockColumns];
    __shared__ double2 sum_of[256];
    __shared__ double factor[kMaxColumns];
    __shared__ unsigned long long need_bits; // 2^spread, whose bits have its order
    const int tid = threadIdx.x;
    if (tid < kMaxColumns / kBlockColumns) least_of[tid] = 0xffffffffu;
    if (tid == 0) need_bits = 0u;
    wait_for_previous_launch();
    let_next_launch_start();
    __syncthreads();
    int mode;
    {
        const int c = tid % p.padded, lanes = 256 / p.padded, blocks = p.padded / kBlockColumns;
        unsigned most = 0u, odd = 0u;
        double2 sum = make_double2(0.0, 0.0);
        for (int k0 = tid / p.padded; k0 < kParts; k0 += 6 * lanes) { // lanes 1, 2, 4, 8: six loads of each kind in flight
            unsigned m[6];
            double2 q[6];
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                m[k] = __ldcg(p.part_max + (k0 + k * lanes) * kMaxColumns + c);
                q[k] = __ldcg(p.part_sum + (k0 + k * lanes) * kMaxColumns + c);
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                odd |= m[k] & 0x80000000u;
                most = max(most, m[k] & 0x7fffffffu);
                sum.x += q[k].x;
                sum.y += q[k].y;
            }
        }
        for (int i = tid; i < kParts * blocks; i += 256) atomicMin(least_of + i % blocks, __ldcg(p.part_least + i / blocks * (kMaxColumns / kBlockColumns) + i % blocks));
        most_of[tid] = most;
        sum_of[tid] = sum;
        __syncthreads();
        if (tid < p.padded) {
            for (int k = 1; k < lanes; ++k) {
                most = max(most, most_of[tid + k * p.padded]);
                sum.x += sum_of[tid + k * p.padded].x;
                sum.y += sum_of[tid + k * p.padded].y;
            }
            if (most != 0u) atomicMax(&need_bits, static_cast<unsigned long long>(__double_as_longlong(static_cast<double>(__uint_as_float(most)) * sum.x * sum.x / (2.0 * sum.y * sum.y))));
        }
        __syncthreads();
        if (tid < p.padded) most_of[tid] = most; // the columns'
        __syncthreads();
        if (tid < blocks && tid * kBlockColumns < p.n && least_of[tid] != 0xffffffffu) {
            unsigned largest = 0u;
            for (int k = max(0, min(tid * kBlockColumns, p.n - kBlockColumns)); k < min((tid + 1) * kBlockColumns, p.n); ++k) largest = max(largest, most_of[k]);
            atomicMax(&need_bits, static_cast<unsigned long long>(__double_as_longlong(static_cast<double>(__uint_as_float(largest)) / static_cast<double>(__uint_as_float(least_of[tid])))));
        }
        int repeats = 0;
        if (blockIdx.x == 0) {
#pragma unroll 8
            for (std::int64_t k = tid; k < p.word_pieces; k += 256) repeats |= (__ldcg(p.bases + k) & kTwice) != 0 ? 1 : 0;
        }
        const int non_finite = __syncthreads_or(odd != 0u ? 1 : 0);
        repeats = __syncthreads_or(repeats); // (the first block's: it writes the mode)
        const double need = __longlong_as_double(static_cast<long long>(need_bits));
        const auto serves = [&](int slices, int passes) { return need <= static_cast<double>(1ull << most_spread(BASE, slices, passes)); };
        mode = BASE == 3 && serves(3, 1) ? mode_of(3, 1) : serves(4, 1) ? mode_of(4, 1) : BASE == 3 && serves(3, 2) ? mode_of(3, 2) : mode_of(4, 2);
        if (!serves(4, 2)) mode |= kByEntry;
        if (non_finite != 0) mode |= kNonFinite;
        if (repeats != 0) mode |= kRepeats;
        if (tid < p.padded) {
            const int bits = 8 * slices_of(mode) - 1;
            double f = 0.0, step = 0.0;
            if (most != 0u) {
                // largest = m 2^e, m in [0.5, 1); the largest number of S balanced digits is 0.996 * 2^(8 S - 1)
                const int e = most >= 0x800000u ? static_cast<int>(most >> 23) - 126 : 32 - __clz(most) - 149;
                const int k = bits - e - ((most & 0x7fffffu) > 8220000u || most < 0x800000u ? 1 : 0);
                f = __longlong_as_double(static_cast<long long>(1023 + k) << 52);
                step = __longlong_as_double(static_cast<long long>(1023 - k) << 52);
            }
            factor[tid] = f;
            if (blockIdx.x == 0) {
                const int columns = (p.n + NB - 1) / NB * NB;
                if (tid < columns) p.steps[tid] = step;
                if (tid < columns) p.steps[columns + tid] = step * (slices_of(mode) == 3 ? second_step(3) : second_step(4)); // of the second pass
            }
        }
        if (blockIdx.x == 0 && tid == 0) *p.mode = mode;
        __syncthreads();
    }
    for (std::int64_t i = blockIdx.x * 256 + tid; i < passes_of(mode) * p.total_items; i += gridDim.x * 256) p.totals[i] = make_uint4(0u, 0u, 0u, 0u);
    if (BASE == 3 && slices_of(mode) == 3) pack_records<NB, 3>(p, mode, factor);
    else pack_records<NB, 4>(p, mode, factor);
}

// ---- the sums --------------------------------------------------------------------------------------------------------------

struct digit_params {
    const std::uint32_t *words;
    const std::uint32_t *bounds;
    const std::int64_t *bases;
    std::int64_t pieces;
    int group_pieces, piece_rows;
    const float *scales, *offsets;
    const unsigned char *records;
    const double *steps;
    const int *mode;
    float *partials;         // [run_of + CTA][window of the set][column][gene]: a run's sums, rounded
    long long *totals;       // EXACT: [set][window of the set][codes, ones][column][gene], which the runs add to
    std::int64_t cols;
    std::int64_t group_begin, group_count;
    std::int64_t first_set, set_count; // of the launch
    std::int64_t run_groups; // groups after which a run ends at the latest
    int windows, column_blocks, code_bias;
    int *status;
    int poll_limit;          // test hook (cb200_test_arm_wait_timeout): the loader of G issues no copies and gives up after so many polls; 0: none
};

// Units (column block, window set, group), numbered in this order, are dealt to the CTAs in equal contiguous shares; a run is a CTA's
// consecutive units of one set, cut every run_groups groups.  run_of numbers the runs of an undivided walk; the shares' borders cut them
// further, and run_of + CTA is a number no two runs have.
__host__ __device__ inline std::int64_t run_of(std::int64_t unit, std::int64_t groups, std::int64_t run_groups) {
    return unit / groups * ((groups + run_groups - 1) / run_groups) + unit % groups / run_groups;
}
__device__ __forceinline__ std::int64_t run_end(std::int64_t u, std::int64_t u1, std::int64_t groups, std::int64_t run_groups) {
    const std::int64_t gi = u % groups, last = min((gi / run_groups + 1) * run_groups, groups);
    return min(u + (last - gi), u1);
}
// the CTA whose share [total b / grid, total (b + 1) / grid) holds a unit
__device__ __forceinline__ std::int64_t cta_of(std::int64_t unit, std::int64_t total, std::int64_t grid) { return ((unit + 1) * grid - 1) / total; }
// A walk over the units' tiles, without a division a tile.
struct tile_cursor {
    std::int64_t unit;
    int group, set, wl, windows_of_set; // group: of the launch; set: of the column block
    const int groups, sets, windows, per_set; // windows: from the launch's first one on
    __device__ __forceinline__ int windows_in(int s) const { return min(per_set, windows - s * per_set); }
    __device__ __forceinline__ tile_cursor(const digit_params &p, std::int64_t sets_, std::int64_t first, int per_set_)
        : unit(first), group(static_cast<int>(first % p.group_count)), set(static_cast<int>(first / p.group_count % sets_)), wl(0), windows_of_set(0),
          groups(static_cast<int>(p.group_count)), sets(static_cast<int>(sets_)), windows(p.windows - static_cast<int>(p.first_set) * per_set_), per_set(per_set_) {
        windows_of_set = windows_in(set);
    }
    __device__ __forceinline__ void next() {
        if (++wl < windows_of_set) return;
        wl = 0;
        ++unit;
        if (++group < groups) return;
        group = 0;
        if (++set == sets) set = 0;
        windows_of_set = windows_in(set);
    }
};
// A gene's sum in one column.  A run's sums are below 2^56, totals below 2^63 (qcsr_transpose_exact_rows), so the whole numbers do not leave their 64
// bits: in double precision scale and offset may cancel to the last bits of fp32.
__device__ __forceinline__ double value_of(long long coded, long long present, int code_bias, double scale, double offset, double step) {
    return (scale * static_cast<double>(coded + code_bias * present) + offset * static_cast<double>(present)) * step;
}
// K-major operand, no swizzle (a piece of G): core matrices of 8 columns x 16 cells; the next 16 cells 128 bytes on, the next 8
// columns 512.
__device__ __forceinline__ std::uint64_t smem_desc_digits(std::uint32_t addr) {
    std::uint64_t d = 0;
    d |= static_cast<std::uint64_t>((addr & 0x3ffffu) >> 4);
    d |= static_cast<std::uint64_t>(128u >> 4) << 16;
    d |= static_cast<std::uint64_t>(static_cast<unsigned>(kGPieceRows * 8) >> 4) << 32;
    d |= static_cast<std::uint64_t>(1) << 46; // descriptor version of this architecture
    return d;
}

template<int NB, int SLICES, bool EXACT>
__device__ __forceinline__ void transpose_tiles(const digit_params &p) {
    constexpr int NC = mma_columns(NB, SLICES), kSet = set_windows(NB, SLICES), GPIECE = g_piece_bytes(NB, SLICES), kPieces = ring_pieces(NB, SLICES);
    constexpr std::uint32_t IDESC = instr_desc_i8(NC);
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char *chunk_base = smem + 2 * kTileBytes + kPieces * GPIECE;
    std::uint64_t *a_full = reinterpret_cast<std::uint64_t *>(chunk_base + 2 * kChunkBytes); // [2] scatter warps -> MMA
    std::uint64_t *a_empty = a_full + 2;           // [2] MMA commit -> scatter warps
    std::uint64_t *c_full = a_empty + 2;           // [2] copy engine -> scatter warps (a chunk stage per scatter group)
    std::uint64_t *c_empty = c_full + 2;           // [2] scatter warps -> loader
    std::uint64_t *acc_full = c_empty + 2;         // MMA commit -> scatter warps
    std::uint64_t *acc_empty = acc_full + 1;       // scatter warps -> MMA
    std::uint64_t *mma_drain = acc_empty + 1;      // the MMA warp's own, used once, after an abort
    std::uint64_t *g_full = mma_drain + 1;         // [kPieces]
    std::uint64_t *g_empty = g_full + kPieces;     // [kPieces]
    volatile int *chunk_meta = reinterpret_cast<volatile int *>(g_empty + kPieces); // [2]
    std::uint32_t *tmem_slot = reinterpret_cast<std::uint32_t *>(const_cast<int *>(chunk_meta) + 2);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *fills = reinterpret_cast<volatile int *>(tmem_slot + 2); // [3] of the ring of G and of the groups' chunk stages, once the loaders have ended
    unsigned char *scratch_slot = reinterpret_cast<unsigned char *>(tmem_slot + 5); // where padding words go

    const int tid = threadIdx.x, warp = warp_of_block(), lane = tid & 31;
    const std::uint32_t smem0 = smem_addr(smem), grec0 = smem0 + 2 * kTileBytes, chunk0 = grec0 + kPieces * GPIECE;
    if (tid == 0) {
        for (int b = 0; b < 2; ++b) {
            bar_init(smem_addr(a_full + b), kProducerWarps / 2);
            bar_init(smem_addr(a_empty + b), 1);
            bar_init(smem_addr(c_full + b), 1);
            bar_init(smem_addr(c_empty + b), kProducerWarps / 2);
        }
        for (int s = 0; s < kPieces; ++s) {
            bar_init(smem_addr(g_full + s), 1);
            bar_init(smem_addr(g_empty + s), 1);
        }
        bar_init(smem_addr(acc_full), 1);
        bar_init(smem_addr(acc_empty), kProducerWarps);
        bar_init(smem_addr(mma_drain), 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const std::uint32_t tmem_base = *tmem_slot;
    wait_for_previous_launch();

    const std::int64_t sets = p.set_count;
    const int mode = __ldcg(p.mode);
    // the second pass: as many column blocks again
    const std::int64_t total_units = sets * p.column_blocks * p.group_count * passes_of(mode);
    const std::int64_t u0 = total_units * blockIdx.x / gridDim.x;
    // entry by entry: nothing to do here, it is finish_kernel's work
    const std::int64_t u1 = (mode & kByEntry) != 0 ? u0 : total_units * (blockIdx.x + 1) / gridDim.x;

    if (warp < kProducerWarps) {
        // ================= zero, scatter, read back =================
        const int grp = warp / (kProducerWarps / 2), gtid = tid - grp * kGroupThreads;
        unsigned char *tile = smem + grp * kTileBytes;
        const std::uint32_t chunk_full = smem_addr(c_full + grp), chunk_empty = smem_addr(c_empty + grp);
        const uint4 *chunk = reinterpret_cast<const uint4 *>(chunk_base + grp * kChunkBytes);
        std::uint32_t q = 0, qc = 0; // this group's tiles and chunks
        int run = 0; // runs read back
        const auto scatter = [&](std::uint32_t e) {
            unsigned char *dst = static_cast<int>(e) >= 0 ? tile + ((e >> 8) & 0x7fffu) : scratch_slot;
            dst[0] = static_cast<unsigned char>(e);
            (static_cast<int>(e) >= 0 ? dst + kPlaneBytes : dst + 1)[0] = 1;
        };
        // End of a run: the digits' sums are put together.  TMEM lane = gene within the window; a warp reads the lane quarter its
        // number allows, sixteen columns of one window.  `from` is the run's first unit, `to` the one behind its last.
        const auto put_together = [&](std::int64_t from, std::int64_t to) {
            const std::int64_t set_of_all = from / p.group_count, set = set_of_all % sets;
            const int nwin = static_cast<int>(min(static_cast<std::int64_t>(kSet), p.windows - (p.first_set + set) * kSet));
            bar_wait(smem_addr(acc_full), static_cast<std::uint32_t>(run & 1), abort_flag);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int quarter = warp & 3, wl = NB == 64 ? 0 : warp >> 3, c0 = (NB == 64 ? warp >> 2 : (warp >> 2) & 1) * 16;
            const std::int64_t gene = ((p.first_set + set) * kSet + wl) * kWin + quarter * 32 + lane;
            if (wl < nwin) { // warp-uniform
                double scale = 0.0, offset = 0.0;
                if (!EXACT && gene < p.cols) {
                    scale = p.scales != nullptr ? static_cast<double>(__ldg(p.scales + gene)) : 1.0;
                    offset = p.offsets != nullptr ? static_cast<double>(__ldg(p.offsets + gene)) : 0.0;
                }
                const std::uint32_t at = tmem_base + (static_cast<std::uint32_t>(quarter * 32) << 16) + wl * 2 * NC + c0;
                float *slot = p.partials + (((run_of(to - 1, p.group_count, p.run_groups) + blockIdx.x) * kSet + wl) * NB + c0) * kWin + quarter * 32 + lane;
                unsigned long long *total = reinterpret_cast<unsigned long long *>(p.totals) + ((set_of_all * kSet + wl) * 2 * NB + c0) * kWin + quarter * 32 + lane;
                const double *steps = p.steps + set_of_all / sets * NB + c0;
#pragma unroll
                for (int h = 0; h < 16; h += 8) {
                    long long coded[8], present[8];
#pragma unroll
                    for (int k = 0; k < SLICES; ++k) {
                        int a[8], b[8];
                        tmem_ld8(at + k * NB + h, a);
                        tmem_ld8(at + NC + k * NB + h, b);
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            coded[c] = k == 0 ? a[c] : coded[c] * 256 + a[c];
                            present[c] = k == 0 ? b[c] : present[c] * 256 + b[c];
                        }
                    }
                    if (gene < p.cols && *abort_flag == 0) {
#pragma unroll
                        for (int c = 0; c < 8; ++c) {
                            if constexpr (EXACT) { // whole numbers: the same totals in whatever order and pieces
                                atomicAdd(total + (h + c) * kWin, static_cast<unsigned long long>(coded[c]));
                                atomicAdd(total + (NB + h + c) * kWin, static_cast<unsigned long long>(present[c]));
                            } else {
                                slot[(h + c) * kWin] = static_cast<float>(value_of(coded[c], present[c], p.code_bias, scale, offset, __ldg(steps + h + c)));
                            }
                        }
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) bar_arrive(smem_addr(acc_empty));
            ++run;
        };
        // A run's sums are read once the group has scattered a tile of a later run, so that the MMAs of that have a tile to start with.
        std::int64_t drained = u0, drained_end = u0 < u1 ? run_end(u0, u1, p.group_count, p.run_groups) : u1;
        tile_cursor at(p, sets, u0, kSet);
        if (grp != 0) at.next();
        while (at.unit < u1) {
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
            ++q;
            while (drained_end <= at.unit) {
                put_together(drained, drained_end);
                drained = drained_end;
                drained_end = run_end(drained, u1, p.group_count, p.run_groups);
            }
            at.next();
            at.next();
        }
        while (drained < u1) {
            put_together(drained, drained_end);
            drained = drained_end;
            if (drained < u1) drained_end = run_end(drained, u1, p.group_count, p.run_groups);
        }
    } else if (warp == kProducerWarps) {
        // ================= MMA issuer: one thread, which does the waiting too =================
        if (elect_one()) {
            std::uint32_t q = 0, phase = 0;
            int slot = 0, run = 0;
            for (std::int64_t u = u0; u < u1; ++run) {
                const std::int64_t ub = u, ue = run_end(u, u1, p.group_count, p.run_groups);
                const std::int64_t set = u / p.group_count % sets;
                const int nwin = static_cast<int>(min(static_cast<std::int64_t>(kSet), p.windows - (p.first_set + set) * kSet));
                bar_wait(smem_addr(acc_empty), static_cast<std::uint32_t>((run & 1) ^ 1), abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (; u < ue; ++u) {
                    int s = slot;
                    std::uint32_t ph = phase;
                    for (int wl = 0; wl < nwin; ++wl, ++q) {
                        const std::uint32_t b = q & 1u;
                        bar_wait(smem_addr(a_full + b), (q >> 1) & 1u, abort_flag);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        s = slot;
                        ph = phase;
#pragma unroll
                        for (int piece = 0; piece < kGPieces; ++piece) {
                            if (wl == 0) bar_wait(smem_addr(g_full + s), ph, abort_flag);
                            const std::uint32_t a = smem0 + b * kTileBytes + (piece >> 1) * (kPlaneBytes / 2) + (piece & 1) * 64, g_piece = grec0 + s * GPIECE;
                            const std::uint32_t d = tmem_base + wl * 2 * NC;
#pragma unroll
                            for (int kk = 0; kk < kGPieceRows / 32; ++kk) {
                                mma_i8(d, smem_desc_sw128(a + kk * 32), smem_desc_digits(g_piece + kk * 256), IDESC, u > ub || piece > 0 || kk > 0);
                                mma_i8(d + NC, smem_desc_sw128(a + kPlaneBytes + kk * 32), smem_desc_digits(g_piece + kk * 256), IDESC, u > ub || piece > 0 || kk > 0);
                            }
                            if (wl == nwin - 1) mma_commit(smem_addr(g_empty + s));
                            if (++s == kPieces) { s = 0; ph ^= 1u; }
                        }
                        mma_commit(smem_addr(a_empty + b));
                    }
                    slot = s;
                    phase = ph;
                }
                mma_commit(smem_addr(acc_full));
            }
        }
    } else if (warp == kProducerWarps + 2) {
        // ================= the ring of G =================
        if (elect_one()) {
            int s = 0, issued = 0;
            std::uint32_t ph = 1;
            bool dead = p.poll_limit != 0 && bar_wait(smem_addr(g_full), 0u, abort_flag, p.poll_limit);
            std::int64_t group = u0 % p.group_count, set_of_all = u0 / p.group_count;
            const unsigned char *block = p.records + set_of_all / sets * p.group_count * (kGPieces * GPIECE); // of the column block
            for (std::int64_t u = u0; u < u1 && !dead; ++u) {
                const unsigned char *src = block + group * (kGPieces * GPIECE);
                if (++group == p.group_count) {
                    group = 0;
                    block = p.records + ++set_of_all / sets * p.group_count * (kGPieces * GPIECE);
                }
                for (int piece = 0; piece < kGPieces; ++piece, src += GPIECE) {
                    dead = bar_wait(smem_addr(g_empty + s), ph, abort_flag);
                    if (dead) break; // no new copies once a wait of the CTA has run out
                    ++issued;
                    bar_arrive_expect_tx(smem_addr(g_full + s), GPIECE);
                    bulk_copy_g2s(grec0 + s * GPIECE, src, GPIECE, smem_addr(g_full + s));
                    if (++s == kPieces) { s = 0; ph ^= 1u; }
                }
            }
            fills[0] = issued;
        }
    } else {
        // ================= the words: a warp per scatter group; a tile's lie in the group's eight or sixteen pieces, a lane each =================
        const int ring = warp == kProducerWarps + 1 ? 0 : 1;
        const std::uint32_t full = smem_addr(c_full + ring), empty = smem_addr(c_empty + ring), dst = chunk0 + ring * kChunkBytes;
        tile_cursor at(p, sets, u0, kSet);
        if (ring != 0) at.next();
        // the bounds of the next tile's words are on their way while this one's are copied: 64-bit divisions and loads that were waited
        // for held this warp up for 2,450 cycles a tile, more than its MMAs take
        std::uint32_t lo = 0, hi = 0;
        std::int64_t base = 0;
        const auto fetch = [&]() {
            lo = hi = 0u;
            const std::int64_t piece = (p.group_begin + at.group) * p.group_pieces + lane;
            if (at.unit < u1 && lane < p.group_pieces && piece < p.pieces) {
                const std::uint32_t *bound = p.bounds + piece * (p.windows + 1) + (p.first_set + at.set) * kSet + at.wl;
                lo = __ldcg(bound);
                hi = __ldcg(bound + 1);
                base = __ldcg(p.bases + piece) & (kTwice - 1);
            }
        };
        fetch();
        int done = 0; // chunks issued
        bool dead = false;
        while (at.unit < u1 && !dead) {
            const int words = static_cast<int>(hi - lo);
            const std::uint32_t *src = p.words + base + lo;
            at.next();
            at.next();
            fetch();
            int upto = words;
#pragma unroll
            for (int d = 1; d < kMostGroupPieces; d <<= 1) {
                const int below = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= d) upto += below;
            }
            const int begin = upto - words, total = __shfl_sync(0xffffffffu, upto, kMostGroupPieces - 1);
            int c0 = 0;
            do {
                const int n = min(kChunkEntries, total - c0);
                dead = __any_sync(0xffffffffu, bar_wait(empty, static_cast<std::uint32_t>((done & 1) ^ 1), abort_flag));
                if (dead) break; // no new copies once a wait of the CTA has run out
                if (lane == 0) {
                    chunk_meta[ring] = (n << 1) | (c0 + n >= total ? 1 : 0);
                    if (n > 0) bar_arrive_expect_tx(full, static_cast<std::uint32_t>(n) * 4u);
                    else bar_arrive(full); // a tile without entries still hands over one (empty) chunk
                }
                __syncwarp();
                const int first = max(begin, c0), last = min(begin + words, c0 + n);
                if (first < last)
                    bulk_copy_g2s(dst + (first - c0) * 4, src + (first - begin), static_cast<std::uint32_t>(last - first) * 4u, full);
                __syncwarp();
                ++done;
                c0 += n;
            } while (c0 < total);
        }
        if (lane == 0) fills[1 + ring] = done;
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag != 0) { // every role has ended: what is in flight finishes before the CTA gives up its shared and tensor memory
        if (warp == kProducerWarps) {
            if (elect_one()) drain_mmas(smem_addr(mma_drain)); // by the thread that issued
        } else if (warp == kProducerWarps + 2) {
            if (elect_one()) drain_fills(smem_addr(g_full), kPieces, fills[0]);
        } else if (warp > kProducerWarps && lane == 0) {
            const int ring = warp == kProducerWarps + 1 ? 0 : 1;
            drain_fills(smem_addr(c_full + ring), 1, fills[1 + ring]);
        }
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
    if (tid == 0 && *abort_flag != 0) atomicExch(p.status, 1);
}

// A base of three digits: three or, where G spreads too far for them and not for four, four; the launches before have decided it.
template<int NB, int BASE, bool EXACT>
__global__ void __launch_bounds__(kThreads, 1) qcsr_transpose_digits_kernel(const digit_params p) {
    if constexpr (BASE == 3) {
        wait_for_previous_launch();
        if (slices_of(__ldcg(p.mode)) == 3) {
            transpose_tiles<NB, 3, EXACT>(p);
            return;
        }
    }
    transpose_tiles<NB, 4, EXACT>(p);
}

template<int NB, int SLICES> constexpr std::size_t digits_smem_bytes() {
    return 2 * kTileBytes + ring_pieces(NB, SLICES) * g_piece_bytes(NB, SLICES) + 2 * kChunkBytes + (11 + 2 * ring_pieces(NB, SLICES)) * sizeof(std::uint64_t) + 32;
}

struct finish_params {
    digit_params d;
    const float *g;
    std::int64_t g_ld, first_row, row_begin, row_end; // row_begin, row_end: of the launch; first_row: of the words
    const unsigned short *odd_rows; // from the first group of the call
    std::int64_t odd_from;          // its first row
    float *out;
    std::int64_t out_ld;
    std::int64_t grid; // CTAs of the main kernel
    int n, out_vector;
    float alpha, beta;
};

__host__ __device__ constexpr int finish_threads(int nb) { return nb / 16 * kWin; }
__host__ __device__ constexpr int finish_pitch(int nb) { return nb + 4; } // of a gene's results in shared memory: 16-byte stores of a warp's 32 genes meet no bank twice
constexpr int finish_smem_bytes(int nb) { return kWin * nb * 8 + std::max(kWin * (nb / 4) * 16, kWin * finish_pitch(nb) * 4); }
// f(word, gene within the window, row), a word of the window to a lane and 32 at a time, for the warp's share of the pieces of the row range that
// wanted(first row, base) lets through.  Lanes without a word of the range have kPadding.
template<typename W, typename F>
__device__ __forceinline__ void each_words(const finish_params &p, std::int64_t window, int share, int shares, W &&wanted, F &&f) {
    const int lane = threadIdx.x & 31;
    const std::int64_t piece1 = (p.row_end - p.first_row + p.d.piece_rows - 1) / p.d.piece_rows;
    for (std::int64_t piece = (p.row_begin - p.first_row) / p.d.piece_rows + share; piece < piece1; piece += shares) {
        const std::int64_t base = __ldcg(p.d.bases + piece);
        if (!wanted(p.first_row + piece * p.d.piece_rows, base)) continue;
        const std::uint32_t *at = p.d.bounds + piece * (p.d.windows + 1) + window;
        const int words = static_cast<int>(__ldcg(at + 1) - __ldcg(at));
        const std::uint32_t *w = p.d.words + (base & (kTwice - 1)) + __ldcg(at);
        const std::int64_t group_row = p.first_row + piece / p.d.group_pieces * kRows;
        for (int i0 = 0; i0 < words; i0 += 32) {
            const std::uint32_t e = i0 + lane < words ? __ldcg(w + i0 + lane) : kPadding;
            const int place = static_cast<int>((e >> 8) & 0x7fffu), gene = (place >> 7) & (kWin - 1);
            const std::int64_t row = group_row + (place >> 14) * 128 + ((((place >> 4) & 7) ^ (gene & 7)) << 4) + (place & 15);
            f(row >= p.row_begin && row < p.row_end ? e : kPadding, gene, row);
        }
    }
}

// What tiles do not hold, in values[gene][column].  by_entry: all of it, in double precision; a warp has every eighth or sixteenth gene to
// itself and takes the words in order, so that the bits are the same on every run.  Otherwise the genes that their cells hold already, in
// whole numbers (whole[gene][column of a quarter] {codes, ones}), and what infinities and NaNs of G come to (flags[gene][column]: 1, 2, 4 for
// a product of +infinity, of -infinity, or neither); the order of neither matters.
template<int NB>
__device__ __noinline__ void beside_tiles(const finish_params &p, int mode, bool by_entry, std::int64_t window, const float2 *meta, double *values,
                                          unsigned long long *whole) {
    constexpr int kFinish = finish_threads(NB), kWarps = kFinish / 32, kQuarter = NB / 4;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c0 = static_cast<int>(blockIdx.y) * NB;
    for (int i = tid; i < kWin * NB; i += kFinish) values[i] = 0.0;
    __syncthreads();
    if (by_entry) {
        each_words(p, window, 0, 1, [](std::int64_t, std::int64_t) { return true; }, [&](std::uint32_t e, int gene, std::int64_t row) {
            std::uint32_t todo = __ballot_sync(0xffffffffu, e != kPadding && gene % kWarps == warp);
            while (todo != 0u) {
                const int j = __ffs(todo) - 1;
                todo &= todo - 1u;
                const int code = static_cast<int>(static_cast<signed char>(__shfl_sync(0xffffffffu, e, j) & 0xffu)) + p.d.code_bias, gj = __shfl_sync(0xffffffffu, gene, j);
                const std::int64_t rj = __shfl_sync(0xffffffffu, row, j);
                const double value = static_cast<double>(fmaf(static_cast<float>(code), meta[gj].x, meta[gj].y));
                for (int c = lane; c < NB; c += 32)
                    if (c0 + c < p.n) values[gj * NB + c] += value * static_cast<double>(__ldg(p.g + rj * p.g_ld + c0 + c));
            }
        });
        __syncthreads();
        return;
    }
    if ((mode & kNonFinite) != 0) {
        static_assert(kWin * NB * sizeof(int) <= kWin * kQuarter * 16, "shares the memory");
        __shared__ unsigned settled[kWin / 32]; // genes whose sums are NaN in every column: nothing changes them any more
        int *flags = reinterpret_cast<int *>(whole);
        for (int i = tid; i < kWin * NB; i += kFinish) flags[i] = 0;
        if (tid < kWin / 32) settled[tid] = 0u;
        __syncthreads();
        const auto is_nan = [](int f) { return (f & 4) != 0 || (f & 3) == 3; };
        unsigned odd = 0u; // the piece's cells with an infinity or a NaN in these columns; most pieces have none
        const auto has_odd = [&](std::int64_t first, std::int64_t) {
            odd = 0u;
            for (int i = 0; i < p.d.piece_rows / 16; ++i) {
                const unsigned short *at = p.odd_rows + ((first - p.odd_from) / 16 + i) * odd_chunks(p.n) + c0 / 32;
                odd |= static_cast<unsigned>(__ldcg(at) | (NB > 32 ? __ldcg(at + 1) : 0)) << (16 * i);
            }
            return odd != 0u;
        };
        each_words(p, window, warp, kWarps, has_odd, [&](std::uint32_t e, int gene, std::int64_t row) {
            const bool mine = e != kPadding && (odd >> ((row - p.odd_from) & (p.d.piece_rows - 1)) & 1u) != 0u &&
                              (*const_cast<volatile unsigned *>(settled + gene / 32) >> (gene & 31) & 1u) == 0u;
            std::uint32_t todo = __ballot_sync(0xffffffffu, mine);
            while (todo != 0u) {
                const int j = __ffs(todo) - 1;
                todo &= todo - 1u;
                const int code = static_cast<int>(static_cast<signed char>(__shfl_sync(0xffffffffu, e, j) & 0xffu)) + p.d.code_bias, gj = __shfl_sync(0xffffffffu, gene, j);
                const std::int64_t rj = __shfl_sync(0xffffffffu, row, j);
                const float value = fmaf(static_cast<float>(code), meta[gj].x, meta[gj].y);
                bool all = true;
                for (int c = lane; c < NB && c0 + c < p.n; c += 32) {
                    const float g = __ldg(p.g + rj * p.g_ld + c0 + c), product = value * g;
                    const int flag = isfinite(g) ? 0 : isnan(product) ? 4 : product > 0.0f ? 1 : 2;
                    int had = *const_cast<volatile int *>(flags + gj * NB + c);
                    if ((flag & ~had) != 0) had = atomicOr(flags + gj * NB + c, flag) | flag;
                    all = all && is_nan(had);
                }
                if (__all_sync(0xffffffffu, all) && lane == 0) atomicOr(settled + gj / 32, 1u << (gj & 31));
            }
        });
        __syncthreads();
        for (int i = tid; i < kWin * NB; i += kFinish)
            if (flags[i] != 0) values[i] = is_nan(flags[i]) ? CUDART_NAN : flags[i] == 1 ? CUDART_INF : -CUDART_INF;
        __syncthreads();
    }
    if ((mode & kRepeats) == 0) return;
    const double rest = slices_of(mode) == 3 ? second_step(3) : second_step(4);
    for (int quarter = 0; quarter < 4; ++quarter)
        for (int pass = 0; pass < passes_of(mode); ++pass) {
            for (int i = tid; i < kWin * kQuarter * 2; i += kFinish) whole[i] = 0u;
            __syncthreads();
            each_words(p, window, warp, kWarps, [](std::int64_t, std::int64_t base) { return (base & kTwice) != 0; }, [&](std::uint32_t e, int gene, std::int64_t row) {
                std::uint32_t todo = __ballot_sync(0xffffffffu, e >= kAgain);
                while (todo != 0u) {
                    const int j = __ffs(todo) - 1;
                    todo &= todo - 1u;
                    const int code = static_cast<signed char>(__shfl_sync(0xffffffffu, e, j) & 0xffu), gj = __shfl_sync(0xffffffffu, gene, j);
                    const std::int64_t rj = __shfl_sync(0xffffffffu, row, j);
                    const int c = quarter * kQuarter + lane;
                    if (lane < kQuarter && c0 + c < p.n) {
                        const double step = __ldg(p.d.steps + c0 + c);
                        const float g = __ldg(p.g + rj * p.g_ld + c0 + c);
                        const double scaled = step != 0.0 && isfinite(g) ? static_cast<double>(g) / step : 0.0;
                        int q = __double2int_rn(scaled);
                        if (pass != 0) q = __double2int_rn((scaled - static_cast<double>(q)) / rest);
                        atomicAdd(whole + (gj * kQuarter + lane) * 2, static_cast<unsigned long long>(static_cast<long long>(code) * q));
                        atomicAdd(whole + (gj * kQuarter + lane) * 2 + 1, static_cast<unsigned long long>(static_cast<long long>(q)));
                    }
                }
            });
            __syncthreads();
            for (int i = tid; i < kWin * kQuarter; i += kFinish) {
                const int gene = i / kQuarter, c = quarter * kQuarter + i % kQuarter;
                values[gene * NB + c] += value_of(static_cast<long long>(whole[2 * i]), static_cast<long long>(whole[2 * i + 1]), p.d.code_bias, static_cast<double>(meta[gene].x),
                                                  static_cast<double>(meta[gene].y), __ldg(p.d.steps + pass * p.d.column_blocks * NB + c0 + c));
            }
            __syncthreads();
        }
}

// G'[genes of one window, columns of one block] = beta * G' + alpha * (the sums of the set's runs, added in run order; EXACT: the totals).
// What genes that a cell holds again (kAgain) and infinities and NaNs of G come to is added here.  Where G spreads too far for fixed point, or a scale or a zero-point of the window is not
// finite (0 * infinity, in a product of sums, would reach cells that hold no entry), or a wait of the main kernel ran out: everything, entry by entry
// (beside_tiles, which is no part of this function's registers: two CTAs of 512 threads to an SM, or the 262 of 33,538 genes take two rounds, 12
// us instead of 9).
// A thread has a gene and sixteen columns, so that a warp's loads are contiguous; the results change places in shared memory, so that
// its stores are too (10.6 us otherwise).
template<int NB, bool EXACT>
__global__ void __launch_bounds__(finish_threads(NB), 1024 / finish_threads(NB)) finish_kernel(const __grid_constant__ finish_params p) {
    extern __shared__ __align__(16) double beside[]; // [kWin][NB], and behind it [kWin][NB / 4] {codes, ones}, later the results
    constexpr int kSet = set_windows(NB, kMostSlices);
    static_assert(kSet == set_windows(NB, 3), "the sets of a launch do not follow from its mode");
    __shared__ float2 meta[kWin];
    wait_for_previous_launch();
    const int tid = threadIdx.x;
    const std::int64_t sets = p.d.set_count;
    const int wl = static_cast<int>(blockIdx.x % kSet);
    const std::int64_t set = blockIdx.x / kSet, window = (p.d.first_set + set) * kSet + wl;
    const int c0 = static_cast<int>(blockIdx.y) * NB;
    if (window >= p.d.windows) return;
    int odd = 0;
    if (tid < kWin) {
        const std::int64_t gene = window * kWin + tid;
        float2 so = make_float2(0.0f, 0.0f);
        if (gene < p.d.cols) so = make_float2(p.d.scales != nullptr ? __ldg(p.d.scales + gene) : 1.0f, p.d.offsets != nullptr ? __ldg(p.d.offsets + gene) : 0.0f);
        meta[tid] = so;
        odd = isfinite(so.x) && isfinite(so.y) ? 0 : 1;
    }
    const int2 head = __ldcg(reinterpret_cast<const int2 *>(p.d.status)); // {status, mode}
    const int mode = head.y;
    const bool by_entry = __syncthreads_or(odd) != 0 || (mode & kByEntry) != 0 || head.x != 0, more = by_entry || (mode & (kRepeats | kNonFinite)) != 0;
    if (more) beside_tiles<NB>(p, mode, by_entry, window, meta, beside, reinterpret_cast<unsigned long long *>(beside + kWin * NB));
    const int passes = passes_of(mode), c = tid / kWin * 16;
    // the set's slots: the CTAs whose shares meet its runs, run after run, pass after pass
    const std::int64_t total = sets * p.d.column_blocks * p.d.group_count * passes, L = p.d.group_count, cuts = (L + p.d.run_groups - 1) / p.d.run_groups;
    const int gl = tid & (kWin - 1);
    const bool mine = window * kWin + gl < p.d.cols && c0 + c < p.n;
    float *results = reinterpret_cast<float *>(beside + kWin * NB);
    constexpr int kPitch = finish_pitch(NB), kAtOnce = EXACT ? 8 : 16; // columns
#pragma unroll 1
    for (int h = 0; h < 16; h += kAtOnce) {
        double sum[kAtOnce];
#pragma unroll
        for (int k = 0; k < kAtOnce; ++k) sum[k] = more ? beside[gl * NB + c + h + k] : 0.0;
        for (int pass = 0; pass < passes && !by_entry && mine; ++pass) {
            const std::int64_t block = static_cast<std::int64_t>(pass) * p.d.column_blocks + blockIdx.y, set_of_all = block * sets + set;
            if constexpr (EXACT) {
                const double scale = static_cast<double>(meta[gl].x), offset = static_cast<double>(meta[gl].y);
                const long long *at = p.d.totals + ((set_of_all * kSet + wl) * 2 * NB + c + h) * kWin + gl;
                const double *steps = p.d.steps + block * NB + c + h;
                long long coded[kAtOnce], present[kAtOnce];
#pragma unroll
                for (int k = 0; k < kAtOnce; ++k) {
                    coded[k] = __ldcg(at + k * kWin);
                    present[k] = __ldcg(at + (NB + k) * kWin);
                }
#pragma unroll
                for (int k = 0; k < kAtOnce; ++k) sum[k] += value_of(coded[k], present[k], p.d.code_bias, scale, offset, __ldg(steps + k));
            } else {
                for (std::int64_t cut = 0; cut < cuts; ++cut) {
                    const std::int64_t from = set_of_all * L + cut * p.d.run_groups, to = min(from + p.d.run_groups, (set_of_all + 1) * L);
                    const std::int64_t last = cta_of(to - 1, total, p.grid);
                    for (std::int64_t b = cta_of(from, total, p.grid); b <= last; ++b) {
                        const float *slot = p.d.partials + (((set_of_all * cuts + cut + b) * kSet + wl) * NB + c) * kWin + gl;
                        float u[kAtOnce];
#pragma unroll
                        for (int k = 0; k < kAtOnce; ++k) u[k] = __ldcg(slot + k * kWin);
#pragma unroll
                        for (int k = 0; k < kAtOnce; ++k) sum[k] += static_cast<double>(u[k]);
                    }
                }
            }
        }
#pragma unroll
        for (int k = 0; k < kAtOnce; k += 4)
            *reinterpret_cast<float4 *>(results + gl * kPitch + c + h + k) =
                make_float4(static_cast<float>(sum[k]), static_cast<float>(sum[k + 1]), static_cast<float>(sum[k + 2]), static_cast<float>(sum[k + 3]));
    }
    __syncthreads();
    const int genes = static_cast<int>(min(static_cast<std::int64_t>(kWin), p.d.cols - window * kWin)), columns = min(NB, p.n - c0);
    float *out = p.out + window * kWin * p.out_ld + c0;
    if (p.out_vector != 0) {
#pragma unroll
        for (int i = tid; i < kWin * (NB / 4); i += finish_threads(NB)) {
            const int gene = i / (NB / 4), at = i % (NB / 4) * 4;
            if (gene >= genes || at >= columns) continue;
            float4 *dst = reinterpret_cast<float4 *>(out + gene * p.out_ld + at);
            const float4 v = *reinterpret_cast<const float4 *>(results + gene * kPitch + at);
            float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (p.beta != 0.0f) {
                o = *dst;
                o.x *= p.beta; o.y *= p.beta; o.z *= p.beta; o.w *= p.beta;
            }
            *dst = make_float4(fmaf(p.alpha, v.x, o.x), fmaf(p.alpha, v.y, o.y), fmaf(p.alpha, v.z, o.z), fmaf(p.alpha, v.w, o.w));
        }
    } else {
        for (int i = tid; i < kWin * NB; i += finish_threads(NB)) {
            const int gene = i / NB, at = i % NB;
            if (gene >= genes || at >= columns) continue;
            float *dst = out + gene * p.out_ld + at;
            *dst = fmaf(p.alpha, results[gene * kPitch + at], p.beta == 0.0f ? 0.0f : p.beta * *dst);
        }
    }
}

// What a launch with the least workspace takes at a time: groups, and, repeatable, sets of windows.
constexpr std::int64_t kLeastGroups = 2, kLeastSets = 4, kLeastRoundedGroups = 8;
int column_block(std::int64_t n) { return n <= 32 ? 32 : 64; }
int padded_columns(std::int64_t n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : 256; }

// (both with room for a second pass, and for four digits)
std::uint64_t record_bytes(std::int64_t groups, std::int64_t n) {
    const int nb = column_block(n);
    return device_arena::rounded(2u * static_cast<std::uint64_t>(groups) * static_cast<std::uint64_t>((n + nb - 1) / nb) * kRows * static_cast<std::uint64_t>(mma_columns(nb, kMostSlices)));
}
// a run ends with its set, after kRunGroups groups, or with its CTA's share of the units
std::uint64_t partial_bytes(std::int64_t groups, std::int64_t cols, std::int64_t n, int ctas) {
    const std::int64_t nb = column_block(n), per_set = set_windows(static_cast<int>(nb), kMostSlices), windows = (cols + kWin - 1) / kWin;
    const std::int64_t sets = (windows + per_set - 1) / per_set * ((n + nb - 1) / nb), cuts = (groups + kRunGroups - 1) / kRunGroups;
    return device_arena::rounded(static_cast<std::uint64_t>(2 * sets * cuts + ctas) * static_cast<std::uint64_t>(per_set * kWin * nb) * sizeof(float));
}
std::uint64_t odd_bytes(std::int64_t groups, std::int64_t n) {
    return device_arena::rounded(static_cast<std::uint64_t>(groups * (kRows / 16) * odd_chunks(static_cast<int>(n))) * sizeof(unsigned short));
}
// what a launch over `groups` of `all` groups at a time needs, without the words
std::uint64_t launch_bytes(std::int64_t all, std::int64_t groups, std::int64_t cols, std::int64_t n, int ctas) {
    return kRecordsAt + odd_bytes(all, n) + record_bytes(groups, n) + partial_bytes(groups, cols, n, ctas);
}
// ... and a repeatable one over `sets` sets of windows at a time
std::int64_t set_count_of(std::int64_t cols, std::int64_t n) {
    const std::int64_t per_set = set_windows(column_block(n), kMostSlices), windows = (cols + kWin - 1) / kWin;
    return (windows + per_set - 1) / per_set;
}
std::uint64_t total_bytes(std::int64_t sets, std::int64_t n) { // of one pass
    const std::int64_t nb = column_block(n);
    return static_cast<std::uint64_t>(sets * ((n + nb - 1) / nb) * set_windows(static_cast<int>(nb), kMostSlices) * kWin * nb) * 16u;
}
std::uint64_t exact_bytes(std::int64_t all, std::int64_t groups, std::int64_t sets, std::int64_t n) {
    return kRecordsAt + odd_bytes(all, n) + record_bytes(groups, n) + 2u * total_bytes(sets, n);
}
std::int64_t group_count_of(std::int64_t rows) { return (rows + kRows - 1) / kRows; }
std::int64_t piece_count(std::int64_t rows) { return (rows + piece_rows_of(rows) - 1) / piece_rows_of(rows); }
std::uint64_t word_bytes(std::int64_t rows, std::int64_t cols, std::int64_t nnz) {
    const std::int64_t windows = (cols + kWin - 1) / kWin;
    return static_cast<std::uint64_t>(nnz + 4 + piece_count(rows) * (4 * windows + 4)) * 4u;
}
std::uint64_t bound_bytes(std::int64_t rows, std::int64_t cols) { return static_cast<std::uint64_t>(piece_count(rows) * ((cols + kWin - 1) / kWin + 1)) * 4u; }
int build_smem_bytes(std::int64_t cols) {
    const std::int64_t windows = (cols + kWin - 1) / kWin;
    return static_cast<int>((kPieceRows * (windows | 1) + (windows + 31) / 32 * (kPieceRows + 1) + windows) * 4);
}

struct digit_launch {
    digit_params main;       // group_begin, group_count: of the whole row range
    finish_params finish;
    std::int64_t slice;      // groups at a time
    std::int64_t chunk;      // EXACT: sets of windows at a time
    pack_params pack;        // without the groups and what is to be cleared
    bool early; // the launch in front is a kernel of this call
};

// Slice after slice of the groups: the runs' sums are rounded and a slice's are added to G'.  EXACT (a request that has to be
// repeatable): chunk after chunk of the windows and slice after slice of the groups, whose sums meet as whole numbers, so that neither the
// grid nor the room for slices and chunks changes a bit.
template<int NB, int BASE, bool EXACT>
cb200_status launch_digits(const digit_launch &l, int sm_count, cudaStream_t stream) {
    constexpr std::size_t smem = std::max(digits_smem_bytes<NB, BASE>(), digits_smem_bytes<NB, kMostSlices>());
    static_assert(smem <= 232448, "shared memory budget");
    constexpr int finish_smem = finish_smem_bytes(NB), kSet = set_windows(NB, kMostSlices);
    const auto main_kernel = qcsr_transpose_digits_kernel<NB, BASE, EXACT>;
    const auto finish = finish_kernel<NB, EXACT>;
    CB200_CUDA_OK(cudaFuncSetAttribute(main_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    CB200_CUDA_OK(cudaFuncSetAttribute(finish, cudaFuncAttributeMaxDynamicSharedMemorySize, finish_smem));
    const int n = l.finish.n;
    CB200_CUDA_OK(launch_kernel(l.early, column_range_kernel, dim3(kParts), 1024, 0, stream, l.finish.g, l.finish.g_ld, n, l.pack.padded, l.finish.row_begin, l.finish.row_end,
                                const_cast<unsigned *>(l.pack.part_max), const_cast<double2 *>(l.pack.part_sum), const_cast<unsigned *>(l.pack.part_least),
                                l.early ? nullptr : l.main.status));
    count_launch();
    const std::int64_t group_end = l.main.group_begin + l.main.group_count, sets = (l.main.windows + kSet - 1) / kSet;
    const std::int64_t chunk = EXACT ? l.chunk : sets;
    for (std::int64_t first_set = 0; first_set < sets; first_set += chunk) {
        digit_params m = l.main;
        finish_params f = l.finish;
        m.first_set = first_set;
        m.set_count = std::min(chunk, sets - first_set);
        bool clear = true;
        const auto finish_groups = [&](std::int64_t grid) {
            f.d = m;
            f.grid = grid;
            count_launch();
            return launch_kernel(true, finish, dim3(static_cast<unsigned>(m.set_count * kSet), static_cast<unsigned>(m.column_blocks)), finish_threads(NB), finish_smem, stream, f);
        };
        for (std::int64_t begin = l.main.group_begin; begin < group_end; begin += l.slice) {
            m.group_begin = begin;
            m.group_count = std::min(l.slice, group_end - begin);
            // behind the slice's records; EXACT: the same place for all slices
            unsigned char *sums = l.pack.records + record_bytes(EXACT ? l.slice : m.group_count, n);
            m.partials = EXACT ? nullptr : reinterpret_cast<float *>(sums);
            m.totals = EXACT ? reinterpret_cast<long long *>(sums) : nullptr;
            const std::int64_t row0 = l.finish.first_row + begin * kRows, blocks = m.group_count * m.column_blocks;
            pack_params k = l.pack;
            k.first_row = row0;
            k.groups = m.group_count;
            k.odd_rows = l.pack.odd_rows + (begin - l.main.group_begin) * (kRows / 16) * odd_chunks(n);
            k.totals = reinterpret_cast<uint4 *>(m.totals);
            k.total_items = EXACT && clear ? static_cast<std::int64_t>(total_bytes(m.set_count, n) / 16u) : 0;
            CB200_CUDA_OK(launch_kernel(true, pack_digits_kernel<NB, BASE>, dim3(static_cast<unsigned>(std::min<std::int64_t>(blocks * kGPieces, 4 * sm_count))), 256, 0, stream, k));
            clear = false;
            const unsigned grid = static_cast<unsigned>(std::min<std::int64_t>(m.set_count * blocks, sm_count));
            CB200_CUDA_OK(launch_kernel(true, main_kernel, dim3(grid), kThreads, smem, stream, m));
            count_launch(2);
            if (EXACT) continue;
            f.row_begin = std::max(l.finish.row_begin, row0);
            f.row_end = std::min(l.finish.row_end, row0 + m.group_count * kRows);
            f.beta = begin != l.main.group_begin ? 1.0f : l.finish.beta;
            CB200_CUDA_OK(finish_groups(grid));
        }
        if (EXACT) CB200_CUDA_OK(finish_groups(0));
    }
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

} // namespace

cb200_status launch_digit_words(const qcsr_view &x, std::int64_t row_begin, std::int64_t row_end, std::uint32_t *words, std::uint32_t *bounds,
                                std::int64_t *bases, int *status, int *outside, cudaStream_t stream) {
    words_params p{};
    p.row_ptr = x.row_ptr; p.packed_row_ptr = x.packed_row_ptr; p.col_idx = x.col_idx; p.packed = x.packed;
    p.row_begin = row_begin; p.row_end = row_end; p.cols = x.cols; p.windows = static_cast<int>((x.cols + kWin - 1) / kWin);
    p.code_bias = x.bits == 8 ? 128 : 0;
    p.piece_rows = piece_rows_of(x.rows);
    p.words = words; p.bounds = bounds; p.bases = bases; p.status = status; p.outside = outside;
    const int smem = build_smem_bytes(x.cols);
    const unsigned grid = static_cast<unsigned>((row_end - row_begin + p.piece_rows - 1) / p.piece_rows);
    const auto run = [&](auto kernel) {
        const cudaError_t err = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (err == cudaSuccess) kernel<<<grid, kBuildThreads, smem, stream>>>(p);
        return err;
    };
    if (outside != nullptr) CB200_CUDA_OK(x.bits == 8 ? run(digit_words_kernel<8, true>) : run(digit_words_kernel<4, true>));
    else CB200_CUDA_OK(x.bits == 8 ? run(digit_words_kernel<8, false>) : run(digit_words_kernel<4, false>));
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

bool qcsr_transpose_digits_shape_ok(std::int64_t rows, std::int64_t cols, std::int64_t n, int bits, int policy) {
    // the counters of a piece have to fit in shared memory: 190,000 genes
    return (bits == 8 || bits == 4) && policy == CB200_DECODE_PER_GENE_AFFINE && n > 0 && n <= kMaxColumns && rows > 0 && cols > 0 &&
           cols <= 190'000 && build_smem_bytes(cols) <= 210 * 1024;
}
std::uint64_t qcsr_digit_words_bytes_bound(std::int64_t rows, std::int64_t cols, std::int64_t nnz) {
    return device_arena::rounded(word_bytes(rows, cols, nnz)) + device_arena::rounded(bound_bytes(rows, cols)) +
           device_arena::rounded(static_cast<std::uint64_t>(piece_count(rows)) * 8u) + device_arena::rounded(sizeof(int)); // (the last: while they are built)
}
digit_layout digit_words_at(void *memory, const qcsr_view &x) {
    unsigned char *at = static_cast<unsigned char *>(memory);
    digit_layout l;
    l.words = reinterpret_cast<std::uint32_t *>(at);
    at += device_arena::rounded(word_bytes(x.rows, x.cols, x.nnz));
    l.bounds = reinterpret_cast<std::uint32_t *>(at);
    at += device_arena::rounded(bound_bytes(x.rows, x.cols));
    l.bases = reinterpret_cast<std::int64_t *>(at);
    return l;
}
std::uint64_t qcsr_transpose_digits_workspace_bytes(std::int64_t rows, std::int64_t cols, std::int64_t n, bool repeatable) {
    const std::int64_t groups = group_count_of(rows);
    if (repeatable) return exact_bytes(groups, groups, set_count_of(cols, n), n);
    return launch_bytes(groups, groups, cols, n, kMaxCtas);
}
std::uint64_t qcsr_transpose_digits_least_workspace(std::int64_t rows, std::int64_t cols, std::int64_t n, bool repeatable, int sm_count) {
    const std::int64_t groups = group_count_of(rows);
    if (repeatable) return exact_bytes(groups, std::min<std::int64_t>(groups, kLeastGroups), std::min<std::int64_t>(set_count_of(cols, n), kLeastSets), n);
    return launch_bytes(groups, std::min<std::int64_t>(groups, kLeastRoundedGroups), cols, n, std::min(sm_count, kMaxCtas));
}
std::uint64_t qcsr_transpose_digits_once_bytes(std::int64_t rows, std::int64_t cols, std::int64_t n, std::int64_t nnz, int bits, int policy) {
    if (!qcsr_transpose_digits_shape_ok(rows, cols, n, bits, policy)) return 0u;
    // Sparser, a tile is mostly zeroes; fewer entries, and the five launches take longer than the two of the other kernel.  One call, N =
    // 64: 2,000 x 8,000 (1.6 M entries) 48 us against 45, 1,500 x 33,538 (2.7 M) 75 against 75, 4,000 x 4,000 (2.1 M) 49 against 57,
    // 8,191 x 33,538 (14.7 M) 171 against 318; at N = 32 8,000 x 2,000 (2.9 M) 51 against 53, 16,384 x 2,000 (5.9 M) 74 against 108.
    if (static_cast<double>(nnz) < 0.02 * static_cast<double>(rows) * static_cast<double>(cols) || nnz < kLeastOnceEntries || nnz > kMostOnceEntries) return 0u;
    return qcsr_transpose_digits_workspace_bytes(rows, cols, n, false) + qcsr_digit_words_bytes_bound(rows, cols, nnz);
}

cb200_status build_digit_words(const qcsr_view &x, bool refuse_outside, device_arena &arena, cudaStream_t stream, digit_layout *out) {
    *out = digit_layout{};
    if (x.row_ptr == nullptr || (x.nnz != 0 && (x.col_idx == nullptr || x.packed == nullptr)))
        return fail(CB200_STATUS_INVALID_ARGUMENT, "the matrix handed to prepare has null arrays");
    if (x.bits == 4 && x.packed_row_ptr == nullptr) return fail(CB200_STATUS_INVALID_ARGUMENT, "4-bit codes need packed_row_ptr");
    const std::uint64_t words = word_bytes(x.rows, x.cols, x.nnz), bounds = bound_bytes(x.rows, x.cols), bases = static_cast<std::uint64_t>(piece_count(x.rows)) * 8u;
    out->words = static_cast<std::uint32_t *>(arena.take(words));
    out->bounds = static_cast<std::uint32_t *>(arena.take(bounds));
    out->bases = static_cast<std::int64_t *>(arena.take(bases));
    int *outside = static_cast<int *>(arena.take(sizeof(int)));
    cb200_status st = CB200_STATUS_SUCCESS;
    if (out->words == nullptr || out->bounds == nullptr || out->bases == nullptr || outside == nullptr)
        st = fail(CB200_STATUS_INSUFFICIENT_WORKSPACE, "no device memory for the entry words");
    const auto check = [&](cudaError_t err) {
        if (err != cudaSuccess && st == CB200_STATUS_SUCCESS) st = fail(CB200_STATUS_CUDA_ERROR, "building the entry words: %s", cudaGetErrorString(err));
    };
    if (st == CB200_STATUS_SUCCESS) check(cudaMemsetAsync(outside, 0, sizeof(int), stream));
    if (st == CB200_STATUS_SUCCESS) st = launch_digit_words(x, 0, x.rows, out->words, out->bounds, out->bases, nullptr, outside, stream);
    if (st == CB200_STATUS_SUCCESS) {
        int found = 0;
        check(cudaMemcpyAsync(&found, outside, sizeof(int), cudaMemcpyDeviceToHost, stream));
        check(cudaStreamSynchronize(stream));
        if (st == CB200_STATUS_SUCCESS && refuse_outside && found != 0) st = fail(CB200_STATUS_INVALID_SHAPE, "a column index lies outside the matrix");
    }
    arena.give_back(outside, sizeof(int));
    if (st != CB200_STATUS_SUCCESS) {
        arena.give_back(out->bases, bases);
        arena.give_back(out->bounds, bounds);
        arena.give_back(out->words, words);
        *out = digit_layout{};
        return st;
    }
    out->bytes = words + bounds + bases;
    out->src_row_ptr = x.row_ptr; out->src_col_idx = x.col_idx; out->src_packed = x.packed;
    return st;
}

cb200_status launch_qcsr_transpose_digits(const qcsr_view &x, const dense_args &d, std::int64_t row_begin, std::int64_t row_end, void *workspace,
                                          std::uint64_t workspace_bytes, const digit_layout *layout, int slices, bool repeatable, int sm_count, cudaStream_t stream, bool *taken) {
    *taken = false;
    if (row_end <= row_begin || d.dense_dtype != CB200_DTYPE_F32 || !qcsr_transpose_digits_shape_ok(x.rows, x.cols, d.n, x.bits, x.policy)) return CB200_STATUS_SUCCESS;
    if (workspace == nullptr || reinterpret_cast<std::uintptr_t>(workspace) % 256u != 0u || sm_count > kMaxCtas) return CB200_STATUS_SUCCESS;
    if (x.bits == 4 && x.packed_row_ptr == nullptr) return CB200_STATUS_SUCCESS;
    // With less workspace than for the whole range the groups are taken in slices.  A call that has to make its words has room for
    // everything or is another kernel's.
    const std::uint64_t own = qcsr_transpose_digits_workspace_bytes(x.rows, x.cols, d.n, false);
    if (layout == nullptr && workspace_bytes < own + qcsr_digit_words_bytes_bound(x.rows, x.cols, x.nnz)) return CB200_STATUS_SUCCESS;
    const std::int64_t first_row = layout != nullptr ? 0 : row_begin, rows_of_words = layout != nullptr ? x.rows : row_end - row_begin;
    const std::int64_t group_begin = (row_begin - first_row) / kRows, group_count = (row_end - first_row + kRows - 1) / kRows - group_begin;
    std::int64_t slice = group_count, chunk = repeatable ? set_count_of(x.cols, d.n) : 0;
    const auto needs = [&](std::int64_t groups) { return repeatable ? exact_bytes(group_count, groups, chunk, d.n) : launch_bytes(group_count, groups, x.cols, d.n, sm_count); };
    while (chunk > 1 && needs(std::min<std::int64_t>(slice, kLeastGroups)) > workspace_bytes) chunk = (chunk + 1) / 2;
    while (slice > 1 && needs(slice) > workspace_bytes) slice = (slice + 1) / 2;
    if (needs(slice) > workspace_bytes) return CB200_STATUS_SUCCESS;
    if (layout != nullptr && (x.row_ptr != layout->src_row_ptr || x.col_idx != layout->src_col_idx || x.packed != layout->src_packed))
        return fail(CB200_STATUS_STALE_STRUCTURE, "the launch's matrix is not the one the entry words were built from");
    *taken = true;
    unsigned char *ws = static_cast<unsigned char *>(workspace);
    digit_launch l{};
    l.early = layout == nullptr;
    digit_params &p = l.main;
    p.status = reinterpret_cast<int *>(ws);
    l.slice = slice;
    l.chunk = chunk;
    if (layout != nullptr) {
        p.words = layout->words; p.bounds = layout->bounds; p.bases = layout->bases;
    } else {
        const digit_layout made = digit_words_at(ws + own, x);
        const cb200_status st = launch_digit_words(x, row_begin, row_end, made.words, made.bounds, made.bases, p.status, nullptr, stream);
        if (st != CB200_STATUS_SUCCESS) return st;
        p.words = made.words; p.bounds = made.bounds; p.bases = made.bases;
    }
    const int nb = column_block(d.n);
    p.piece_rows = piece_rows_of(x.rows);
    p.group_pieces = kRows / p.piece_rows;
    p.pieces = (rows_of_words + p.piece_rows - 1) / p.piece_rows;
    p.scales = x.scales; p.offsets = x.offsets;
    pack_params &k = l.pack;
    k.g = static_cast<const float *>(d.dense); k.ld = d.dense_ld; k.row_begin = row_begin; k.row_end = row_end;
    k.n = static_cast<int>(d.n); k.padded = padded_columns(d.n);
    k.part_max = reinterpret_cast<const unsigned *>(ws + kPartMaxAt);
    k.part_sum = reinterpret_cast<const double2 *>(ws + kPartSumAt);
    k.part_least = reinterpret_cast<const unsigned *>(ws + kPartLeastAt);
    k.steps = reinterpret_cast<double *>(ws + kStepsAt);
    k.odd_rows = reinterpret_cast<unsigned short *>(ws + kRecordsAt);
    k.records = ws + kRecordsAt + odd_bytes(group_count, d.n);
    k.bases = p.bases; k.word_pieces = p.pieces;
    k.mode = reinterpret_cast<int *>(ws) + 1; // finish_kernel reads both words at once
    p.records = k.records; p.steps = k.steps; p.mode = k.mode;
    p.cols = x.cols;
    p.group_begin = group_begin;
    p.group_count = group_count;
    p.run_groups = kRunGroups;
    p.windows = static_cast<int>((x.cols + kWin - 1) / kWin);
    p.column_blocks = static_cast<int>((d.n + nb - 1) / nb);
    p.code_bias = x.bits == 8 ? 128 : 0;
    p.poll_limit = test_poll_limit();
    finish_params &f = l.finish;
    f.g = static_cast<const float *>(d.dense); f.g_ld = d.dense_ld;
    f.odd_rows = k.odd_rows; f.odd_from = first_row + group_begin * kRows;
    f.first_row = first_row; f.row_begin = row_begin; f.row_end = row_end;
    f.out = d.out; f.out_ld = d.out_ld; f.n = static_cast<int>(d.n);
    f.out_vector = reinterpret_cast<std::uintptr_t>(d.out) % 16u == 0u && d.out_ld % 4 == 0 && d.n % 4 == 0 ? 1 : 0;
    f.alpha = d.alpha; f.beta = d.beta;
    if (repeatable) return nb == 64 ? launch_digits<64, kMostSlices, true>(l, sm_count, stream) : launch_digits<32, kMostSlices, true>(l, sm_count, stream);
    if (slices == 4) return nb == 64 ? launch_digits<64, 4, false>(l, sm_count, stream) : launch_digits<32, 4, false>(l, sm_count, stream);
    return nb == 64 ? launch_digits<64, 3, false>(l, sm_count, stream) : launch_digits<32, 3, false>(l, sm_count, stream);
}

} // namespace cb200
