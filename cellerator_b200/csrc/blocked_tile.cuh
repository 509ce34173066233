// Geometry of the window tiles, the entry-word layout and the W records shared by the tensor-core
// kernels over the window-blocked copy (qcsr_forward_blocked.cu) and over the dense operand tiles
// (qcsr_forward_dense.cu).  Everything here has internal linkage: each translation unit that
// includes the header gets its own copy.
#pragma once

#include "kernels.cuh"
#include "operand_scaling.cuh"
#include "sm100_primitives.cuh"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace cb200 {
namespace {

// Geometry.  A (group, window) tile is 256 cells x 128 genes = 64 KB of bf16, double buffered.
// (512 cells x 64 genes halves the W bytes per unit of work but leaves 13 instead of 26 groups per
// SM on a 1M-cell shard; the coarser deal costs more than the W traffic saves: 8.0 ms against 7.5.)
constexpr int kWin = 128;                    // genes per window
constexpr int kWinShift = 7;
constexpr int kRows = 256;                   // cell rows per group
constexpr int kRowsShift = 8;
constexpr int kSubBlocks = kRows / 128;      // one M = 128 MMA each
constexpr int kProducerWarps = 16;           // zero + scatter; the first kEpilogueWarps of them also write Y
constexpr int kEpilogueWarps = kRows / 32;
constexpr int kProducerThreads = kProducerWarps * 32;
// Measured on the 1M x 33,538 matrix (ms per launch) for (chunk loader warps, chunk stages): (1, 2) 7.11,
// (2, 2) 7.13, (1, 3) 7.36, (2, 4) 7.38, (3, 3) 7.55, (1, 1) 8.96; W stages 4 / 3 / 2: 7.13 / 7.38 / 7.68.
constexpr int kChunkLoaders = 1;                // warps whose elected lane issues entry-chunk copies
constexpr int kThreads = kProducerThreads + 32 * (2 + kChunkLoaders); // + MMA warp + W loader warp + chunk loader warps
constexpr int kABufBytes = kRows * kWin * 2;    // 64 KB
constexpr int kSubBlockBytes = 128 * kWin * 2;  // 16 KB
constexpr int kRowGroupBytes = kWin * 16;       // W slice: 8 columns x kWin genes of bf16
constexpr int kChunkEntries = 2048;
constexpr int kChunkBytes = kChunkEntries * 4;
// chunk stages (template parameter CS of the kernel): 2 when a segment fits one chunk, 3 for denser matrices
constexpr int kMaxWStages = 6;
constexpr std::uint32_t kInvalidEntry = 0x80000000u; // padding of a segment
static_assert(kProducerWarps >= kEpilogueWarps && kABufBytes % (kProducerThreads * 16) == 0, "thread t < kRows owns row t in the epilogue");
static_assert(kABufBytes <= 65536, "an entry holds the byte position in the tile, halved, in 15 bits");

__host__ __device__ constexpr int record_bytes(int n) { return n * kWin * 2 + kWin * 8; }
__host__ __device__ constexpr int fixed_smem_bytes(int cs) { return 2 * kABufBytes + cs * kChunkBytes + kRows * 4 + 512; }
__host__ __device__ constexpr int w_stages(int n, int cs) {
    return (232448 - fixed_smem_bytes(cs)) / record_bytes(n) >= kMaxWStages ? kMaxWStages
                                                                            : (232448 - fixed_smem_bytes(cs)) / record_bytes(n);
}

// Byte position of (row within group, gene within window) in the A tile.  The tile is made of
// sub-blocks of 128 rows; a sub-block is K-major with the 128-byte swizzle: per 64 genes (a "half",
// kHalfBytes; one half when the window is 64 genes wide) 8-row atoms of 1,024 bytes in which row r
// holds its 64 genes in one 128-byte line whose 16-byte pieces are permuted by r mod 8.  The
// permutation spreads the scattered 2-byte stores of one row, and of neighbouring rows, over all
// shared-memory banks.
constexpr int kHalfBytes = 128 * 64 * 2; // 16 KB: 128 rows x 64 genes
__host__ __device__ constexpr std::uint32_t tile_offset(int rl, int gl) {
    return static_cast<std::uint32_t>((rl >> 7) * kSubBlockBytes + (gl >> 6) * kHalfBytes + ((rl & 127) >> 3) * 1024 +
                                      (rl & 7) * 128 + ((((gl & 63) >> 3) ^ (rl & 7)) * 16) + (gl & 7) * 2);
}
// The transpose kernel's tile of the same (group, window): M = gene, K = cell, K-major with the 128-byte
// swizzle: [cell quarter of 64][gene][64 cells], the 16-byte pieces of a gene's line permuted by gene mod 8.
__host__ __device__ constexpr std::uint32_t tile_offset_gene_major(int rl, int gl) {
    return static_cast<std::uint32_t>((rl >> 6) * (kWin * 128) + (gl >> 3) * 1024 + (gl & 7) * 128 + ((((rl & 63) >> 3) ^ (gl & 7)) << 4) +
                                      ((rl & 7) << 1));
}


// K-major operand, no swizzle: LBO = 128 B between the two core matrices one K = 16 step reads,
// SBO = kRowGroupBytes between groups of 8 rows.
__device__ __forceinline__ std::uint64_t smem_desc(std::uint32_t addr) {
    std::uint64_t d = 0;
    d |= static_cast<std::uint64_t>((addr & 0x3ffffu) >> 4);
    d |= static_cast<std::uint64_t>(128u >> 4) << 16;
    d |= static_cast<std::uint64_t>(static_cast<unsigned>(kRowGroupBytes) >> 4) << 32;
    d |= static_cast<std::uint64_t>(1) << 46; // descriptor version of this architecture
    return d;
}
// W [genes][n] (leading dimension ld) -> one record per window of 128 genes: the n x 128 slice of
// W^T in operand layout (byte offset of (column c, gene e) = (c/8)*2048 + (e/8)*128 + (c%8)*16 +
// (e%8)*2, zero for genes >= cols) followed by 128 x {scale, zero-point}.  part 0 writes
// hi = bf16(w) (w itself for a bf16 W); part 1 writes lo = bf16(w - hi), the next 8 mantissa bits.
// both_parts: 2 n columns, hi and then lo.
// With absmax != null the record holds fp16: hi = fp16(w * s), lo = fp16(w * s - hi), s = operand_scale(largest |w|).
// absmax is word 1 of the status block: the largest |w|, written here from absmax_kernel's parts.
// The grid is (windows, column groups): block (w, g) lays out the record's columns [g, g + 1) * columns / gridDim.y of window
// w; the blocks of group 0 also write the window's table.
constexpr int kPackColumns = 16; // columns of W per block of the packing kernel
template<typename WT>
__global__ void __launch_bounds__(256) pack_windows_kernel(const WT *w, std::int64_t ld, std::int64_t cols, int n, int part,
                                                           const float *scales, const float *offsets, int per_gene_offsets,
                                                           unsigned char *records, unsigned *absmax = nullptr, int both_parts = 0) {
    wait_for_previous_launch();
    let_next_launch_start();
    const std::int64_t window = blockIdx.x;
    const int columns = both_parts != 0 ? 2 * n : n; // both_parts: the hi part of the n columns, then their lo part
    unsigned char *rec = records + window * record_bytes(columns);
    __nv_bfloat16 *wt = reinterpret_cast<__nv_bfloat16 *>(rec);
    const bool fp16 = absmax != nullptr;
    float ws = 1.0f;
    if (fp16) {
        const unsigned most = largest_part(absmax + kAbsmaxWord - 1);
        if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) *absmax = most;
        ws = operand_scale(__uint_as_float(most));
    }
    const int group_cols = columns / static_cast<int>(gridDim.y), c_first = static_cast<int>(blockIdx.y) * group_cols;
    for (int i = threadIdx.x; i < group_cols * kWin; i += blockDim.x) {
        const int e = i / group_cols, column = c_first + i % group_cols; // consecutive threads read consecutive columns of one gene
        const int c = column < n ? column : column - n;
        const bool lo = column < n ? part != 0 : true;
        const std::int64_t gene = window * kWin + e;
        float value = 0.0f;
        if (gene < cols) {
            if constexpr (sizeof(WT) == 2) value = __bfloat162float(w[gene * ld + c]);
            else value = w[gene * ld + c];
        }
        const int at = ((column >> 3) * kRowGroupBytes + (e >> 3) * 128 + (column & 7) * 16 + (e & 7) * 2) >> 1;
        if (fp16) {
            const float scaled = value * ws;
            __half h = __float2half_rn(scaled);
            if (lo) h = __float2half_rn(scaled - __half2float(h));
            reinterpret_cast<__half *>(rec)[at] = h;
            continue;
        }
        __nv_bfloat16 v = __float2bfloat16_rn(value);
        if (lo) v = __float2bfloat16_rn(value - __bfloat162float(v));
        wt[at] = v;
    }
    if (blockIdx.y != 0) return;
    float2 *table = reinterpret_cast<float2 *>(rec + columns * kWin * 2);
    for (int e = threadIdx.x; e < kWin; e += blockDim.x) {
        const std::int64_t gene = window * kWin + e;
        float2 so = make_float2(0.0f, 0.0f);
        if (gene < cols) {
            so.x = scales != nullptr ? scales[gene] : 1.0f;
            so.y = (per_gene_offsets && offsets != nullptr) ? offsets[gene] : 0.0f;
        }
        table[e] = so;
    }
}

// The work of a CTA: whole groups, or parts of a group's windows (window_split_plan).
struct window_split {
    int whole;    // groups from this one on are cut
    int parts;
    int per_unit; // parts of a cut group that a unit takes
    int slots;    // per cut group: one a part, or one a pair of parts
    float *sums;  // [(group - whole) * slots + slot][kRows][N], raw accumulators
};
struct window_unit {
    int group, w0, w1;
    int slot;        // where its first sums go; -1: a whole group, written to Y
    int k0, pieces;  // parts of the group's windows that the unit takes: [k0, k0 + pieces)
};
__host__ __device__ __forceinline__ int part_begin(int windows, int parts, int part) { return windows * part / parts; }
__host__ __device__ __forceinline__ int whole_groups_in(const window_split &s, std::int64_t begin, std::int64_t end) {
    const int last = s.whole < static_cast<int>(end) ? s.whole : static_cast<int>(end);
    return last > static_cast<int>(begin) ? last - static_cast<int>(begin) : 0;
}
// units of the groups [begin, end): whole groups first, then the parts of the others
__host__ __device__ __forceinline__ int unit_count(const window_split &s, std::int64_t begin, std::int64_t end) {
    const int whole = whole_groups_in(s, begin, end);
    return whole + (static_cast<int>(end - begin) - whole) * ((s.parts + s.per_unit - 1) / s.per_unit);
}
__device__ __forceinline__ window_unit unit_at(const window_split &s, std::int64_t begin, std::int64_t end, int windows, int u) {
    const int whole = whole_groups_in(s, begin, end);
    if (u < whole) return window_unit{static_cast<int>(begin) + u, 0, windows, -1, 0, s.parts};
    const int units = (s.parts + s.per_unit - 1) / s.per_unit;
    const int cut = (u - whole) / units, part = ((u - whole) - cut * units) * s.per_unit, pieces = min(s.per_unit, s.parts - part);
    const int group = static_cast<int>(begin) + whole + cut;
    return window_unit{group, part_begin(windows, s.parts, part), part_begin(windows, s.parts, part + pieces),
                       (group - s.whole) * s.slots + (s.slots < s.parts ? part / 2 : part), part, pieces};
}
// units of this CTA: blockIdx.x, + gridDim.x, ...
__device__ __forceinline__ int units_of_cta(const window_split &s, std::int64_t begin, std::int64_t end) {
    const int units = unit_count(s, begin, end), first = static_cast<int>(blockIdx.x), step = static_cast<int>(gridDim.x);
    return units > first ? (units - first + step - 1) / step : 0;
}

// Y of the groups that were cut: the parts' sums in order, then what the epilogue of a whole group does.
// result_scale / w_absmax: the powers of two the operands were stored times (null: none).
// paired: the sums of two neighbouring parts are added first.
__global__ void __launch_bounds__(256) add_parts_kernel(const float *sums, int slots, int paired, int whole, int first_group, std::int64_t row_end,
                                                        int n, float *y, std::int64_t y_ld, float alpha, float beta, const float *bias,
                                                        int epilogue, float result_scale, const unsigned *w_absmax) {
    wait_for_previous_launch();
    const std::int64_t group = first_group + static_cast<int>(blockIdx.x);
    const float *in = sums + (group - whole) * slots * kRows * n;
    float scale = alpha * result_scale;
    if (w_absmax != nullptr) scale /= operand_scale(__uint_as_float(__ldg(w_absmax)));
    const int pieces = kRows * n / 4;
    for (int i = blockIdx.y * 256 + threadIdx.x; i < pieces; i += gridDim.y * 256) {
        const int r = i / (n / 4), c = (i % (n / 4)) * 4;
        const std::int64_t row = group * kRows + r;
        if (row >= row_end) break;
        const auto sum_at = [&](int k) {
            return k < slots ? *reinterpret_cast<const float4 *>(in + static_cast<std::int64_t>(k) * kRows * n + 4 * static_cast<std::int64_t>(i)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        };
        const auto add = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
        float4 v = sum_at(0);
        const int pair = paired != 0 ? 2 : 1;
        if (pair == 2 && slots > 1) v = add(v, sum_at(1));
#pragma unroll 1
        for (int k = pair; k < slots; k += 4) { // four in flight
            const float4 t0 = sum_at(k), t1 = sum_at(k + 1), t2 = sum_at(k + 2), t3 = sum_at(k + 3);
            if (pair == 2) {
                v = add(v, k + 1 < slots ? add(t0, t1) : t0);
                if (k + 2 < slots) v = add(v, k + 3 < slots ? add(t2, t3) : t2);
            } else {
                v = add(v, t0);
                if (k + 1 < slots) v = add(v, t1);
                if (k + 2 < slots) v = add(v, t2);
                if (k + 3 < slots) v = add(v, t3);
            }
        }
        float *out = y + row * y_ld + c;
        v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
        if (beta != 0.0f) {
            const float4 o = *reinterpret_cast<const float4 *>(out);
            v.x = fmaf(beta, o.x, v.x); v.y = fmaf(beta, o.y, v.y); v.z = fmaf(beta, o.z, v.z); v.w = fmaf(beta, o.w, v.w);
        }
        if (epilogue != CB200_EPILOGUE_NONE) {
            v.x = finish_output(v.x, bias, c, epilogue); v.y = finish_output(v.y, bias, c + 1, epilogue);
            v.z = finish_output(v.z, bias, c + 2, epilogue); v.w = finish_output(v.w, bias, c + 3, epilogue);
        }
        *reinterpret_cast<float4 *>(out) = v;
    }
}
inline cb200_status launch_add_parts(const window_split &s, bool pairs, std::int64_t group_begin, std::int64_t group_end, std::int64_t row_end, int n, float *y,
                                     std::int64_t y_ld, float alpha, float beta, const float *bias, int epilogue, float result_scale,
                                     const unsigned *w_absmax, cudaStream_t stream) {
    const int first = static_cast<int>(group_begin) + whole_groups_in(s, group_begin, group_end), cut = static_cast<int>(group_end) - first;
    if (cut <= 0) return CB200_STATUS_SUCCESS;
    CB200_CUDA_OK(launch_kernel(true, add_parts_kernel, dim3(static_cast<unsigned>(cut), static_cast<unsigned>(n / 8)), 256, 0, stream, s.sums, s.slots,
                                pairs && s.slots == s.parts ? 1 : 0, s.whole,
                                first, row_end, n, y, y_ld, alpha, beta, bias, epilogue, result_scale, w_absmax));
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}
// The split of a launch: groups are cut where the workspace holds the sums behind its `used` bytes.
inline window_split split_of_launch(const qcsr_view &x, std::int64_t n, std::int64_t columns, void *workspace, std::uint64_t workspace_bytes, std::uint64_t used,
                                    int sm_count) {
    const window_split_plan plan = qcsr_window_split(x.rows, x.cols, columns, sm_count);
    const std::uint64_t at = device_arena::rounded(used), sums = qcsr_window_split_bytes(x.rows, x.cols, n, columns, sm_count);
    if (sums == 0u || workspace_bytes < at + sums) return window_split{0x7fffffff, plan.parts, 1, 1, nullptr};
    return window_split{static_cast<int>(plan.whole), plan.parts, plan.per_unit, plan.slots, reinterpret_cast<float *>(static_cast<unsigned char *>(workspace) + at)};
}

} // namespace
} // namespace cb200
