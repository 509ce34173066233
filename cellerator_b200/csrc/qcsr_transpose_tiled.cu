// Gene-side transpose  G' = alpha * deq(X)^T * G + beta * G'  with fp32 FMAs from the CSR arrays alone, for matrices that are
// seen once.
//
// Reference counterpart: csr_spmm_bwd_rhs_kernel_ (src/compute/sparse/ops/kernels/base_sparse/csr_spmm_bwd_rhs_kernel_.cuh:1-22),
// one atomicAdd per (stored entry, output column).  qcsr_transpose_atomic_kernel (qcsr_transpose.cu) still sends a row of N
// floats to L2 for every stored entry and runs at the rate at which L2 adds them: 4 TB/s, 1.3 ms for 8,191 x 33,538 with 15 M
// entries at N = 64.
//
// Here a CTA holds a tile of up to 512 rows of G in shared memory and takes a range of up to 512 genes at a time.  It sorts the
// entries of (tile, range) by gene in shared memory (counting sort of one-word entries {row of the tile, code}), then a warp
// per gene walks the gene's entries, reads their rows of G from the tile and keeps the sum in registers: one vector reduction
// per (gene, tile) instead of one per entry.
//
// What bounds it: the LSU data pipe, 80 % busy: 56.7 M wavefronts of shared memory for 14.6 M entries, 40 M of them loads (rows
// of G are two wavefronts per entry at N = 64) and 14 M the sort's atomics; 281 us, and 48 us of the pass over the indices, whose
// 256 CTAs of 1,024 threads are dealt unevenly to 148 SMs.  A tile of 512 rows is what leaves room for the entries of 512 genes;
// smaller tiles would make the runs per gene too short to pay for their start and the reduction (27 entries at 5 % density),
// more rows do not fit.  8,191 x 33,538, 14.7 M entries: N = 64 1.37 -> 0.31 ms, N = 50 2.54 -> 0.32 ms; 16,384 rows at N = 128
// (two column tiles, sorted twice) 4.33 -> 1.12 ms.
//
// Where a row's entries of a range start comes from a pass over the indices that also sets the output to beta * G': for range j
// the first entry whose gene, or any before it, reaches j * width.  That is a partition of the row whatever its order; entries
// of a row that does not ascend may then lie in a range that is not theirs, and those are added one by one.
#include "kernels.cuh"

#include <algorithm>
#include <cstring>

namespace cb200 {
namespace {

constexpr int kTileRows = 512;
constexpr int kTileGenes = 512;
constexpr int kTileThreads = 1024;
constexpr int kTileWarps = kTileThreads / 32;
constexpr int kTileWords = 16 * 1024;                      // entries of a sorted batch, every gene's padded to a multiple of 4
constexpr int kBatch = kTileWords - 3 * kTileGenes;         // entries of a sorted batch before the padding
constexpr int kStepsPerWarp = (kBatch / kTileWarps + 31) / 32; // 15
constexpr int kStepGroup = 5;                              // steps whose loads are in flight together
constexpr std::uint32_t kNoEntry = 0xffffffffu;
constexpr int kMaxRanges = 1023;

struct tiled_transpose_params {
    const std::int64_t *row_ptr;
    const std::int64_t *packed_row_ptr;
    const std::int32_t *col_idx;
    const std::uint8_t *packed;
    const float *scales;
    const float *offsets;
    const float *g;
    float *out;
    std::int64_t g_ld, out_ld;
    std::int64_t row_begin, rows, cols;
    int n, policy;
    float alpha, beta;
    std::int32_t *starts; // [ranges + 1][rows]
    int *status;
    int ranges, width;    // ranges of `width` genes
    int tiles, tile_rows; // tiles of `tile_rows` rows
    int start_rows;       // rows per CTA of the pass over the indices
    int pairs;            // column tiles x tiles x ranges
    int out_vector;       // rows of G' take 16-byte reductions
    int scale_output;     // the pass over the indices also sets G' to beta * G'
};

// starts[j][row] for every range j, and G' = beta * G'.  An entry whose range lies beyond the one of the entry before it is a
// candidate for the start of every range in between; the earliest candidate wins.  The entries of the CTA's rows are one
// stretch of the CSR arrays, which the warps take 256 at a time whatever rows they belong to.
constexpr int kStartRows = 32;  // most rows of a CTA
constexpr int kStartSteps = 8;

// gene / width: the product with 2^32 / width, rounded up, is at most one too high for genes below 2^31 and widths to 512
__device__ __forceinline__ unsigned range_of(unsigned gene, unsigned width, unsigned reciprocal) {
    const unsigned q = width == 1u ? gene : __umulhi(gene, reciprocal);
    return q * width > gene ? q - 1u : q;
}

__global__ void __launch_bounds__(kTileThreads) transpose_starts_kernel(const tiled_transpose_params p) {
    extern __shared__ int transpose_starts[]; // [ranges + 1][kStartRows + 1]
    __shared__ int row_start[kStartRows + 1]; // from the CTA's first entry
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && threadIdx.x == 0 && p.status != nullptr) *p.status = 0;
    const std::int64_t row0 = static_cast<std::int64_t>(blockIdx.x) * p.start_rows;
    if (row0 < p.rows) {
        const int rows = static_cast<int>(min(static_cast<std::int64_t>(p.start_rows), p.rows - row0));
        const std::int64_t base = __ldg(p.row_ptr + p.row_begin + row0);
        if (threadIdx.x <= rows) row_start[threadIdx.x] = static_cast<int>(__ldg(p.row_ptr + p.row_begin + row0 + threadIdx.x) - base);
        __syncthreads();
        for (int j = warp; j <= p.ranges; j += kTileWarps)
            if (lane < rows) transpose_starts[j * (kStartRows + 1) + lane] = row_start[lane + 1] - row_start[lane];
        __syncthreads();
        const int end = row_start[rows];
        const std::int32_t *cols = p.col_idx + base;
        const unsigned reciprocal = 0xffffffffu / static_cast<unsigned>(p.width) + 1u;
        int r = 0, first = 0, next = row_start[1]; // row of the lane's entry, and where it starts and ends
        for (int at = warp * (32 * kStartSteps); at < end; at += kTileWarps * 32 * kStartSteps) {
            unsigned gene[kStartSteps];
#pragma unroll
            for (int u = 0; u < kStartSteps; ++u) gene[u] = at + u * 32 + lane < end ? static_cast<unsigned>(__ldg(cols + at + u * 32 + lane)) : 0u;
            unsigned before = at > 0 ? range_of(static_cast<unsigned>(__ldg(cols + at - 1)), p.width, reciprocal) : 0u;
#pragma unroll
            for (int u = 0; u < kStartSteps; ++u) {
                const int e = at + u * 32 + lane;
                const unsigned range = range_of(gene[u], p.width, reciprocal);
                unsigned last = __shfl_up_sync(0xffffffffu, range, 1);
                if (lane == 0) last = before;
                before = __shfl_sync(0xffffffffu, range, 31);
                if (e >= end) continue;
                while (e >= next) {
                    first = next;
                    next = row_start[++r + 1];
                }
                if (range > last || e == first) {
                    const int reach = min(static_cast<int>(range), p.ranges - 1);
                    for (int j = e == first ? 0 : static_cast<int>(last) + 1; j <= reach; ++j) atomicMin(&transpose_starts[j * (kStartRows + 1) + r], e - first);
                }
            }
        }
        __syncthreads();
        for (int j = warp; j <= p.ranges; j += kTileWarps)
            if (lane < rows) p.starts[static_cast<std::int64_t>(j) * p.rows + row0 + lane] = transpose_starts[j * (kStartRows + 1) + lane];
    }
    if (p.scale_output == 0) return;
    const std::int64_t total = p.cols * p.n;
    for (std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * kTileThreads + threadIdx.x; i < total; i += static_cast<std::int64_t>(gridDim.x) * kTileThreads) {
        float *dst = p.out + (i / p.n) * p.out_ld + i % p.n;
        *dst = p.beta == 0.0f ? 0.0f : p.beta * *dst;
    }
}

// v * b + c on both halves, one instruction
__device__ __forceinline__ float2 fma2(float v, float2 b, float2 c) {
    const float2 vv = make_float2(v, v);
    unsigned long long vp, bp, cp;
    memcpy(&vp, &vv, 8);
    memcpy(&bp, &b, 8);
    memcpy(&cp, &c, 8);
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cp) : "l"(vp), "l"(bp));
    memcpy(&c, &cp, 8);
    return c;
}

// Inclusive sum over the CTA's threads; `sums` holds a word per warp.  Ends with every thread past a barrier.
__device__ __forceinline__ int scan_block(int v, int *sums, int *total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, v, off);
        if (lane >= off) v += below;
    }
    __syncthreads();
    if (lane == 31) sums[warp] = v;
    __syncthreads();
    int upto = sums[lane];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int below = __shfl_up_sync(0xffffffffu, upto, off);
        if (lane >= off) upto += below;
    }
    *total = __shfl_sync(0xffffffffu, upto, 31);
    const int below = __shfl_sync(0xffffffffu, upto, warp == 0 ? 0 : warp - 1);
    return v + (warp == 0 ? 0 : below);
}

template<int NC> struct tile_memory {
    float g[(kTileRows + 1) * NC];   // the last row is zero: what padding entries multiply
    std::uint32_t words[kTileWords]; // sorted entries: row of the tile << 8 | code
    int head[kTileGenes];            // entries of a gene counted, then the next free word
    int first[kTileGenes + 1];       // first word of a gene
    float2 meta[kTileGenes];
    int run_end[kTileRows + 1];      // entries of the range in the rows up to and with one
    int run_shift[kTileRows];        // entry of the row minus its place among the range's entries
    std::int64_t entries[kTileRows], codes[kTileRows];
    float row_offset[kTileRows + 1]; // the padding entries' is 0
    int sums[kTileWarps];
};

// NC columns of G at a time (32 or 64).
template<int BITS, int NC>
__global__ void __launch_bounds__(kTileThreads, 1) qcsr_transpose_tiled_kernel(const tiled_transpose_params p) {
    extern __shared__ __align__(16) unsigned char tile_smem[];
    tile_memory<NC> &m = *reinterpret_cast<tile_memory<NC> *>(tile_smem);
    constexpr int kLanes = NC / 4;        // lanes that hold a row, four columns each
    constexpr int kGroups = 32 / kLanes;  // entries a warp reads at once: 2 or 4
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    const int pair0 = static_cast<int>(static_cast<std::int64_t>(p.pairs) * blockIdx.x / gridDim.x);
    const int pair1 = static_cast<int>(static_cast<std::int64_t>(p.pairs) * (blockIdx.x + 1) / gridDim.x);
    int loaded = -1; // (column tile, tile) in shared memory
    int rows = 0, col0 = 0;
    std::int64_t row0 = 0;
    for (int pair = pair0; pair < pair1; ++pair) {
        const int tile = pair / p.ranges, range = pair - tile * p.ranges;
        const int g0 = range * p.width, genes = static_cast<int>(min(static_cast<std::int64_t>(p.width), p.cols - g0));
        __syncthreads();
        if (tile != loaded) {
            loaded = tile;
            col0 = tile / p.tiles * NC;
            row0 = static_cast<std::int64_t>(tile % p.tiles) * p.tile_rows;
            rows = static_cast<int>(min(static_cast<std::int64_t>(p.tile_rows), p.rows - row0));
            for (int i = tid; i < (kTileRows + 1) * NC; i += kTileThreads) {
                const int r = i / NC, c = col0 + i % NC;
                m.g[i] = r < rows && c < p.n ? p.alpha * __ldg(p.g + (p.row_begin + row0 + r) * p.g_ld + c) : 0.0f;
            }
            if (tid == 0) m.row_offset[kTileRows] = 0.0f;
            if (tid < rows) {
                const std::int64_t row = p.row_begin + row0 + tid;
                m.entries[tid] = __ldg(p.row_ptr + row);
                m.codes[tid] = p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row) : m.entries[tid];
                m.row_offset[tid] = row_policy && p.offsets != nullptr ? __ldg(p.offsets + row) : 0.0f;
            }
        }
        if (tid < genes)
            m.meta[tid] = make_float2(p.scales != nullptr ? __ldg(p.scales + g0 + tid) : 1.0f,
                                      !row_policy && p.offsets != nullptr ? __ldg(p.offsets + g0 + tid) : 0.0f);
        int count = 0, first_entry = 0;
        if (tid < rows) {
            const std::int32_t *starts = p.starts + static_cast<std::int64_t>(range) * p.rows + row0 + tid;
            first_entry = __ldg(starts);
            count = __ldg(starts + p.rows) - first_entry;
        }
        int total;
        const int upto = scan_block(count, m.sums, &total);
        if (tid < rows) {
            m.run_end[tid + 1] = upto;
            m.run_shift[tid] = first_entry - (upto - count);
        }
        if (tid == 0) m.run_end[0] = 0;
        __syncthreads();

        for (int taken = 0; taken < total; taken += kBatch) {
            // entries [taken, taken + kBatch) of the range, in equal parts to the warps: counted per gene, and kept in registers
            // as {gene of the range, row of the tile, code} for the placing
            const int batch_end = min(total, taken + kBatch), share = (batch_end - taken + kTileWarps - 1) / kTileWarps;
            const int from = min(batch_end, taken + warp * share), to = min(batch_end, from + share);
            if (tid < kTileGenes) m.head[tid] = 0;
            __syncthreads();
            int r = 0; // row of the lane's entry
            {
                int lo = 0, hi = rows - 1; // last row that starts at or before `from`
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (m.run_end[mid] <= from) lo = mid;
                    else hi = mid - 1;
                }
                r = lo;
            }
            std::uint32_t mine[kStepsPerWarp];
#pragma unroll
            for (int i0 = 0; i0 < kStepsPerWarp; i0 += kStepGroup) {
                std::uint32_t gene[kStepGroup], code[kStepGroup];
#pragma unroll
                for (int i = 0; i < kStepGroup; ++i) {
                    const int q = from + (i0 + i) * 32 + lane;
                    gene[i] = code[i] = 0u;
                    mine[i0 + i] = kNoEntry;
                    if (q < to) {
                        while (q >= m.run_end[r + 1]) ++r;
                        const int e = q + m.run_shift[r];
                        gene[i] = static_cast<std::uint32_t>(__ldg(p.col_idx + m.entries[r] + e));
                        code[i] = __ldg(p.packed + m.codes[r] + (BITS == 8 ? e : e >> 1));
                        mine[i0 + i] = static_cast<std::uint32_t>(r) << 8 | (BITS == 4 ? static_cast<std::uint32_t>(e & 1) : 0u);
                    }
                }
#pragma unroll
                for (int i = 0; i < kStepGroup; ++i) {
                    if (mine[i0 + i] == kNoEntry) continue;
                    const std::uint32_t local = gene[i] - static_cast<std::uint32_t>(g0);
                    const std::uint32_t c = BITS == 8 ? code[i] : (mine[i0 + i] & 1u) ? code[i] >> 4 : code[i] & 0xfu;
                    const std::uint32_t row = mine[i0 + i] >> 8;
                    mine[i0 + i] = local << 18 | row << 8 | c;
                    if (local < static_cast<std::uint32_t>(genes)) {
                        atomicAdd(&m.head[local], 1);
                    } else { // the row does not ascend: this gene belongs to another range
                        mine[i0 + i] = kNoEntry;
                        const float offset = row_policy ? m.row_offset[row] : p.offsets != nullptr ? __ldg(p.offsets + gene[i]) : 0.0f;
                        const float value = fmaf(static_cast<float>(c), p.scales != nullptr ? __ldg(p.scales + gene[i]) : 1.0f, offset);
                        for (int c0 = 0; c0 < NC && col0 + c0 < p.n; ++c0) atomicAdd(p.out + gene[i] * p.out_ld + col0 + c0, value * m.g[row * NC + c0]);
                    }
                }
            }
            __syncthreads();
            const int own = tid < kTileGenes ? m.head[tid] : 0, padded = (own + 3) & ~3;
            int all;
            const int end = scan_block(padded, m.sums, &all);
            if (tid < kTileGenes) {
                m.first[tid] = end - padded;
                m.head[tid] = end - padded;
                for (int k = end - padded + own; k < end; ++k) m.words[k] = static_cast<std::uint32_t>(kTileRows) << 8;
                if (tid == kTileGenes - 1) m.first[kTileGenes] = end;
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < kStepsPerWarp; ++i)
                if (mine[i] != kNoEntry) m.words[atomicAdd(&m.head[mine[i] >> 18], 1)] = mine[i] & 0x3ffffu;
            __syncthreads();
            // a warp per gene: kGroups entries at a time, a lane holding four columns
            const int group = lane / kLanes;
            const unsigned char *g_lane = reinterpret_cast<const unsigned char *>(m.g) + (lane % kLanes) * 16;
            for (int gene = warp; gene < genes; gene += kTileWarps) {
                const int first = m.first[gene], last = m.first[gene + 1];
                if (first == last) continue;
                const float2 meta = m.meta[gene];
                float2 acc0 = make_float2(0.0f, 0.0f), acc1 = acc0;
                const auto add = [&](std::uint32_t word) {
                    const float value = fmaf(static_cast<float>(static_cast<int>(word & 0xffu)), meta.x, row_policy ? m.row_offset[word >> 8] : meta.y);
                    const float4 row = *reinterpret_cast<const float4 *>(g_lane + (NC == 64 ? word & ~0xffu : (word & ~0xffu) >> 1));
                    acc0 = fma2(value, make_float2(row.x, row.y), acc0);
                    acc1 = fma2(value, make_float2(row.z, row.w), acc1);
                };
                int k = first;
                if constexpr (kGroups == 2) {
                    for (; k + 8 <= last; k += 8) {
                        const uint4 w = *reinterpret_cast<const uint4 *>(m.words + k + 4 * group);
                        add(w.x); add(w.y); add(w.z); add(w.w);
                    }
                    if (k < last) {
                        const uint2 w = *reinterpret_cast<const uint2 *>(m.words + k + 2 * group);
                        add(w.x); add(w.y);
                    }
                } else {
                    for (; k + 8 <= last; k += 8) {
                        const uint2 w = *reinterpret_cast<const uint2 *>(m.words + k + 2 * group);
                        add(w.x); add(w.y);
                    }
                    if (k < last) add(m.words[k + group]);
                }
                float acc[4] = {acc0.x, acc0.y, acc1.x, acc1.y};
#pragma unroll
                for (int off = kLanes; off < 32; off <<= 1) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
                }
                const int col = col0 + lane * 4;
                if (lane < kLanes && col < p.n) {
                    float *dst = p.out + static_cast<std::int64_t>(g0 + gene) * p.out_ld + col;
                    if (p.out_vector) {
                        atomicAdd(reinterpret_cast<float4 *>(dst), make_float4(acc[0], acc[1], acc[2], acc[3]));
                    } else {
                        for (int c = 0; c < 4 && col + c < p.n; ++c) atomicAdd(dst + c, acc[c]);
                    }
                }
            }
            if (taken + kBatch < total) __syncthreads();
        }
    }
}

template<int BITS, int NC>
cb200_status launch_tiles(const tiled_transpose_params &p, int sm_count, cudaStream_t stream) {
    constexpr int smem = static_cast<int>(sizeof(tile_memory<NC>));
    CB200_CUDA_OK(cudaFuncSetAttribute(qcsr_transpose_tiled_kernel<BITS, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    qcsr_transpose_tiled_kernel<BITS, NC><<<static_cast<unsigned>(std::min(p.pairs, sm_count)), kTileThreads, smem, stream>>>(p);
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

// Fewest ranges the genes take, and most: as many as fill whole waves of CTAs with (column tile, tile, range) pairs.
int fewest_ranges(std::int64_t cols) { return static_cast<int>(std::min<std::int64_t>((cols + kTileGenes - 1) / kTileGenes, kMaxRanges + 1)); }
int ranges_for(std::int64_t cols, int tiles, int sm_count) {
    const int least = fewest_ranges(cols);
    const std::int64_t waves = (static_cast<std::int64_t>(least) * tiles + sm_count - 1) / sm_count;
    return static_cast<int>(std::max<std::int64_t>(least, std::min<std::int64_t>({waves * sm_count / tiles, cols, kMaxRanges})));
}

// The starts of a launch over `rows` rows.  T = column tiles x tiles of 512 rows take at most least + (sm_count - 1) / T ranges
// (ranges_for), and rows <= 512 T: (ranges + 1) * rows is at most (least + 1) * rows + 512 * sm_count.
std::uint64_t starts_bytes(std::int64_t rows, int least, int sm_count) {
    return (static_cast<std::uint64_t>(least + 1) * static_cast<std::uint64_t>(rows) + static_cast<std::uint64_t>(kTileRows) * static_cast<std::uint64_t>(sm_count)) * 4u;
}
// A launch over more rows than the workspace holds the starts of takes them slice by slice.  A slice is dear only
// when it has few tiles: 400,000 x 33,538 at N = 64 take 15.3 ms in four slices (32 MB of starts), 15.1 in 28 (4 MB) and 15.5 in 61.
constexpr std::uint64_t kMostStartsBytes = 32ull << 20;
constexpr std::int64_t kLeastSlice = 8 * kTileRows;
std::int64_t slice_rows(std::int64_t rows, int least, std::uint64_t bytes, int sm_count) {
    if (bytes >= starts_bytes(rows, least, sm_count)) return rows;
    const std::uint64_t fixed = starts_bytes(0, least, sm_count);
    if (bytes < fixed) return 0;
    return static_cast<std::int64_t>((bytes - fixed) / (4u * static_cast<std::uint64_t>(least + 1))) / kTileRows * kTileRows;
}

} // namespace

std::uint64_t qcsr_transpose_tiled_workspace_bytes(std::int64_t rows, std::int64_t cols, int sm_count) {
    if (rows == 0 || cols == 0 || fewest_ranges(cols) > kMaxRanges) return 0u;
    return 256u + std::min(starts_bytes(rows, fewest_ranges(cols), sm_count), kMostStartsBytes);
}

cb200_status launch_qcsr_transpose_tiled(const qcsr_view &x, const dense_args &d, std::int64_t row_begin, std::int64_t row_end,
                                         void *workspace, std::uint64_t workspace_bytes, int sm_count, cudaStream_t stream, bool *taken) {
    *taken = false;
    const std::int64_t rows = row_end - row_begin;
    if (rows <= 0 || x.nnz == 0 || workspace == nullptr || (x.bits == 4 && x.packed_row_ptr == nullptr)) return CB200_STATUS_SUCCESS;
    const int least = fewest_ranges(x.cols);
    if (least > kMaxRanges || workspace_bytes <= 256u || x.cols > (1ll << 21)) return CB200_STATUS_SUCCESS;
    const std::int64_t most = slice_rows(rows, least, std::min(workspace_bytes - 256u, kMostStartsBytes), sm_count);
    if (most < std::min(rows, kLeastSlice)) return CB200_STATUS_SUCCESS;
    // equal slices, of whole tiles but for the last
    const std::int64_t slices = (rows + most - 1) / most;
    const std::int64_t slice = slices == 1 ? rows : std::min(most, ((rows + slices - 1) / slices + kTileRows - 1) / kTileRows * kTileRows);
    const int nc = d.n <= 32 ? 32 : 64;
    const int column_tiles = static_cast<int>((d.n + nc - 1) / nc);
    {
        const std::int64_t tiles = (slice + kTileRows - 1) / kTileRows;
        const std::int64_t tile_rows = (slice + tiles - 1) / tiles;
        const double per_row = static_cast<double>(x.nnz) / static_cast<double>(x.rows);
        // a gene needs a few entries per tile to be worth its turn, and the sort a few thousand entries to be worth its barriers
        if (per_row * static_cast<double>(rows) < 50000.0 || per_row * static_cast<double>(tile_rows) < 3.0 * static_cast<double>(x.cols)) return CB200_STATUS_SUCCESS;
        if (static_cast<std::int64_t>(column_tiles) * tiles * kMaxRanges > 0x7fffffff) return CB200_STATUS_SUCCESS;
    }
    tiled_transpose_params p{};
    p.row_ptr = x.row_ptr; p.packed_row_ptr = x.packed_row_ptr; p.col_idx = x.col_idx; p.packed = x.packed; p.scales = x.scales;
    p.offsets = x.offsets; p.g = static_cast<const float *>(d.dense); p.out = d.out; p.g_ld = d.dense_ld; p.out_ld = d.out_ld;
    p.cols = x.cols; p.n = static_cast<int>(d.n); p.policy = x.policy; p.alpha = d.alpha; p.beta = d.beta;
    p.status = static_cast<int *>(workspace);
    p.starts = reinterpret_cast<std::int32_t *>(static_cast<unsigned char *>(workspace) + 256);
    p.out_vector = reinterpret_cast<std::uintptr_t>(d.out) % 16u == 0u && d.out_ld % 4 == 0 && d.n % 4 == 0 ? 1 : 0;
    *taken = true;
    for (std::int64_t first = row_begin; first < row_end; first += slice) {
        p.row_begin = first;
        p.rows = std::min(slice, row_end - first);
        p.tiles = static_cast<int>((p.rows + kTileRows - 1) / kTileRows);
        p.tile_rows = static_cast<int>((p.rows + p.tiles - 1) / p.tiles);
        p.ranges = ranges_for(x.cols, p.tiles * column_tiles, sm_count);
        p.width = static_cast<int>((x.cols + p.ranges - 1) / p.ranges);
        p.ranges = static_cast<int>((x.cols + p.width - 1) / p.width);
        p.pairs = column_tiles * p.tiles * p.ranges;
        p.scale_output = first == row_begin ? 1 : 0;
        const std::size_t smem = static_cast<std::size_t>(p.ranges + 1) * (kStartRows + 1) * sizeof(int);
        if (smem > 48u * 1024u)
            CB200_CUDA_OK(cudaFuncSetAttribute(transpose_starts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
        p.start_rows = p.rows >= 32ll * sm_count ? kStartRows : 8;
        const unsigned grid = static_cast<unsigned>(std::max<std::int64_t>((p.rows + p.start_rows - 1) / p.start_rows, sm_count));
        transpose_starts_kernel<<<grid, kTileThreads, smem, stream>>>(p);
        count_launch();
        CB200_CUDA_OK(cudaGetLastError());
        cb200_status st;
        if (x.bits == 8) st = nc == 32 ? launch_tiles<8, 32>(p, sm_count, stream) : launch_tiles<8, 64>(p, sm_count, stream);
        else st = nc == 32 ? launch_tiles<4, 32>(p, sm_count, stream) : launch_tiles<4, 64>(p, sm_count, stream);
        if (st != CB200_STATUS_SUCCESS) return st;
    }
    return CB200_STATUS_SUCCESS;
}

} // namespace cb200
