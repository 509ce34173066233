// Fused dequantise + SpMM over a quantized CSR matrix:  Y = alpha * deq(X) * W + beta * Y, fp32 products, codes and indices
// read at launch; and the dispatch of the forward schedules.
//
// The Cellerator reference has no fused kernel for this layout; it decodes to a float array
// (include/Cellerator/quantized/portable_dequantize_kernel.cuh:7-19) and then runs
// csr_spmm_fwd_kernel_ (src/compute/sparse/project/kernels/csr_spmm_fwd_kernel_.cuh:1-22), one
// thread per (row, output column), every thread re-reading the row.
#include "kernels.cuh"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

namespace cb200 {
namespace {

struct fwd_params {
    const std::int64_t *row_ptr;
    const std::int64_t *packed_row_ptr;
    const std::int32_t *col_idx;
    const std::uint8_t *packed;
    const float *scales;
    const float *offsets;
    const void *w;
    float *y;
    std::int64_t w_ld, y_ld;
    std::int64_t row_begin, row_end;
    int n;
    int policy;
    float alpha, beta;
    const float *bias;
    int epilogue;
    int lanes;      // lanes that serve one entry, a power of two
    int group_rows, warps; // rows and warps per CTA
    union {
        unsigned full_groups; // CTAs of that many rows; the others take a quarter of them
        int short_rows;       // a warp per row: rows of fewer than 64 entries on average
    };
    int parts;       // sums of parts the shared memory of a CTA holds
    int packed_rows; // W is the re-laid copy: rows at a pitch of 16 bytes
    int out_vector; // rows of Y can be written 16 bytes at a time
    int *status;    // status word of the launch (this kernel waits on nothing: it clears it)
};

// Code of entry `local` (index within its row) for a row whose packed bytes start at `row_bytes`.
template<int BITS>
__device__ __forceinline__ unsigned load_code(const std::uint8_t *row_bytes, std::int64_t local) {
    if constexpr (BITS == 8) {
        return __ldg(row_bytes + local);
    } else {
        const unsigned byte = __ldg(row_bytes + (local >> 1));
        return (local & 1) ? (byte >> 4) : (byte & 0xfu);
    }
}

// A lane's V consecutive columns of a W row, as fp32 (bf16 widens exactly).
template<typename WT, int V>
struct w_slice {
    static constexpr int bytes = V * static_cast<int>(sizeof(WT));
    static constexpr int words = bytes >= 4 ? bytes / 4 : 1;
    std::uint32_t r[words];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < words; ++i) r[i] = 0u;
    }
    __device__ __forceinline__ void load(const unsigned char *src) {
        // volatile: a batch of loads is issued before the first of its multiplies
        if constexpr (bytes == 16)
            asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "l"(src));
        else if constexpr (bytes == 8) asm volatile("ld.global.nc.v2.b32 {%0, %1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "l"(src));
        else if constexpr (bytes == 4) asm volatile("ld.global.nc.b32 %0, [%1];" : "=r"(r[0]) : "l"(src));
        else {
            unsigned short t;
            asm volatile("ld.global.nc.b16 %0, [%1];" : "=h"(t) : "l"(src));
            r[0] = t;
        }
    }
    // acc += v * w; pairs of columns with the two-wide fp32 FMA (half the issue slots)
    __device__ __forceinline__ void fma_into(float (&acc)[V], float v) const {
        if constexpr (V == 1) {
            acc[0] = fmaf(v, sizeof(WT) == 2 ? __uint_as_float(r[0] << 16) : __uint_as_float(r[0]), acc[0]);
        } else {
            const float2 vv = make_float2(v, v);
            unsigned long long vp;
            memcpy(&vp, &vv, 8);
#pragma unroll
            for (int i = 0; i < V; i += 2) {
                float2 b;
                if constexpr (sizeof(WT) == 2) bf16x2_to_f32(r[i / 2], b.x, b.y);
                else b = make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1]));
                float2 a = make_float2(acc[i], acc[i + 1]);
                unsigned long long ap, bp;
                memcpy(&ap, &a, 8);
                memcpy(&bp, &b, 8);
                asm volatile("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(ap) : "l"(vp), "l"(bp));
                memcpy(&a, &ap, 8);
                acc[i] = a.x;
                acc[i + 1] = a.y;
            }
        }
    }
};

constexpr int kGatherRuns = 2;      // runs of 32 entries a warp decodes at a time
constexpr int kSegment = 32 * kGatherRuns;
constexpr int kGatherMaxWarps = 16; // most warps per CTA
constexpr int kGatherMaxRows = 8;   // most rows per CTA
constexpr int kGatherParts = 64;    // most sums of parts the shared memory of a CTA holds
constexpr int kRowParts = 16;       // most parts of a row
constexpr int kPartEntries = 128;   // entries of a part, for rows of up to 16 of them

// Entries per part of a row of `len` entries (a multiple of 16): a function of the length alone.
__device__ __forceinline__ int part_size(int len) {
    if (len <= kPartEntries) return kPartEntries;
    const int parts = min(kRowParts, (len + kPartEntries - 1) / kPartEntries);
    return ((len + parts - 1) / parts + 15) / 16 * 16;
}

// The stream of entries is read once: it must not push rows of W out of L1.
__device__ __forceinline__ std::int32_t load_index_once(const std::int32_t *src) {
    std::int32_t v;
    asm("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(src));
    return v;
}

// Rows of W gathered straight into registers, for any N and any leading dimension.
//
// A row of X is cut into parts by its length alone (about 128 entries each, 16 parts at most), and the row's sum is the sum of
// its parts in order.  A warp decodes 64 entries at a time, two per lane with coalesced loads (the raw pairs of the next 64 are
// in flight meanwhile), into a staging line of {gene, value}; then a group of `lanes` lanes serves one entry, a lane holding V
// columns (16 bytes where N and the operand's alignment allow), so one load instruction brings 32 / lanes rows of W.
//
// The order of a part's sum follows from N and W's type alone (summing_lanes): entry e belongs to class e modulo C, a class is
// summed in order, the classes pairwise.  With 16-byte slices the classes are the C groups of lanes; narrower ones leave
// 32 / lanes groups, each of which keeps SETS = C * lanes / 32 sums.  So a row's sum has the same bits whatever rows stand
// beside it, whichever of the two kernels below runs, and whether W was re-laid: in a shard, a chunk, a routed call.
//
// What bounds it: rows of W out of L2 (33,538 x 64 bf16: 12.4 TB/s at 125,000 rows of 1,800 entries, 96 Gnnz/s) or, where W
// fits L1, instruction issue (2,000 x 32 fp32, 20,000 rows of 360: 82 Gnnz/s).  Before, a row was one warp's work from end to
// end (600 us for 4,099 x 1,800 at N = 64, now 110: the longest row decided) or one lane group's in the gene-tiled kernel (820
// us for 20,000 x 340 at N = 32, now 84: 40 CTAs for 148 SMs), and a width that is no power of two went column by column
// through 2-byte loads (2.6 ms for 4,099 x 1,800 at N = 50 bf16, now 118 us).
template<int BITS, typename WT, int V, int SETS, int RUNS>
struct gather_warp {
    static constexpr int SEG = 32 * RUNS; // entries decoded at a time
    static constexpr int U = V * sizeof(WT) > 4 ? 4 : 8; // rows of W in flight per lane
    static_assert(U % SETS == 0 && SETS * V * sizeof(WT) <= 16, "a batch holds every class equally often");
    // 32 x 32 -> 64-bit products for the addresses; operands whose rows lie 4 GB or more apart are served with V == 1
    using stride_t = typename std::conditional<V == 1, std::uint64_t, std::uint32_t>::type;

    const fwd_params &p;
    int2 *stage;
    int lane, lanes, per_step, group, col;
    bool holds; // fewer than V of the columns, where W was re-laid
    bool row_policy;
    const unsigned char *wcol;
    stride_t w_row_bytes;
    float acc[SETS][V];
    int gene[RUNS];
    unsigned code[RUNS];
    float scale[RUNS], offset[RUNS];

    __device__ __forceinline__ gather_warp(const fwd_params &params, int2 *line) : p(params), stage(line) {
        lane = threadIdx.x & 31;
        lanes = p.lanes;
        per_step = 32 / lanes; // both powers of two
        group = lane / lanes;
        col = (blockIdx.y * 32 + lane % lanes) * V;
        holds = col < p.n;
        row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
        wcol = static_cast<const unsigned char *>(p.w) + (holds ? col : 0) * static_cast<int>(sizeof(WT));
        w_row_bytes = static_cast<stride_t>(p.w_ld * static_cast<std::int64_t>(sizeof(WT)));
        clear();
    }
    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int k = 0; k < SETS; ++k) {
#pragma unroll
            for (int i = 0; i < V; ++i) acc[k][i] = 0.0f;
        }
    }
    __device__ __forceinline__ const unsigned char *w_at(int g) const {
        return wcol + static_cast<std::uint64_t>(static_cast<std::uint32_t>(g)) * w_row_bytes;
    }
    // Entries [at, at + SEG) of a row that ends, for this warp, at `to`.  Lanes past the end read the last entry again (no
    // branches in the loop); the multiply leaves them out.
    __device__ __forceinline__ void fetch_raw(const std::int32_t *cols, const std::uint8_t *codes, int at, int to) {
        if (at >= to) return;
        cols += at;
        codes += BITS == 8 ? at : at >> 1; // `at` is even
        if (at + SEG <= to) {
#pragma unroll
            for (int i = 0; i < RUNS; ++i) {
                gene[i] = load_index_once(cols + lane + i * 32);
                code[i] = load_code<BITS>(codes, lane + i * 32);
            }
        } else {
#pragma unroll
            for (int i = 0; i < RUNS; ++i) {
                const int e = min(lane + i * 32, to - at - 1);
                gene[i] = load_index_once(cols + e);
                code[i] = load_code<BITS>(codes, e);
            }
        }
    }
    __device__ __forceinline__ void fetch_meta(std::int64_t row, int at, int to) {
        if (at >= to) return;
        if (p.scales != nullptr && p.offsets != nullptr && !row_policy) {
#pragma unroll
            for (int i = 0; i < RUNS; ++i) {
                scale[i] = __ldg(p.scales + gene[i]);
                offset[i] = __ldg(p.offsets + gene[i]);
            }
        } else {
            const float row_offset = (row_policy && p.offsets != nullptr) ? __ldg(p.offsets + row) : 0.0f;
#pragma unroll
            for (int i = 0; i < RUNS; ++i) {
                scale[i] = p.scales != nullptr ? __ldg(p.scales + gene[i]) : 1.0f;
                offset[i] = (!row_policy && p.offsets != nullptr) ? __ldg(p.offsets + gene[i]) : row_offset;
            }
        }
    }
    __device__ __forceinline__ void put() {
#pragma unroll
        for (int i = 0; i < RUNS; ++i)
            stage[i * 32 + lane] = make_int2(gene[i], __float_as_int(fmaf(static_cast<float>(code[i]), scale[i], offset[i])));
    }
    // acc += the `count` staged entries
    __device__ __forceinline__ void multiply(int count) {
        const int batch = U * per_step; // entries per batch of loads
        int done = 0;
        for (; done + batch <= count; done += batch) {
            w_slice<WT, V> w[U];
            float v[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int2 e = stage[done + u * per_step + group];
                v[u] = __int_as_float(e.y);
                w[u].load(w_at(e.x));
            }
#pragma unroll
            for (int u = 0; u < U; ++u) w[u].fma_into(acc[u % SETS], v[u]);
        }
        constexpr int T = U / 2 > SETS ? U / 2 : SETS;
        for (; done < count; done += T * per_step) { // entries past the end add nothing
            w_slice<WT, V> w[T];
            float v[T];
#pragma unroll
            for (int u = 0; u < T; ++u) {
                const int src = done + u * per_step + group;
                const int2 e = stage[min(src, count - 1)];
                v[u] = src < count ? __int_as_float(e.y) : 0.0f;
                w[u].load(w_at(e.x));
            }
#pragma unroll
            for (int u = 0; u < T; ++u) {
                if (done + u * per_step + group >= count) w[u].zero();
                w[u].fma_into(acc[u % SETS], v[u]);
            }
        }
    }
    // the classes' sums together, in acc[0] of every lane group
    __device__ __forceinline__ void reduce() {
        for (int off = lanes; off < 32; off <<= 1) {
#pragma unroll
            for (int k = 0; k < SETS; ++k) {
#pragma unroll
                for (int i = 0; i < V; ++i) acc[k][i] += __shfl_xor_sync(0xffffffffu, acc[k][i], off);
            }
        }
#pragma unroll
        for (int step = 1; step < SETS; step <<= 1) {
#pragma unroll
            for (int k = 0; k < SETS; k += 2 * step) {
#pragma unroll
                for (int i = 0; i < V; ++i) acc[k][i] += acc[k + step][i];
            }
        }
    }
    __device__ __forceinline__ void write_row(std::int64_t row, float (&v)[V]) const {
        if (!holds || lane >= lanes) return;
        float *out = p.y + row * p.y_ld + col;
#pragma unroll
        for (int i = 0; i < V; ++i) v[i] *= p.alpha;
        if (V >= 4 && p.out_vector) {
            if (p.beta != 0.0f) {
                float4 o[(V + 3) / 4];
#pragma unroll
                for (int i = 0; i < V / 4; ++i) o[i] = *reinterpret_cast<const float4 *>(out + 4 * i);
#pragma unroll
                for (int i = 0; i < V / 4; ++i) {
                    v[4 * i + 0] = fmaf(p.beta, o[i].x, v[4 * i + 0]); v[4 * i + 1] = fmaf(p.beta, o[i].y, v[4 * i + 1]);
                    v[4 * i + 2] = fmaf(p.beta, o[i].z, v[4 * i + 2]); v[4 * i + 3] = fmaf(p.beta, o[i].w, v[4 * i + 3]);
                }
            }
            if (p.epilogue != CB200_EPILOGUE_NONE) {
#pragma unroll
                for (int i = 0; i < V; ++i) v[i] = finish_output(v[i], p.bias, col + i, p.epilogue);
            }
#pragma unroll
            for (int i = 0; i < V / 4; ++i)
                *reinterpret_cast<float4 *>(out + 4 * i) = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
        } else {
#pragma unroll
            for (int i = 0; i < V; ++i) {
                if (col + i >= p.n) break;
                if (p.beta != 0.0f) v[i] = fmaf(p.beta, out[i], v[i]);
                out[i] = finish_output(v[i], p.bias, col + i, p.epilogue);
            }
        }
    }
};

// A warp per row: no tables, no barriers.  For rows of a few entries (RUNS == 1: 32 at a time) and narrow operands, where the
// other kernel's start and end cost more than the entries.
template<int BITS, typename WT, int V, int SETS, int RUNS>
__global__ void __launch_bounds__(128, 8) qcsr_fwd_row_kernel(const fwd_params p) {
    constexpr int SEG = 32 * RUNS;
    __shared__ __align__(16) int2 staging[4][SEG];
    const int warp = threadIdx.x >> 5;
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && p.status != nullptr) *p.status = 0;
    const std::int64_t row = p.row_begin + static_cast<std::int64_t>(blockIdx.x) * 4 + warp;
    if (row >= p.row_end) return;
    gather_warp<BITS, WT, V, SETS, RUNS> g(p, staging[warp]);
    const std::int64_t start = __ldg(p.row_ptr + row);
    const int len = static_cast<int>(__ldg(p.row_ptr + row + 1) - start);
    const std::int32_t *cols = p.col_idx + start;
    const std::uint8_t *codes = p.packed + (p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row) : start);
    const int share = part_size(len);
    float total[V];
    int at = 0, to = min(len, share);
    g.fetch_raw(cols, codes, at, to);
    g.fetch_meta(row, at, to);
    for (bool first = true;;) {
        g.put();
        const int count = min(SEG, to - at);
        const bool part_done = at + SEG >= to;
        at = part_done ? to : at + SEG;
        if (part_done) to = min(len, to + share);
        g.fetch_raw(cols, codes, at, to);
        __syncwarp();
        g.multiply(count);
        g.fetch_meta(row, at, to);
        __syncwarp();
        if (!part_done) continue;
        g.reduce();
#pragma unroll
        for (int i = 0; i < V; ++i) total[i] = first ? g.acc[0][i] : total[i] + g.acc[0][i];
        first = false;
        g.clear();
        if (at >= len) break;
    }
    g.write_row(row, total);
}

// A CTA owns `group_rows` consecutive rows and deals their parts to its warps, so that a long row does not hold up the
// others; sums of parts meet in shared memory.
// SHORT_END: the CTAs from p.full_groups on take a quarter of the rows.
template<int BITS, typename WT, int V, int SETS, bool SHORT_END>
__global__ void __launch_bounds__(kGatherMaxWarps * 32, 2) qcsr_fwd_gather_kernel(const fwd_params p) {
    __shared__ std::int64_t row_start[kGatherMaxRows], code_start[kGatherMaxRows];
    __shared__ int row_len[kGatherMaxRows], row_share[kGatherMaxRows], first_part[kGatherMaxRows + 1];
    extern __shared__ __align__(16) int2 staging[];         // [warp][64], then the sums
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    float *sums = reinterpret_cast<float *>(staging + warps * kSegment); // [p.parts][V][lanes]
    std::int64_t row0 = p.row_begin + static_cast<std::int64_t>(blockIdx.x) * p.group_rows;
    int most_rows = p.group_rows;
    if constexpr (SHORT_END)
        if (blockIdx.x >= p.full_groups) {
            most_rows = p.group_rows >> 2;
            row0 = p.row_begin + static_cast<std::int64_t>(p.full_groups) * p.group_rows + static_cast<std::int64_t>(blockIdx.x - p.full_groups) * most_rows;
        }
    const int rows = static_cast<int>(min(static_cast<std::int64_t>(most_rows), p.row_end - row0));
    if (warp == 0) {
        int len = 0;
        if (lane < rows) {
            const std::int64_t start = __ldg(p.row_ptr + row0 + lane);
            len = static_cast<int>(__ldg(p.row_ptr + row0 + lane + 1) - start);
            row_start[lane] = start;
            row_len[lane] = len;
            code_start[lane] = p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row0 + lane) : start;
        }
        const int share = part_size(len);
        if (lane < rows) row_share[lane] = share;
        int upto = lane < rows ? (len <= share ? 1 : (len + share - 1) / share) : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int below = __shfl_up_sync(0xffffffffu, upto, off);
            if (lane >= off) upto += below;
        }
        if (lane == 0) first_part[0] = 0;
        if (lane < rows) first_part[lane + 1] = upto;
    }
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && p.status != nullptr) *p.status = 0;
    __syncthreads();
    gather_warp<BITS, WT, V, SETS, kGatherRuns> g(p, staging + warp * kSegment);
    const int lanes = g.lanes;
    // rounds of rows whose parts the shared sums hold (one row's always do)
    for (int ra = 0; ra < rows;) {
        const int base = first_part[ra];
        int rb = ra + 1;
        while (rb < rows && first_part[rb + 1] - base <= p.parts) ++rb;
        const int end = first_part[rb];
        int part = base + warp, r = ra, at = 0, to = 0; // a part of a row: entries [at, to) of row r
        const auto open_part = [&]() {
            r = __popc(__ballot_sync(0xffffffffu, lane < rows && first_part[lane] <= part)) - 1;
            at = (part - first_part[r]) * row_share[r];
            to = min(row_len[r], at + row_share[r]);
        };
        if (part < end) {
            open_part();
            g.fetch_raw(p.col_idx + row_start[r], p.packed + code_start[r], at, to);
            g.fetch_meta(row0 + r, at, to);
        }
        while (part < end) {
            g.put();
            const int count = min(kSegment, to - at), r_now = r, part_now = part;
            // the next 64 entries of the part, or the first of this warp's next part
            const bool part_done = at + kSegment >= to;
            if (!part_done) {
                at += kSegment;
            } else {
                part += warps;
                if (part < end) open_part();
                else at = to;
            }
            g.fetch_raw(p.col_idx + row_start[r], p.packed + code_start[r], at, to);
            __syncwarp();
            g.multiply(count);
            g.fetch_meta(row0 + r, at, to);
            if (part_done) {
                g.reduce();
                if (first_part[r_now + 1] - first_part[r_now] == 1) {
                    g.write_row(row0 + r_now, g.acc[0]);
                } else if (lane < lanes) {
#pragma unroll
                    for (int i = 0; i < V; ++i) sums[((part_now - base) * V + i) * lanes + lane] = g.acc[0][i];
                }
                g.clear();
            }
            __syncwarp();
        }
        __syncthreads();
        for (int row = ra + warp; row < rb; row += warps) {
            const int first = first_part[row] - base, last = first_part[row + 1] - base;
            if (last - first == 1) continue;
            float total[V];
#pragma unroll
            for (int i = 0; i < V; ++i) total[i] = sums[(first * V + i) * lanes + (lane & (lanes - 1))];
            for (int k = first + 1; k < last; ++k) {
#pragma unroll
                for (int i = 0; i < V; ++i) total[i] += sums[(k * V + i) * lanes + (lane & (lanes - 1))];
            }
            g.write_row(row0 + row, total);
        }
        ra = rb;
        if (ra < rows) __syncthreads();
    }
}

// Rows and warps per CTA for a launch over `rows` rows; *group_rows == 0: a warp per row (none of it touches the order of a
// row's sum).  Measured from 64 to 1,000,000 rows of 24 to 1,800 entries.
//  - About 8,192 entries make a CTA long enough to hide its start and end and short enough to leave many of them
//    (125,000 x 1,800 at N = 64: 2.50 ms with 4 rows, 2.57 with 8, 2.64 with 32).
//  - Where few rows leave the SMs short of CTAs, 16 warps share the longest row (1,024 x 1,800: 0.10 ms, 8 warps 0.14) and
//    fewer rows per CTA keep at least two CTAs per SM (512 x 1,800: 38 us with one, 67 with 8).
//  - Of CTAs of eight warps the last third of a resident wave takes a quarter of the rows each: the launch ends when the
//    longest of them does (20,000 x 2,000 at N = 32: 85 -> 81 us, 10,000 x 4,000 at N = 64: 93 -> 82; a whole wave of them 87
//    and 87, an eighth of the rows each 98 and 98).  Those of 16 warps share few long rows, and gain nothing.
//  - Many rows of a few entries, or of W rows of 32 bytes and less, run with a warp per row (200,000 x 24 at N = 32: 108 us,
//    dealt out by parts 128; 20,000 x 240 at N = 16 bf16: 39 us against 44).
void gather_shape(const qcsr_view &x, std::int64_t rows, std::int64_t w_row_bytes, int sm_count, fwd_params *p) {
    const double mean = static_cast<double>(x.nnz) / static_cast<double>(std::max<std::int64_t>(x.rows, 1));
    p->warps = rows <= 8ll * sm_count || (rows <= 64ll * sm_count && mean >= 512.0) ? kGatherMaxWarps : 8;
    p->group_rows = 0;
    if (rows >= 64ll * sm_count && (mean < 64.0 || w_row_bytes <= 32)) return;
    p->group_rows = 1;
    while (p->group_rows < 8 && 2 * p->group_rows * mean <= 8192.0 && rows >= 4ll * sm_count * p->group_rows) p->group_rows *= 2;
    p->full_groups = static_cast<unsigned>((rows + p->group_rows - 1) / p->group_rows);
    if (p->warps != kGatherMaxWarps && p->group_rows >= 4) { // four CTAs of 64 registers a thread are resident
        const std::int64_t short_end = std::min<std::int64_t>(rows, 4ll * sm_count * p->group_rows / 3);
        p->full_groups = static_cast<unsigned>((rows - short_end) / p->group_rows);
    }
}

// Lanes that serve one entry when a lane holds v columns.
int gather_lanes(int n, int v) {
    int lanes = 1;
    while (lanes < 32 && lanes * v < n) lanes *= 2;
    return lanes;
}
// At least four lanes per entry, or the sums of the 32 / lanes groups cost more to bring together than the wider loads save
// (20,000 x 240, N = 8 bf16: 35 us with 4 lanes of 4 bytes, 40 with one of 16).
int narrowed(int n, int v) {
    while (v > 1 && n <= 3 * v) v /= 2;
    return v;
}
// 32 / the classes of a part's entries: the lanes of the widest slices N allows, re-laid W included.
int summing_lanes(int n, int widest) { return gather_lanes(n, narrowed(n, widest)); }

template<int BITS, typename WT, int V, int SETS>
cb200_status launch_gather(fwd_params p, cudaStream_t stream) {
    const int tile = 32 * V;
    p.lanes = gather_lanes(p.n, V);
    p.out_vector = p.out_vector && p.n % V == 0;
    const std::int64_t rows = p.row_end - p.row_begin;
    const unsigned tiles = static_cast<unsigned>((p.n + tile - 1) / tile);
    if (p.group_rows == 0) {
        const dim3 grid(static_cast<unsigned>((rows + 3) / 4), tiles);
        if (p.short_rows) qcsr_fwd_row_kernel<BITS, WT, V, SETS, 1><<<grid, 128, 0, stream>>>(p);
        else qcsr_fwd_row_kernel<BITS, WT, V, SETS, 2><<<grid, 128, 0, stream>>>(p);
    } else {
        const std::int64_t left = rows - static_cast<std::int64_t>(p.full_groups) * p.group_rows;
        const bool short_end = left > 0;
        const unsigned groups = p.full_groups + static_cast<unsigned>(short_end ? (left + p.group_rows / 4 - 1) / (p.group_rows / 4) : 0);
        p.parts = std::min(kGatherParts, 32 * 1024 / static_cast<int>(V * p.lanes * sizeof(float)));
        const std::size_t smem = static_cast<std::size_t>(p.warps) * kSegment * sizeof(int2) +
                                 static_cast<std::size_t>(p.parts) * V * p.lanes * sizeof(float);
        if (short_end) qcsr_fwd_gather_kernel<BITS, WT, V, SETS, true><<<dim3(groups, tiles), p.warps * 32, smem, stream>>>(p);
        else qcsr_fwd_gather_kernel<BITS, WT, V, SETS, false><<<dim3(groups, tiles), p.warps * 32, smem, stream>>>(p);
    }
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

// W with its rows at a pitch of 16 bytes: a thread writes one 16-byte piece, zeros past column n.
template<typename WT>
__global__ void __launch_bounds__(256) pack_rows_kernel(const WT *w, std::int64_t w_ld, int n, std::int64_t cols, int pieces, uint4 *out) {
    constexpr int V = 16 / static_cast<int>(sizeof(WT));
    const std::int64_t i = static_cast<std::int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= cols * pieces) return;
    const std::int64_t gene = i / pieces;
    const int col = static_cast<int>(i % pieces) * V;
    const WT *src = w + gene * w_ld + col;
    WT piece[V];
#pragma unroll
    for (int k = 0; k < V; ++k) piece[k] = col + k < n ? src[k] : WT(0.0f);
    uint4 v;
    memcpy(&v, piece, 16);
    out[i] = v;
}

// An operand whose rows are no multiple of 16 bytes is gathered in 8-, 4- or 2-byte slices, one entry per load instruction
// where 16-byte slices would serve two to four.  Re-laying it takes a pass over W (5 us at 33,538 x 50 bf16) and takes a
// quarter off the gather (46 -> 62 Gnnz/s there), so it needs a million entries, and more of them than W has rows by far.
bool gather_packs(const qcsr_view &x, std::int64_t n, int dense_dtype) {
    const std::int64_t elem = dense_dtype == CB200_DTYPE_BF16 ? 2 : 4;
    return (n * elem) % 16 != 0 && x.nnz >= (1ll << 20) && x.nnz >= 32 * x.cols;
}

template<int BITS, typename WT, int V>
cb200_status launch_sets(const fwd_params &p, cudaStream_t stream) {
    constexpr int widest = 16 / static_cast<int>(sizeof(WT));
    switch (gather_lanes(p.n, V) / summing_lanes(p.n, widest)) {
    case 8: if constexpr (8 * V <= widest) return launch_gather<BITS, WT, V, 8>(p, stream); [[fallthrough]];
    case 4: if constexpr (4 * V <= widest) return launch_gather<BITS, WT, V, 4>(p, stream); [[fallthrough]];
    case 2: if constexpr (2 * V <= widest) return launch_gather<BITS, WT, V, 2>(p, stream); [[fallthrough]];
    default: return launch_gather<BITS, WT, V, 1>(p, stream);
    }
}

// Columns per lane: the widest slice, up to 16 bytes, that divides N and the rows' alignment.
template<int BITS, typename WT>
cb200_status dispatch_gather(const fwd_params &p, cudaStream_t stream) {
    constexpr int widest = 16 / static_cast<int>(sizeof(WT));
    int v = p.w_ld * static_cast<std::int64_t>(sizeof(WT)) <= 0xffffffffll ? widest : 1;
    while (v > 1 && (p.n % v != 0 || reinterpret_cast<std::uintptr_t>(p.w) % (v * sizeof(WT)) != 0u || p.w_ld % v != 0)) v /= 2;
    if (p.packed_rows) v = widest; // the lane that holds the last columns of a row may hold fewer than v
    v = narrowed(p.n, v);
    switch (v) {
    case 8: if constexpr (widest == 8) return launch_gather<BITS, WT, 8, 1>(p, stream); [[fallthrough]];
    case 4: return launch_sets<BITS, WT, 4>(p, stream);
    case 2: return launch_sets<BITS, WT, 2>(p, stream);
    default: return launch_sets<BITS, WT, 1>(p, stream);
    }
}

} // namespace

std::uint64_t qcsr_gather_workspace_bytes(std::int64_t cols, std::int64_t nnz, std::int64_t n, int dense_dtype) {
    qcsr_view x{};
    x.cols = cols;
    x.nnz = nnz;
    if (!gather_packs(x, n, dense_dtype)) return 256u;
    const std::uint64_t row = (static_cast<std::uint64_t>(n) * (dense_dtype == CB200_DTYPE_BF16 ? 2u : 4u) + 15u) / 16u * 16u;
    return 256u + static_cast<std::uint64_t>(cols) * row;
}

cb200_status launch_qcsr_forward(const qcsr_view &x, const dense_args &d, std::int64_t row_begin,
                                 std::int64_t row_end, fwd_schedule schedule, const void *persistent,
                                 const blocked_layout *blocked, bool split_products, void *workspace,
                                 std::uint64_t workspace_bytes, int sm_count, cudaStream_t stream) {
    if (row_end <= row_begin || d.n == 0) return CB200_STATUS_SUCCESS;
    if (row_end - row_begin > 0x7fffffffll) return fail(CB200_STATUS_INVALID_SHAPE, "row range too large for one launch");
    if (schedule == fwd_schedule::tensor_blocked && blocked != nullptr) {
        // a row range that does not start on a group boundary runs the exact kernel below
        bool taken = false;
        const cb200_status st = launch_qcsr_forward_blocked(x, d, row_begin, row_end, workspace, workspace_bytes, *blocked,
                                                            split_products, sm_count, stream, &taken);
        if (st != CB200_STATUS_SUCCESS || taken) return st;
    }
    if (schedule == fwd_schedule::tensor_windows) {
        bool taken = false;
        const cb200_status st = launch_qcsr_forward_mma(x, d, row_begin, row_end, workspace, workspace_bytes,
                                                        static_cast<const std::int32_t *>(persistent), sm_count, stream,
                                                        &taken);
        if (st != CB200_STATUS_SUCCESS || taken) return st;
    }
    if (schedule == fwd_schedule::gene_tiled) {
        bool taken = false;
        const cb200_status st = launch_qcsr_forward_tiled(x, d, row_begin, row_end, static_cast<int *>(workspace),
                                                          static_cast<const std::int32_t *>(persistent), sm_count,
                                                          stream, &taken);
        if (st != CB200_STATUS_SUCCESS || taken) return st;
    }
    fwd_params p{};
    p.row_ptr = x.row_ptr; p.packed_row_ptr = x.packed_row_ptr; p.col_idx = x.col_idx; p.packed = x.packed;
    p.scales = x.scales; p.offsets = x.offsets; p.w = d.dense; p.y = d.out; p.w_ld = d.dense_ld; p.y_ld = d.out_ld;
    p.row_begin = row_begin; p.row_end = row_end; p.n = static_cast<int>(d.n); p.policy = x.policy;
    p.alpha = d.alpha; p.beta = d.beta; p.bias = d.bias; p.epilogue = d.epilogue;

    p.out_vector = reinterpret_cast<std::uintptr_t>(d.out) % 16u == 0u && d.out_ld % 4 == 0 ? 1 : 0;
    p.status = workspace_bytes >= sizeof(int) ? static_cast<int *>(workspace) : nullptr;
    const bool bf16 = d.dense_dtype == CB200_DTYPE_BF16;
    gather_shape(x, row_end - row_begin, d.n * (bf16 ? 2 : 4), sm_count, &p);
    if (p.group_rows == 0) p.short_rows = x.nnz < 64 * x.rows ? 1 : 0;
    if (gather_packs(x, d.n, d.dense_dtype) && workspace_bytes >= qcsr_gather_workspace_bytes(x.cols, x.nnz, d.n, d.dense_dtype)) {
        const int per_piece = bf16 ? 8 : 4, pieces = static_cast<int>((d.n + per_piece - 1) / per_piece);
        uint4 *packed = reinterpret_cast<uint4 *>(static_cast<unsigned char *>(workspace) + 256);
        const unsigned grid = static_cast<unsigned>((x.cols * pieces + 255) / 256);
        if (bf16) pack_rows_kernel<<<grid, 256, 0, stream>>>(static_cast<const __nv_bfloat16 *>(d.dense), d.dense_ld, p.n, x.cols, pieces, packed);
        else pack_rows_kernel<<<grid, 256, 0, stream>>>(static_cast<const float *>(d.dense), d.dense_ld, p.n, x.cols, pieces, packed);
        count_launch();
        p.w = packed;
        p.w_ld = static_cast<std::int64_t>(pieces) * per_piece;
        p.packed_rows = 1;
    }
    if (x.bits == 8) {
        if (bf16) return dispatch_gather<8, __nv_bfloat16>(p, stream);
        return dispatch_gather<8, float>(p, stream);
    }
    if (x.bits == 4) {
        if (x.packed_row_ptr == nullptr) return fail(CB200_STATUS_INVALID_ARGUMENT, "4-bit codes need packed_row_ptr");
        if (bf16) return dispatch_gather<4, __nv_bfloat16>(p, stream);
        return dispatch_gather<4, float>(p, stream);
    }
    return fail(CB200_STATUS_UNSUPPORTED, "forward SpMM supports 8-bit and 4-bit codes, got %d", x.bits);
}

} // namespace cb200
