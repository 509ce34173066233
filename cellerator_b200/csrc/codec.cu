// Device codec of the quantized CSR layout: quantise a float-per-entry array into packed
// codes and decode it back.
//
// Reference counterpart: portable_backend::launch_quantize_block / launch_dequantize_block
// (include/Cellerator/quantized/portable_backend.cuh:23-61), whose kernels give each THREAD a
// row (portable_quantize_kernel.cuh:7-19, portable_dequantize_kernel.cuh:7-19) and run
// pack_row_values / unpack_row_values (packing.cuh:13-260).  Here each WARP takes a row so
// that loads of genes, values and codes are coalesced; the byte layout is the same: code i of
// a row sits in byte i/cpb of the row at bit shift (i mod cpb)*bits, unused lanes of the last
// byte are 0.
//
// Rounding follows the reference's HOST rule (access.cuh:104-131): true IEEE division, round
// half away from zero, clamp.  The decode is a rounded product followed by a rounded sum
// (numeric.cuh:34-36 as compiled for a host without FMA contraction), so decoded floats are
// bit-identical to the host codec as well.
#include "kernels.cuh"

#include <type_traits>

namespace cb200 {
namespace {

struct codec_params {
    const std::int64_t *row_ptr;
    const std::int64_t *packed_row_ptr;
    const std::int32_t *col_idx;
    std::uint8_t *packed;
    const float *scales;
    const float *offsets;
    float *values;
    std::int64_t row_begin, row_end;
    int policy;
    int cols;
};

// The rule itself: a true division, round half away from zero, clamp.
template<int BITS>
__device__ __noinline__ unsigned quantize_exact(float value, float scale, float offset) {
    constexpr int max_code = (1 << BITS) - 1;
    if (scale == 0.0f) return 0u;
    const float q = __fdiv_rn(__fsub_rn(value, offset), scale);
    const float shifted = q >= 0.0f ? __fadd_rn(q, 0.5f) : __fsub_rn(q, 0.5f);
    // A float -> int conversion that overflows (or a NaN) is undefined in the host codec; on the
    // x86-64 hosts it runs on the conversion yields INT_MIN, which the rule then maps to code 0.
    // The device conversion would saturate to INT_MAX instead, so that case is decided here.
    if (!(shifted < 2147483648.0f)) return 0u;
    int rounded = static_cast<int>(shifted);
    if (rounded < 0) return 0u;
    if (rounded > max_code) rounded = max_code;
    return static_cast<unsigned>(rounded);
}

// The same code, mostly without the division: the quotient by way of the approximate reciprocal is within a few units of its
// 24th bit, so the nearest whole number is that of the exact quotient wherever it is not close to a half.  One value in a
// thousand is, and goes the exact way, as do scales and quotients out of the ordinary.  Quotients below -1/4 and more than 1/4
// above the largest code are 0 and the largest code by either rule.
template<int BITS>
__device__ __forceinline__ bool quantize_fast(float value, float scale, float offset, unsigned *code) {
    constexpr float max_code = static_cast<float>((1 << BITS) - 1), whole_bits = 12582912.0f; // 1.5 * 2^23: rounds to whole numbers
    float reciprocal;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(reciprocal) : "f"(scale));
    const float q = __fmul_rn(__fsub_rn(value, offset), reciprocal);
    const float bounded = fminf(fmaxf(q, -0.25f), max_code + 0.25f);
    const float shifted = __fadd_rn(bounded, whole_bits);
    *code = __float_as_uint(shifted) & ((1u << BITS) - 1u);
    return fabsf(scale) < 1.0e30f && fabsf(q) < 1.0e9f && fabsf(bounded - __fsub_rn(shifted, whole_bits)) < 0.4995f;
}

template<int BITS>
__device__ __forceinline__ unsigned quantize_one(float value, float scale, float offset) {
    unsigned code;
    return quantize_fast<BITS>(value, scale, offset, &code) ? code : quantize_exact<BITS>(value, scale, offset);
}

template<int BITS>
__global__ void __launch_bounds__(256) quantize_rows_kernel(const codec_params p) {
    constexpr int CPB = 8 / BITS;
    const int lane = threadIdx.x & 31;
    const std::int64_t row = p.row_begin + (static_cast<std::int64_t>(blockIdx.x) * (blockDim.x >> 5)) + (threadIdx.x >> 5);
    if (row >= p.row_end) return;
    const std::int64_t begin = __ldg(p.row_ptr + row);
    const std::int64_t end = __ldg(p.row_ptr + row + 1);
    const std::int64_t value_base = __ldg(p.row_ptr + p.row_begin);
    std::uint8_t *out = p.packed + (p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row) : begin);
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    const float row_offset = (row_policy && p.offsets != nullptr) ? __ldg(p.offsets + row) : 0.0f;
    const std::int64_t nbytes = (end - begin + CPB - 1) / CPB;
    for (std::int64_t byte = lane; byte < nbytes; byte += 32) {
        unsigned packed = 0u;
#pragma unroll
        for (int slot = 0; slot < CPB; ++slot) {
            const std::int64_t idx = begin + byte * CPB + slot;
            if (idx < end) {
                const int gene = __ldg(p.col_idx + idx);
                const float scale = p.scales != nullptr ? __ldg(p.scales + gene) : 1.0f;
                const float offset = row_policy ? row_offset : (p.offsets != nullptr ? __ldg(p.offsets + gene) : 0.0f);
                packed |= quantize_one<BITS>(p.values[idx - value_base], scale, offset) << (slot * BITS);
            }
        }
        out[byte] = static_cast<std::uint8_t>(packed);
    }
}

template<int BITS>
__global__ void __launch_bounds__(256) dequantize_rows_kernel(const codec_params p) {
    constexpr int CPB = 8 / BITS;
    constexpr unsigned MASK = (1u << BITS) - 1u;
    const int lane = threadIdx.x & 31;
    const std::int64_t row = p.row_begin + (static_cast<std::int64_t>(blockIdx.x) * (blockDim.x >> 5)) + (threadIdx.x >> 5);
    if (row >= p.row_end) return;
    const std::int64_t begin = __ldg(p.row_ptr + row);
    const std::int64_t end = __ldg(p.row_ptr + row + 1);
    const std::int64_t value_base = __ldg(p.row_ptr + p.row_begin);
    const std::uint8_t *in = p.packed + (p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + row) : begin);
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    const float row_offset = (row_policy && p.offsets != nullptr) ? __ldg(p.offsets + row) : 0.0f;
    for (std::int64_t idx = begin + lane; idx < end; idx += 32) {
        const std::int64_t local = idx - begin;
        const unsigned byte = in[local / CPB];
        const unsigned code = (byte >> (static_cast<int>(local % CPB) * BITS)) & MASK;
        const int gene = __ldg(p.col_idx + idx);
        const float scale = p.scales != nullptr ? __ldg(p.scales + gene) : 1.0f;
        const float offset = row_policy ? row_offset : (p.offsets != nullptr ? __ldg(p.offsets + gene) : 0.0f);
        p.values[idx - value_base] = __fadd_rn(__fmul_rn(static_cast<float>(code), scale), offset);
    }
}

// Both directions for large matrices, 8- and 4-bit codes.
//
// A warp-wide look-up of scale or zero-point touches one 128-byte line for every two entries of a 5 %-dense row, and L1 takes
// a line per cycle: the two look-ups of every entry held the kernels above to 120 (coding) and 280 (decoding) G entries/s on
// 33,538 genes.  Here one CTA per SM keeps {scale, zero-point} of a range of genes in shared memory, where 32 such look-ups
// take six or seven cycles, and goes through its rows once per range: genes ascend in a row, so a range is a contiguous piece
// of it, found by bisection.  Pieces are cut at multiples of 32 entries (bytes, for 4-bit codes); the few entries on the wrong
// side of a cut, and any that a row which does not ascend has out of place, are looked up in global memory.  CTAs get equal
// shares of the entries, and a CTA's warps draw blocks of at most 1,536 of them, so that a long row holds up nobody.
//
// 100,000 x 33,538, 180 M entries of 8 bits: coding 1.74 -> 0.42 ms, decoding 0.76 -> 0.37 ms with an entry to a lane; with four
// neighbouring ones (16-byte loads and stores, a step of 384 entries, decoding of 512) 0.785 -> 0.66-0.70 ms together, 4.7 TB/s.
// Bound by issue (65 % of the slots when coding) and by the latency of the one step of loads a warp has in flight at 32 warps per SM.
// Measured on the way there: two groups a step 0.73 ms, four 0.83 (coding: registers; for decoding alone 0.663, three 0.674), one
// 0.86; groups that hold a neighbour row's entries too, masked entry by entry, 0.76; the row's start looked up in global memory for each
// block 0.70; a rest of a row in steps of its own length 0.82 (three copies of the step for the instruction cache); more than 196 KB of
// shared memory, which leaves L1 28 KB, 0.82; reciprocals in the table, so that an entry that goes the exact way looks its scale
// up in global memory, 0.70.
constexpr int kTableThreads = 1024;
constexpr int kTableGenes = 20 * 1024; // genes of a range: 160 KB
constexpr int kTableRows = 2 * 1024;   // rows of a CTA between two loads of the table: 40 KB of places

// first row in [lo, hi] whose start is at least `target` (one warp; the rows' starts ascend)
__device__ __forceinline__ std::int64_t first_row_from(const std::int64_t *row_ptr, std::int64_t lo, std::int64_t hi, std::int64_t target) {
    const int lane = threadIdx.x & 31;
    while (hi > lo) { // 32 probes at a time; row hi is known to satisfy, or to be the end
        const std::int64_t step = (hi - lo + 31) / 32, at = min(hi, lo + step * lane);
        const int last = __popc(__ballot_sync(0xffffffffu, at < hi && __ldg(row_ptr + at) < target)); // probes below the target
        if (last == 0) return lo;
        const std::int64_t next_hi = last == 32 ? hi : min(hi, lo + step * last);
        lo = lo + step * (last - 1) + 1;
        hi = next_hi;
    }
    return lo;
}

template<int BITS, bool CODE>
__global__ void __launch_bounds__(kTableThreads, 1) codec_table_kernel(const codec_params p, int range_genes, int ranges, bool quads) {
    constexpr int CPB = 8 / BITS, kQuads = CODE ? 3 : 4, U = BITS == 8 ? 6 : 4; // steps of loads in flight, what 64 registers hold
    constexpr int kTableBlock = BITS == 8 ? 1536 : 1024; // units (entries, bytes) a warp draws: four steps of 384, three of 512
    extern __shared__ __align__(16) float2 codec_table[];
    std::int64_t *begins = reinterpret_cast<std::int64_t *>(codec_table + range_genes); // [kTableRows] first entry of the row
    int *from = reinterpret_cast<int *>(begins + kTableRows);       // [kTableRows] first unit of the row in this range
    int *upto = from + kTableRows;                                  // [kTableRows] ... and past its last
    int *blocks = upto + kTableRows;                                // [kTableRows] blocks of this range up to and with the row
    __shared__ std::int64_t share[2];
    __shared__ int warp_sum[kTableThreads / 32], carry, next_block;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const std::int64_t base = __ldg(p.row_ptr + p.row_begin), total = __ldg(p.row_ptr + p.row_end) - base;
    if (warp < 2) {
        const std::int64_t b = blockIdx.x + warp;
        const std::int64_t row = b == gridDim.x ? p.row_end
                                                : first_row_from(p.row_ptr, p.row_begin, p.row_end, base + total / gridDim.x * b);
        if (lane == 0) share[warp] = b == 0 ? p.row_begin : row;
    }
    __syncthreads();
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    const auto scale_of = [&](int g) { return p.scales != nullptr ? __ldg(p.scales + g) : 1.0f; };
    const auto offset_of = [&](int g) { return !row_policy && p.offsets != nullptr ? __ldg(p.offsets + g) : 0.0f; };
    // 8-bit: a lane per entry, steps laid so that a warp's accesses are whole lines (units are counted from the last multiple
    // of 32 before the row's first entry); 4-bit: a lane per byte, two entries
    const auto lead_of = [](std::int64_t begin) { return CPB == 1 ? static_cast<int>(begin & 31) : 0; };
    for (std::int64_t r0 = share[0]; r0 < share[1]; r0 += kTableRows) {
        const int rows = static_cast<int>(min(static_cast<std::int64_t>(kTableRows), share[1] - r0));
        for (int range = 0; range < ranges; ++range) {
            const int g0 = range * range_genes, genes = min(range_genes, p.cols - g0);
            __syncthreads();
            if (threadIdx.x == 0) carry = next_block = 0;
            for (int g = threadIdx.x; g < genes; g += kTableThreads) codec_table[g] = make_float2(scale_of(g0 + g), offset_of(g0 + g));
            __syncthreads();
            // the rows' pieces, and the blocks they are cut into
            for (int r1 = 0; r1 < rows; r1 += kTableThreads) {
                const int r = r1 + threadIdx.x;
                int count = 0;
                if (r < rows) {
                    const std::int64_t begin = __ldg(p.row_ptr + r0 + r);
                    const int len = static_cast<int>(__ldg(p.row_ptr + r0 + r + 1) - begin), lead = lead_of(begin);
                    const int units = lead + (len + CPB - 1) / CPB;
                    const int first = range == 0 ? 0 : upto[r];
                    int last = units;
                    if (range != ranges - 1) { // first entry of a gene beyond the range
                        int lo = max(0, first - lead) * CPB, hi = len;
                        while (lo < hi) {
                            const int mid = (lo + hi) >> 1;
                            if (__ldg(p.col_idx + begin + mid) < g0 + genes) lo = mid + 1;
                            else hi = mid;
                        }
                        last = max(first, min(units, ((lo / CPB + lead) / 32) * 32));
                    }
                    if (range == 0) begins[r] = begin;
                    from[r] = first;
                    upto[r] = last;
                    count = (last - first + kTableBlock - 1) / kTableBlock;
                }
                int sum = count;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int below = __shfl_up_sync(0xffffffffu, sum, off);
                    if (lane >= off) sum += below;
                }
                if (lane == 31) warp_sum[warp] = sum;
                __syncthreads();
                if (warp == 0) {
                    int all = lane < kTableThreads / 32 ? warp_sum[lane] : 0;
#pragma unroll
                    for (int off = 1; off < 32; off <<= 1) {
                        const int below = __shfl_up_sync(0xffffffffu, all, off);
                        if (lane >= off) all += below;
                    }
                    if (lane < kTableThreads / 32) warp_sum[lane] = all;
                }
                __syncthreads();
                if (r < rows) blocks[r] = carry + (warp == 0 ? 0 : warp_sum[warp - 1]) + sum;
                __syncthreads();
                if (threadIdx.x == 0) carry += warp_sum[kTableThreads / 32 - 1];
                __syncthreads();
            }
            const int all_blocks = carry;
            const auto draw = [&] { return lane == 0 ? atomicAdd(&next_block, 1) : 0; };
            for (int drawn = BITS == 8 ? draw() : 0;;) { // the next one early (4-bit: 0.6 % slower so)
                if constexpr (BITS == 4) drawn = draw();
                const int block = __shfl_sync(0xffffffffu, drawn, 0);
                if (block >= all_blocks) break;
                if constexpr (BITS == 8) drawn = draw();
                int lo = 0, hi = rows - 1; // first row with blocks[row] > block
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (blocks[mid] > block) hi = mid;
                    else lo = mid + 1;
                }
                const int r = lo, start = from[r] + (block - (r == 0 ? 0 : blocks[r - 1])) * kTableBlock;
                const int stop = min(upto[r], start + kTableBlock);
                const std::int64_t begin = begins[r];
                const int lead = lead_of(begin); // 8-bit: a row's units end with it
                const int len = BITS == 8 ? stop - lead : static_cast<int>(__ldg(p.row_ptr + r0 + r + 1) - begin);
                const float row_offset = (row_policy && p.offsets != nullptr) ? __ldg(p.offsets + r0 + r) : 0.0f;
                std::uint8_t *codes = p.packed + (p.packed_row_ptr != nullptr ? __ldg(p.packed_row_ptr + r0 + r) : begin) - lead;
                const std::int32_t *cols = p.col_idx + begin - lead;
                float *values = p.values + (begin - base) - lead;
                // U * 32 units from `at`; entries of unit x: [x * CPB, x * CPB + CPB), those in [lead, lead + len) are there
                const auto step = [&](auto whole, int at) {
                    const std::int32_t *step_cols = cols + (at + lane) * CPB;
                    float *step_values = values + (at + lane) * CPB;
                    std::uint8_t *step_codes = codes + at + lane;
                    const int first = lead - (at + lane) * CPB, last = min(lead + len, stop * CPB) - (at + lane) * CPB;
                    const auto there = [&](int u, int k) {
                        const int e = u * 32 * CPB + k;
                        return decltype(whole)::value || (e >= first && e < last);
                    };
                    int gene[U][CPB];
                    float value[U][CPB];
                    unsigned code[U];
#pragma unroll
                    for (int u = 0; u < U; ++u) {
                        code[u] = 0u;
                        if (!CODE && there(u, 0)) code[u] = __ldg(step_codes + u * 32);
#pragma unroll
                        for (int k = 0; k < CPB; ++k) {
                            gene[u][k] = g0;
                            value[u][k] = 0.0f;
                            if (there(u, k)) {
                                gene[u][k] = __ldg(step_cols + u * 32 * CPB + k);
                                if (CODE) value[u][k] = __ldg(step_values + u * 32 * CPB + k);
                            }
                        }
                    }
                    float2 meta[U][CPB];
                    bool elsewhere = false;
#pragma unroll
                    for (int u = 0; u < U; ++u) {
#pragma unroll
                        for (int k = 0; k < CPB; ++k) {
                            const unsigned local = static_cast<unsigned>(gene[u][k] - g0);
                            elsewhere |= local >= static_cast<unsigned>(genes);
                            meta[u][k] = codec_table[min(local, static_cast<unsigned>(genes - 1))];
                        }
                    }
                    if (elsewhere) {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
#pragma unroll
                            for (int k = 0; k < CPB; ++k)
                                if (static_cast<unsigned>(gene[u][k] - g0) >= static_cast<unsigned>(genes))
                                    meta[u][k] = make_float2(scale_of(gene[u][k]), offset_of(gene[u][k]));
                        }
                    }
                    if constexpr (CODE) {
                        unsigned packed[U] = {};
                        bool sure = true;
#pragma unroll
                        for (int u = 0; u < U; ++u) {
#pragma unroll
                            for (int k = 0; k < CPB; ++k) {
                                if (row_policy) meta[u][k].y = row_offset;
                                unsigned c;
                                sure &= quantize_fast<BITS>(value[u][k], meta[u][k].x, meta[u][k].y, &c) || !there(u, k);
                                packed[u] |= there(u, k) ? c << (k * BITS) : 0u;
                            }
                        }
                        if (!sure) { // a thousandth of the values
#pragma unroll
                            for (int u = 0; u < U; ++u) {
                                packed[u] = 0u;
#pragma unroll
                                for (int k = 0; k < CPB; ++k)
                                    if (there(u, k)) packed[u] |= quantize_one<BITS>(value[u][k], meta[u][k].x, meta[u][k].y) << (k * BITS);
                            }
                        }
#pragma unroll
                        for (int u = 0; u < U; ++u)
                            if (there(u, 0)) step_codes[u * 32] = static_cast<std::uint8_t>(packed[u]);
                    } else {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
#pragma unroll
                            for (int k = 0; k < CPB; ++k) {
                                const float v = __fadd_rn(__fmul_rn(static_cast<float>((code[u] >> (k * BITS)) & ((1u << BITS) - 1u)), meta[u][k].x),
                                                          row_policy ? row_offset : meta[u][k].y);
                                if (there(u, k)) step_values[u * 32 * CPB + k] = v;
                            }
                        }
                    }
                };
                // 8-bit, arrays on 16 bytes: groups of four entries, a lane kQuads of them per step; the entries before the first group and behind
                // the last, three at most of each, are a lane's each, loaded before the steps and finished after them
                if constexpr (BITS == 8) {
                    if (quads && ((reinterpret_cast<std::uintptr_t>(cols) | reinterpret_cast<std::uintptr_t>(values)) & 15u) == 0u && (reinterpret_cast<std::uintptr_t>(codes) & 3u) == 0u) {
                        const int first = max(lead, start), last = stop, first4 = (first + 3) & ~3, last4 = last & ~3;
                        const auto meta_of = [&](int gene) {
                            const unsigned local = static_cast<unsigned>(gene - g0);
                            float2 m = local < static_cast<unsigned>(genes) ? codec_table[local] : make_float2(scale_of(gene), offset_of(gene));
                            if (row_policy) m.y = row_offset;
                            return m;
                        };
                        int edge = lane < 3 ? first + lane : max(last4, first4) + lane - 3;
                        if (lane < 3 ? edge >= min(first4, last) : lane >= 6 || edge >= last) edge = -1;
                        int edge_gene = g0;
                        float edge_value = 0.0f;
                        unsigned edge_code = 0u;
                        if (edge >= 0) {
                            edge_gene = __ldg(cols + edge);
                            if constexpr (CODE) edge_value = __ldg(values + edge);
                            else edge_code = __ldg(codes + edge);
                        }
                        const auto quad_step = [&](auto whole, int at) {
                            const int e0 = at + lane * 4;
                            const auto there = [&](int q) { return decltype(whole)::value || (e0 + q * 128 >= first4 && e0 + q * 128 < last4); };
                            const std::int32_t *step_cols = cols + e0;
                            float *step_values = values + e0;
                            std::uint8_t *step_codes = codes + e0;
                            int4 gene[kQuads];
                            float4 value[kQuads];
                            std::uint32_t code[kQuads];
#pragma unroll
                            for (int q = 0; q < kQuads; ++q) {
                                gene[q] = make_int4(g0, g0, g0, g0);
                                value[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                code[q] = 0u;
                                if (!there(q)) continue;
                                gene[q] = __ldg(reinterpret_cast<const int4 *>(step_cols + q * 128));
                                if constexpr (CODE) value[q] = __ldg(reinterpret_cast<const float4 *>(step_values + q * 128));
                                else code[q] = __ldg(reinterpret_cast<const std::uint32_t *>(step_codes + q * 128));
                            }
#pragma unroll
                            for (int q = 0; q < kQuads; ++q) {
                                const int g[4] = {gene[q].x, gene[q].y, gene[q].z, gene[q].w};
                                const float v[4] = {value[q].x, value[q].y, value[q].z, value[q].w};
                                float2 meta[4];
                                bool elsewhere = false;
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const unsigned local = static_cast<unsigned>(g[k] - g0);
                                    elsewhere |= local >= static_cast<unsigned>(genes);
                                    meta[k] = codec_table[min(local, static_cast<unsigned>(genes - 1))];
                                    if (row_policy) meta[k].y = row_offset;
                                }
                                if (elsewhere) {
#pragma unroll
                                    for (int k = 0; k < 4; ++k) meta[k] = meta_of(g[k]);
                                }
                                if constexpr (CODE) {
                                    std::uint32_t packed = 0u;
                                    bool sure = true;
#pragma unroll
                                    for (int k = 0; k < 4; ++k) {
                                        unsigned c;
                                        sure &= quantize_fast<8>(v[k], meta[k].x, meta[k].y, &c);
                                        packed |= c << (8 * k);
                                    }
                                    if (!sure && there(q)) { // a thousandth of the values
                                        packed = 0u;
#pragma unroll
                                        for (int k = 0; k < 4; ++k) packed |= quantize_one<8>(v[k], meta[k].x, meta[k].y) << (8 * k);
                                    }
                                    if (there(q)) *reinterpret_cast<std::uint32_t *>(step_codes + q * 128) = packed;
                                } else {
                                    float w[4];
#pragma unroll
                                    for (int k = 0; k < 4; ++k) w[k] = __fadd_rn(__fmul_rn(static_cast<float>(code[q] >> (8 * k) & 0xffu), meta[k].x), meta[k].y);
                                    if (there(q)) *reinterpret_cast<float4 *>(step_values + q * 128) = make_float4(w[0], w[1], w[2], w[3]);
                                }
                            }
                        };
                        for (int at = first4; at < last4; at += kQuads * 128) {
                            if (at + kQuads * 128 <= last4) quad_step(std::true_type{}, at);
                            else quad_step(std::false_type{}, at);
                        }
                        if (edge >= 0) {
                            const float2 m = meta_of(edge_gene);
                            if constexpr (CODE) codes[edge] = static_cast<std::uint8_t>(quantize_one<8>(edge_value, m.x, m.y));
                            else values[edge] = __fadd_rn(__fmul_rn(static_cast<float>(edge_code), m.x), m.y);
                        }
                        continue;
                    }
                }
                for (int at = start; at < stop; at += U * 32) {
                    if (at >= lead && at + U * 32 <= stop && (at + U * 32) * CPB <= lead + len) step(std::true_type{}, at);
                    else step(std::false_type{}, at);
                }
            }
        }
    }
}

// The table costs a CTA per SM and a pass over scales and zero-points each: below two million entries, or for rows that leave
// most of a warp idle, the plain kernels are as fast.  The row range's share of the entries is taken from its share of the rows.
template<bool CODE>
cb200_status launch_codec_table(const qcsr_view &x, const codec_params &p, int sm_count, cudaStream_t stream, bool *taken) {
    *taken = false;
    if (x.bits != 8 && x.bits != 4) return CB200_STATUS_SUCCESS;
    const double entries = static_cast<double>(x.nnz) / static_cast<double>(x.rows) * static_cast<double>(p.row_end - p.row_begin);
    if (entries < 2.0e6 || x.nnz < 64 * x.rows || x.cols > 16ll * kTableGenes) return CB200_STATUS_SUCCESS;
    const int ranges = static_cast<int>((x.cols + kTableGenes - 1) / kTableGenes);
    const int range_genes = (static_cast<int>(x.cols) + ranges - 1) / ranges;
    // Groups of four where a row's piece of a range fills at least half a step of them (1,000,000 rows of 80 entries: 1.00 ms one by one,
    // 1.20 in groups; 300,000 x 30,000, 180 entries in two ranges, 0.71 one by one; 60,000 rows of 800: 0.39 and 0.33).
    const bool quads = x.nnz >= 192ll * ranges * x.rows;
    const std::size_t smem = static_cast<std::size_t>(range_genes) * sizeof(float2) + 5u * kTableRows * sizeof(int);
    const auto kernel = x.bits == 8 ? codec_table_kernel<8, CODE> : codec_table_kernel<4, CODE>;
    CB200_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    kernel<<<static_cast<unsigned>(sm_count), kTableThreads, smem, stream>>>(p, range_genes, ranges, quads);
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    *taken = true;
    return CB200_STATUS_SUCCESS;
}

cb200_status check(const qcsr_view &x, std::int64_t row_begin, std::int64_t row_end, const void *values) {
    if (x.row_ptr == nullptr || x.col_idx == nullptr || x.packed == nullptr || values == nullptr)
        return fail(CB200_STATUS_INVALID_ARGUMENT, "codec needs row_ptr, col_idx, packed_values and values");
    if (row_begin < 0 || row_end > x.rows || row_begin > row_end)
        return fail(CB200_STATUS_INVALID_SHAPE, "row range [%lld,%lld) outside 0..%lld", (long long)row_begin,
                    (long long)row_end, (long long)x.rows);
    if (x.bits != 8 && x.packed_row_ptr == nullptr)
        return fail(CB200_STATUS_INVALID_ARGUMENT, "sub-byte codes need packed_row_ptr");
    return CB200_STATUS_SUCCESS;
}

codec_params make_params(const qcsr_view &x, std::int64_t row_begin, std::int64_t row_end, float *values) {
    codec_params p{};
    p.row_ptr = x.row_ptr; p.packed_row_ptr = x.packed_row_ptr; p.col_idx = x.col_idx;
    p.packed = const_cast<std::uint8_t *>(x.packed); p.scales = x.scales; p.offsets = x.offsets;
    p.values = values; p.row_begin = row_begin; p.row_end = row_end; p.policy = x.policy;
    p.cols = static_cast<int>(x.cols);
    return p;
}


// ---- Blocked-ELL codec (blocked_ell.cuh:120-231): one warp per row, lane = packed byte ------

struct bell_codec_params {
    std::int64_t rows, cols;
    int block_size, ell_cols, width;
    std::int64_t row_stride;
    const std::uint32_t *block_col_idx;
    std::uint8_t *packed;
    const float *scales;
    const float *offsets;
    float *values;
    std::int64_t row_begin, row_end;
    int policy;
};

// gene of slot `slot` of a row in block row `row_block`, -1 for an empty block
__device__ __forceinline__ std::int64_t bell_gene(const bell_codec_params &p, std::int64_t row_block, int slot) {
    const std::uint32_t bc = __ldg(p.block_col_idx + row_block * p.width + slot / p.block_size);
    if (bc == 0xffffffffu) return -1;
    return static_cast<std::int64_t>(bc) * p.block_size + slot % p.block_size;
}

template<int BITS>
__global__ void __launch_bounds__(256) bell_quantize_kernel(const bell_codec_params p) {
    constexpr int CPB = 8 / BITS;
    const int lane = threadIdx.x & 31;
    const std::int64_t row = p.row_begin + (static_cast<std::int64_t>(blockIdx.x) * (blockDim.x >> 5)) + (threadIdx.x >> 5);
    if (row >= p.row_end) return;
    std::uint8_t *out = p.packed + row * p.row_stride;
    const float *in = p.values + (row - p.row_begin) * p.ell_cols;
    const std::int64_t row_block = row / p.block_size;
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    const float row_offset = (row_policy && p.offsets != nullptr) ? __ldg(p.offsets + row) : 0.0f;
    const int used = (p.ell_cols + CPB - 1) / CPB;
    for (std::int64_t byte = lane; byte < p.row_stride; byte += 32) {
        unsigned packed = 0u;
        if (byte < used) {
#pragma unroll
            for (int slot_in = 0; slot_in < CPB; ++slot_in) {
                const int slot = static_cast<int>(byte) * CPB + slot_in;
                if (slot < p.ell_cols) {
                    const std::int64_t gene = bell_gene(p, row_block, slot);
                    const std::int64_t safe = (gene >= 0 && gene < p.cols) ? gene : 0; // never index past cols
                    const float scale = p.scales != nullptr ? __ldg(p.scales + safe) : 1.0f;
                    const float offset = row_policy ? row_offset : (p.offsets != nullptr ? __ldg(p.offsets + safe) : 0.0f);
                    packed |= quantize_one<BITS>(in[slot], scale, offset) << (slot_in * BITS);
                }
            }
        }
        out[byte] = static_cast<std::uint8_t>(packed);
    }
}

template<int BITS>
__global__ void __launch_bounds__(256) bell_dequantize_kernel(const bell_codec_params p) {
    constexpr int CPB = 8 / BITS;
    constexpr unsigned MASK = (1u << BITS) - 1u;
    const int lane = threadIdx.x & 31;
    const std::int64_t row = p.row_begin + (static_cast<std::int64_t>(blockIdx.x) * (blockDim.x >> 5)) + (threadIdx.x >> 5);
    if (row >= p.row_end) return;
    const std::uint8_t *in = p.packed + row * p.row_stride;
    float *out = p.values + (row - p.row_begin) * p.ell_cols;
    const std::int64_t row_block = row / p.block_size;
    const bool row_policy = p.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    const float row_offset = (row_policy && p.offsets != nullptr) ? __ldg(p.offsets + row) : 0.0f;
    for (int slot = lane; slot < p.ell_cols; slot += 32) {
        const std::int64_t gene = bell_gene(p, row_block, slot);
        float v = 0.0f;
        if (gene >= 0 && gene < p.cols) {
            const unsigned code = (static_cast<unsigned>(in[slot / CPB]) >> ((slot % CPB) * BITS)) & MASK;
            const float scale = p.scales != nullptr ? __ldg(p.scales + gene) : 1.0f;
            const float offset = row_policy ? row_offset : (p.offsets != nullptr ? __ldg(p.offsets + gene) : 0.0f);
            v = __fadd_rn(__fmul_rn(static_cast<float>(code), scale), offset);
        }
        out[slot] = v;
    }
}

cb200_status bell_check(const qbell_view &x, std::int64_t row_begin, std::int64_t row_end, const void *values) {
    if (x.block_col_idx == nullptr || x.packed == nullptr || values == nullptr)
        return fail(CB200_STATUS_INVALID_ARGUMENT, "Blocked-ELL codec needs block_col_idx, packed_values and values");
    if (x.block_size <= 0 || x.ell_cols < 0 || x.ell_cols % x.block_size != 0)
        return fail(CB200_STATUS_INVALID_SHAPE, "ell_cols must be a multiple of block_size");
    if (row_begin < 0 || row_end > x.rows || row_begin > row_end)
        return fail(CB200_STATUS_INVALID_SHAPE, "row range outside the matrix");
    const std::int64_t need = (static_cast<std::int64_t>(x.ell_cols) * x.bits + 7) / 8;
    if (x.row_stride_bytes < need) return fail(CB200_STATUS_INVALID_SHAPE, "row_stride_bytes smaller than a packed row");
    return CB200_STATUS_SUCCESS;
}

bell_codec_params bell_params_of(const qbell_view &x, std::int64_t row_begin, std::int64_t row_end, float *values) {
    bell_codec_params p{};
    p.rows = x.rows; p.cols = x.cols; p.block_size = x.block_size; p.ell_cols = x.ell_cols;
    p.width = x.ell_cols / x.block_size; p.row_stride = x.row_stride_bytes; p.block_col_idx = x.block_col_idx;
    p.packed = const_cast<std::uint8_t *>(x.packed); p.scales = x.scales; p.offsets = x.offsets; p.values = values;
    p.row_begin = row_begin; p.row_end = row_end; p.policy = x.policy;
    return p;
}

} // namespace

cb200_status launch_qbell_quantize_rows(const qbell_view &x, std::int64_t row_begin, std::int64_t row_end,
                                        const float *values_by_slot, cudaStream_t stream) {
    const cb200_status ok = bell_check(x, row_begin, row_end, values_by_slot);
    if (ok != CB200_STATUS_SUCCESS) return ok;
    if (row_end == row_begin) return CB200_STATUS_SUCCESS;
    const bell_codec_params p = bell_params_of(x, row_begin, row_end, const_cast<float *>(values_by_slot));
    const unsigned grid = static_cast<unsigned>((row_end - row_begin + 7) / 8);
    switch (x.bits) {
    case 8: bell_quantize_kernel<8><<<grid, 256, 0, stream>>>(p); break;
    case 4: bell_quantize_kernel<4><<<grid, 256, 0, stream>>>(p); break;
    case 2: bell_quantize_kernel<2><<<grid, 256, 0, stream>>>(p); break;
    case 1: bell_quantize_kernel<1><<<grid, 256, 0, stream>>>(p); break;
    default: return fail(CB200_STATUS_UNSUPPORTED, "bits must be 1, 2, 4 or 8, got %d", x.bits);
    }
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

cb200_status launch_qbell_dequantize_rows(const qbell_view &x, std::int64_t row_begin, std::int64_t row_end,
                                          float *values_by_slot, cudaStream_t stream) {
    const cb200_status ok = bell_check(x, row_begin, row_end, values_by_slot);
    if (ok != CB200_STATUS_SUCCESS) return ok;
    if (row_end == row_begin) return CB200_STATUS_SUCCESS;
    const bell_codec_params p = bell_params_of(x, row_begin, row_end, values_by_slot);
    const unsigned grid = static_cast<unsigned>((row_end - row_begin + 7) / 8);
    switch (x.bits) {
    case 8: bell_dequantize_kernel<8><<<grid, 256, 0, stream>>>(p); break;
    case 4: bell_dequantize_kernel<4><<<grid, 256, 0, stream>>>(p); break;
    case 2: bell_dequantize_kernel<2><<<grid, 256, 0, stream>>>(p); break;
    case 1: bell_dequantize_kernel<1><<<grid, 256, 0, stream>>>(p); break;
    default: return fail(CB200_STATUS_UNSUPPORTED, "bits must be 1, 2, 4 or 8, got %d", x.bits);
    }
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

cb200_status launch_quantize_rows(const qcsr_view &x, std::int64_t row_begin, std::int64_t row_end,
                                  const float *values, int sm_count, cudaStream_t stream) {
    const cb200_status ok = check(x, row_begin, row_end, values);
    if (ok != CB200_STATUS_SUCCESS) return ok;
    if (row_end == row_begin) return CB200_STATUS_SUCCESS;
    const codec_params p = make_params(x, row_begin, row_end, const_cast<float *>(values));
    bool taken = false;
    const cb200_status st = launch_codec_table<true>(x, p, sm_count, stream, &taken);
    if (st != CB200_STATUS_SUCCESS || taken) return st;
    const unsigned grid = static_cast<unsigned>((row_end - row_begin + 7) / 8);
    switch (x.bits) {
    case 8: quantize_rows_kernel<8><<<grid, 256, 0, stream>>>(p); break;
    case 4: quantize_rows_kernel<4><<<grid, 256, 0, stream>>>(p); break;
    case 2: quantize_rows_kernel<2><<<grid, 256, 0, stream>>>(p); break;
    case 1: quantize_rows_kernel<1><<<grid, 256, 0, stream>>>(p); break;
    default: return fail(CB200_STATUS_UNSUPPORTED, "bits must be 1, 2, 4 or 8, got %d", x.bits);
    }
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

cb200_status launch_dequantize_rows(const qcsr_view &x, std::int64_t row_begin, std::int64_t row_end,
                                    float *values, int sm_count, cudaStream_t stream) {
    const cb200_status ok = check(x, row_begin, row_end, values);
    if (ok != CB200_STATUS_SUCCESS) return ok;
    if (row_end == row_begin) return CB200_STATUS_SUCCESS;
    const codec_params p = make_params(x, row_begin, row_end, values);
    bool taken = false;
    const cb200_status st = launch_codec_table<false>(x, p, sm_count, stream, &taken);
    if (st != CB200_STATUS_SUCCESS || taken) return st;
    const unsigned grid = static_cast<unsigned>((row_end - row_begin + 7) / 8);
    switch (x.bits) {
    case 8: dequantize_rows_kernel<8><<<grid, 256, 0, stream>>>(p); break;
    case 4: dequantize_rows_kernel<4><<<grid, 256, 0, stream>>>(p); break;
    case 2: dequantize_rows_kernel<2><<<grid, 256, 0, stream>>>(p); break;
    case 1: dequantize_rows_kernel<1><<<grid, 256, 0, stream>>>(p); break;
    default: return fail(CB200_STATUS_UNSUPPORTED, "bits must be 1, 2, 4 or 8, got %d", x.bits);
    }
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

} // namespace cb200
