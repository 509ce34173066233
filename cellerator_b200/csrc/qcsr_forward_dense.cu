// Quantized CSR forward projection on the tensor cores from dense operand tiles kept at prepare
// (schedule "tensor_dense"):
//     Y[cells, N] = alpha * deq(X)[cells, genes] * W[genes, N] + beta * Y,   N in {32, 64, 128}.
// The tiles are built from the window-blocked copy (qcsr_forward_blocked.cu), whose geometry and W
// records they share (blocked_tile.cuh).  Reference counterpart: csr_spmm_fwd over dequantised values
// (src/compute/sparse/ops/base_sparse.cu); the reference keeps no such copy, its prepared_operation only
// has room for one (persistent_kernel_state, operation_core.hh:126-129).
#include "blocked_tile.cuh"

#include <algorithm>

namespace cb200 {
namespace {

// Dense operand tiles (schedule "tensor_dense").
//
// Above a few per cent of density the scatter is the whole cost of a window, and it repeats the
// same work on every launch: the matrix does not change between launches.  So prepare can run the
// scatter once and keep its result: for every (group, window) the 64 KB operand tile, in exactly the
// shared-memory image the MMA reads (K-major, 128-byte swizzle), stored as two 32 KB half-stages
// (64 genes each; inside a half-stage the two 128-row sub-blocks follow each other).  A launch then
// only streams: the copy engine brings half-stages into a ring, one thread issues the MMAs, the
// accumulators of a group are double buffered in TMEM so that writing Y overlaps the next group.
// The kernel moves 2 bytes per matrix element (decoded bf16) instead of ~5 per stored entry, which
// is more HBM traffic above ~40 % density only in theory: below it the tile build, not HBM, bounds
// the blocked kernel.  Cost: rows x genes x 2 bytes of device memory per prepared operation.

constexpr int kDenseStageBytes = kSubBlocks * kHalfBytes; // 32 KB: 256 rows x 64 genes
constexpr int kDenseBStages = 3;
constexpr int kDenseALoaders = 2;                          // warps whose elected lane issues half-stage copies, in turn
constexpr int kDenseThreads = kRows + 32 * (2 + kDenseALoaders); // 8 epilogue warps, MMA warp, W loader warp, A loader warps
__host__ __device__ constexpr int dense_a_stages(int n) {
    return (232448 - 1024 - kDenseBStages * n * kWin * 2) / kDenseStageBytes > 6
               ? 6
               : (232448 - 1024 - kDenseBStages * n * kWin * 2) / kDenseStageBytes;
}

// One CTA per (group, window) segment of the window-blocked copy: zero a tile in shared memory,
// decode and scatter the segment's entries exactly as the blocked kernel does, write the tile out.
__global__ void __launch_bounds__(512) densify_kernel(const std::uint32_t *entries, const std::int64_t *seg_ptr,
                                                      const float *scales, const float *gene_offsets,
                                                      const float *row_offsets, std::int64_t rows, std::int64_t cols,
                                                      int windows, int baked, unsigned char *tiles) {
    extern __shared__ __align__(16) unsigned char tile[];
    const std::int64_t seg = blockIdx.x;
    const std::int64_t group = seg / windows;
    const std::int64_t gene0 = (seg % windows) * kWin;
    const int tid = threadIdx.x;
#pragma unroll
    for (int k = 0; k < kABufBytes / (512 * 16); ++k)
        *reinterpret_cast<uint4 *>(tile + k * (512 * 16) + tid * 16) = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const std::int64_t lo = seg_ptr[seg], hi = seg_ptr[seg + 1];
    for (std::int64_t i = lo + tid; i < hi; i += 512) {
        const std::uint32_t e = entries[i];
        if (static_cast<int>(e) < 0) continue; // padding
        if (baked != 0) {
            *reinterpret_cast<unsigned short *>(tile + (((e >> 16) & 0x7fffu) << 1)) = static_cast<unsigned short>(e & 0xffffu);
            continue;
        }
        const std::int64_t gene = gene0 + ((e >> 8) & (kWin - 1));
        const std::uint32_t off = ((e >> 15) & 0x7fffu) << 1;
        if (gene >= cols) continue;
        const float scale = scales != nullptr ? __ldg(scales + gene) : 1.0f;
        float add = gene_offsets != nullptr ? __ldg(gene_offsets + gene) : 0.0f;
        if (row_offsets != nullptr) {
            const std::int64_t row = group * kRows + (((off / kSubBlockBytes) << 7) | (((off >> 10) & 15u) << 3) | ((off >> 7) & 7u));
            add = row < rows ? __ldg(row_offsets + row) : 0.0f;
        }
        *reinterpret_cast<__nv_bfloat16 *>(tile + off) = __float2bfloat16_rn(fmaf(static_cast<float>(e & 0xffu), scale, add));
    }
    __syncthreads();
    unsigned char *out = tiles + static_cast<std::size_t>(seg) * kABufBytes;
#pragma unroll
    for (int k = 0; k < kABufBytes / (512 * 16); ++k) {
        const int o = k * (512 * 16) + tid * 16; // tile image: [sub-block][half][16 KB]; stored: [half][sub-block][16 KB]
        const int sb = o / kSubBlockBytes, half = (o / kHalfBytes) % (kWin / 64);
        *reinterpret_cast<uint4 *>(out + half * kDenseStageBytes + sb * kHalfBytes + (o % kHalfBytes)) =
            *reinterpret_cast<const uint4 *>(tile + o);
    }
}

struct dense_params {
    const unsigned char *tiles;   // [group][window][half][sub-block][16 KB]
    const unsigned char *records; // W windows in operand layout, record_bytes(N) apart
    float *y;
    std::int64_t y_ld;
    std::int64_t row_end; // rows >= row_end are computed but not written
    std::int64_t group_begin, group_end;
    window_split split;
    int windows;
    float alpha, beta;
    const float *bias;
    int epilogue;
    int *status;
    int poll_limit; // test hook (cb200_test_arm_wait_timeout): the W loader issues no copies and gives up after so many polls; 0: none
    std::uint32_t idesc;       // bf16 or fp16 operands
    float result_scale;        // fp16 tiles: 1 / (the power of two the values were stored times)
    const unsigned *w_absmax;  // fp16 operands: largest |W| of this launch as float bits; else null
};

template<int NC>
__global__ void __launch_bounds__(kDenseThreads, 1) qcsr_fwd_dense_kernel(const dense_params p) {
    constexpr int SA = dense_a_stages(NC);
    constexpr int SB = kDenseBStages;
    constexpr int WREC = NC * kWin * 2;       // bytes of one W window in operand layout
    constexpr int REC = record_bytes(NC);     // distance of the windows' records in global memory
    constexpr int kAccCols = kSubBlocks * NC; // one accumulator set: a group's rows x N
    constexpr int kTmemCols = 2 * kAccCols < 32 ? 32 : 2 * kAccCols;
    const std::uint32_t IDESC = p.idesc;
    static_assert(SA >= 2, "the half-stage ring needs two stages");
    extern __shared__ __align__(1024) unsigned char smem[];
    // [SA][half-stage] | [SB][W window] | barriers | tmem slot | abort
    std::uint64_t *bars = reinterpret_cast<std::uint64_t *>(smem + SA * kDenseStageBytes + SB * WREC);
    std::uint64_t *a_full = bars;              // [SA] copy engine -> MMA
    std::uint64_t *a_empty = a_full + SA;      // [SA] MMA commit -> A loaders
    std::uint64_t *b_full = a_empty + SA;      // [SB] copy engine -> MMA
    std::uint64_t *b_empty = b_full + SB;      // [SB] MMA commit -> W loader
    std::uint64_t *acc_full = b_empty + SB;    // [2]  MMA commit -> epilogue warps
    std::uint64_t *acc_empty = acc_full + 2;   // [2]  epilogue warps -> MMA (one arrival per warp)
    std::uint64_t *mma_drain = acc_empty + 2;  // the MMA warp's own, used once, after an abort
    std::uint32_t *tmem_slot = reinterpret_cast<std::uint32_t *>(mma_drain + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    volatile int *fills = reinterpret_cast<volatile int *>(tmem_slot + 2); // [1 + kDenseALoaders] of the W ring, and behind each A loader's last, once they have ended

    const int tid = threadIdx.x, warp = warp_of_block(), lane = tid & 31;
    const std::uint32_t smem0 = smem_addr(smem);
    const std::uint32_t bstage0 = smem0 + SA * kDenseStageBytes;

    if (tid == 0) {
        for (int s = 0; s < SA; ++s) {
            bar_init(smem_addr(a_full + s), 1);
            bar_init(smem_addr(a_empty + s), 1);
        }
        for (int s = 0; s < SB; ++s) {
            bar_init(smem_addr(b_full + s), 1);
            bar_init(smem_addr(b_empty + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            bar_init(smem_addr(acc_full + b), 1);
            bar_init(smem_addr(acc_empty + b), kEpilogueWarps);
        }
        bar_init(smem_addr(mma_drain), 1);
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

    const int my_units = units_of_cta(p.split, p.group_begin, p.group_end);
    const auto unit_of = [&](int i) { return unit_at(p.split, p.group_begin, p.group_end, p.windows, static_cast<int>(blockIdx.x) + i * static_cast<int>(gridDim.x)); };

    if (warp < kEpilogueWarps) {
        // ================= thread t writes row t of the group: TMEM lane = row within the sub-block =================
        const int sub = tid >> 7;
        int use = 0; // accumulators used by the CTA
        for (int gi = 0; gi < my_units; ++gi) {
            const window_unit unit = unit_of(gi);
            const std::int64_t row = static_cast<std::int64_t>(unit.group) * kRows + tid;
            const float alpha = p.alpha * p.result_scale / (p.w_absmax != nullptr ? operand_scale(__uint_as_float(__ldg(p.w_absmax))) : 1.0f);
            const auto load = [&](std::uint32_t ab, int c, float (&v)[32]) {
                tmem_ld32(tmem_base + (static_cast<std::uint32_t>((warp & 3) * 32) << 16) + ab * kAccCols + sub * NC + c, v);
            };
            const auto wait = [&]() {
                const std::uint32_t ab = static_cast<std::uint32_t>(use & 1);
                bar_wait(smem_addr(acc_full + ab), static_cast<std::uint32_t>((use >> 1) & 1), abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                return ab;
            };
            const auto release = [&](std::uint32_t ab) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(smem_addr(acc_empty + ab));
                ++use;
            };
            if (unit.slot >= 0) { // parts of a cut group
                for (int k = 0; k < unit.pieces; ++k) {
                    const std::uint32_t ab = wait();
                    float *out = p.split.sums + (static_cast<std::int64_t>(unit.slot + k) * kRows + tid) * NC;
#pragma unroll 1
                    for (int c = 0; c < NC; c += 32) {
                        float v[32];
                        load(ab, c, v);
#pragma unroll
                        for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4 *>(out + c + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
                    }
                    release(ab);
                }
            } else if (NC > 64) { // one part
                const std::uint32_t ab = wait();
#pragma unroll
                for (int c = 0; c < NC; c += 32) {
                    float v[32];
                    load(ab, c, v);
                    if (row < p.row_end) store_row(p.y + row * p.y_ld + c, v, alpha, p.beta, p.bias, c, p.epilogue);
                }
                release(ab);
            } else { // the parts of a whole group, added in order in registers
                constexpr int COLS = NC > 64 ? 32 : NC;
                float sum[COLS / 32][32];
                for (int k = 0; k < unit.pieces; ++k) {
                    const std::uint32_t ab = wait();
#pragma unroll
                    for (int h = 0; h < COLS / 32; ++h) {
                        float v[32];
                        load(ab, h * 32, v);
#pragma unroll
                        for (int i = 0; i < 32; ++i) sum[h][i] = k == 0 ? v[i] : sum[h][i] + v[i];
                    }
                    release(ab);
                }
                if (row < p.row_end) {
#pragma unroll
                    for (int h = 0; h < COLS / 32; ++h) store_row(p.y + row * p.y_ld + h * 32, sum[h], alpha, p.beta, p.bias, h * 32, p.epilogue);
                }
            }
        }
    } else if (warp == kEpilogueWarps) {
        // ================= MMA issuer =================
        long long qa = 0, qb = 0;
        int use = 0;
        for (int g = 0; g < my_units; ++g) {
            const window_unit unit = unit_of(g);
            for (int k = unit.k0, w = unit.w0; k < unit.k0 + unit.pieces; ++k, ++use) {
                const std::uint32_t ab = static_cast<std::uint32_t>(use & 1);
                const int first = w, end = part_begin(p.windows, p.split.parts, k + 1);
                bar_wait(smem_addr(acc_empty + ab), static_cast<std::uint32_t>(((use >> 1) & 1) ^ 1), abort_flag);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (; w < end; ++w, ++qb) {
                    const int s = static_cast<int>(qb % SB);
                    bar_wait(smem_addr(b_full + s), static_cast<std::uint32_t>((qb / SB) & 1), abort_flag);
                    const std::uint32_t b_tile = bstage0 + s * WREC;
                    for (int half = 0; half < kWin / 64; ++half, ++qa) {
                        const int sa = static_cast<int>(qa % SA);
                        bar_wait(smem_addr(a_full + sa), static_cast<std::uint32_t>((qa / SA) & 1), abort_flag);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        if (elect_one()) {
                            const std::uint32_t a_stage = smem0 + sa * kDenseStageBytes;
#pragma unroll
                            for (int kk = 0; kk < 4; ++kk) {
                                const std::uint64_t db = smem_desc(b_tile + (half * 4 + kk) * 256);
#pragma unroll
                                for (int sb = 0; sb < kSubBlocks; ++sb)
                                    mma_bf16(tmem_base + ab * kAccCols + sb * NC, smem_desc_sw128(a_stage + sb * kHalfBytes + kk * 32), db,
                                             IDESC, w > first || half > 0 || kk > 0);
                            }
                            mma_commit(smem_addr(a_empty + sa));
                            if (half == kWin / 64 - 1) {
                                mma_commit(smem_addr(b_empty + s));
                                if (w == end - 1) mma_commit(smem_addr(acc_full + ab));
                            }
                        }
                        __syncwarp();
                    }
                }
            }
        }
    } else if (warp == kEpilogueWarps + 1) {
        // ================= W loader =================
        if (elect_one()) {
            int q = 0;
            bool dead = p.poll_limit != 0 && bar_wait(smem_addr(b_full), 0u, abort_flag, p.poll_limit);
            for (int g = 0; g < my_units && !dead; ++g) {
                const window_unit unit = unit_of(g);
                for (int w = unit.w0; w < unit.w1; ++w, ++q) {
                    const int s = q % SB;
                    dead = bar_wait(smem_addr(b_empty + s), static_cast<std::uint32_t>(((q / SB) & 1) ^ 1), abort_flag);
                    if (dead) break; // no new copies once a wait of the CTA has run out
                    bar_arrive_expect_tx(smem_addr(b_full + s), WREC);
                    bulk_copy_g2s(bstage0 + s * WREC, p.records + static_cast<std::size_t>(w) * REC, WREC, smem_addr(b_full + s));
                }
            }
            fills[0] = q;
        }
    } else {
        // ================= A loaders: half-stages in turn =================
        if (elect_one()) {
            int q = 0, issued = 0; // half-stages of this CTA: every loader counts all of them and issues its own; one behind its last
            bool dead = false;
            for (int g = 0; g < my_units && !dead; ++g) {
                const window_unit unit = unit_of(g);
                const unsigned char *src = p.tiles + (static_cast<std::size_t>(unit.group) * p.windows + unit.w0) * (kWin / 64) * kDenseStageBytes;
                for (int h = 0; h < (unit.w1 - unit.w0) * (kWin / 64); ++h, ++q, src += kDenseStageBytes) {
                    if (q % kDenseALoaders != warp - kEpilogueWarps - 2) continue;
                    const int s = q % SA;
                    dead = bar_wait(smem_addr(a_empty + s), static_cast<std::uint32_t>(((q / SA) & 1) ^ 1), abort_flag);
                    if (dead) break;
                    issued = q + 1;
                    bar_arrive_expect_tx(smem_addr(a_full + s), kDenseStageBytes);
                    bulk_copy_g2s(smem0 + s * kDenseStageBytes, src, kDenseStageBytes, smem_addr(a_full + s));
                }
            }
            fills[warp - kEpilogueWarps - 1] = issued;
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*abort_flag != 0) { // every role has ended: what is in flight finishes before the CTA gives up its shared and tensor memory
        if (warp == kEpilogueWarps) {
            if (elect_one()) drain_mmas(smem_addr(mma_drain));
        } else if (warp == kEpilogueWarps + 1) {
            if (elect_one()) drain_fills(smem_addr(b_full), SB, fills[0]);
        } else if (warp > kEpilogueWarps) {
            if (elect_one()) drain_fills(smem_addr(a_full), SA, fills[warp - kEpilogueWarps - 1], kDenseALoaders);
        }
        __syncthreads();
    }
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTmemCols) : "memory");
    }
    if (tid == 0 && *abort_flag != 0 && p.status != nullptr) atomicExch(p.status, 1);
}

template<int NC>
cb200_status launch_dense(const dense_params &p, int sm_count, cudaStream_t stream) {
    constexpr std::size_t smem = dense_a_stages(NC) * kDenseStageBytes + kDenseBStages * NC * kWin * 2 +
                                 (2 * dense_a_stages(NC) + 2 * kDenseBStages + 5) * sizeof(std::uint64_t) + (3 + kDenseALoaders) * sizeof(int);
    static_assert(smem <= 232448, "shared memory budget");
    CB200_CUDA_OK(cudaFuncSetAttribute(qcsr_fwd_dense_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    const unsigned grid = static_cast<unsigned>(std::min(unit_count(p.split, p.group_begin, p.group_end), sm_count));
    CB200_CUDA_OK(launch_kernel(true, qcsr_fwd_dense_kernel<NC>, grid, kDenseThreads, smem, stream, p));
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    return CB200_STATUS_SUCCESS;
}

} // namespace

std::uint64_t qcsr_dense_tile_bytes(std::int64_t rows, std::int64_t cols) {
    const std::uint64_t groups = static_cast<std::uint64_t>((rows + kRows - 1) / kRows);
    const std::uint64_t windows = static_cast<std::uint64_t>((cols + kWin - 1) / kWin);
    return groups * windows * static_cast<std::uint64_t>(kABufBytes);
}

// Turns the window-blocked copy into dense operand tiles (decoded bf16 values, scales and offsets of
// `x` baked in); the entry words go back to the arena.  *built is false, with the copy left as it was,
// when the arena has no room for the tiles.  Waits for `stream`.
cb200_status densify_blocked_layout(const qcsr_view &x, blocked_layout *layout, device_arena &arena, cudaStream_t stream,
                                    bool *built) {
    *built = false;
    if (layout == nullptr || layout->seg_ptr == nullptr) return CB200_STATUS_SUCCESS;
    const std::int64_t segments = layout->groups * layout->windows;
    const std::uint64_t bytes = static_cast<std::uint64_t>(segments) * kABufBytes;
    unsigned char *tiles = static_cast<unsigned char *>(arena.take(bytes));
    if (tiles == nullptr) return CB200_STATUS_SUCCESS; // out of memory is not an error of the prepare: the blocked copy stays
    const bool row_policy = x.policy == CB200_DECODE_COLUMN_SCALE_ROW_OFFSET;
    cudaError_t err = cudaFuncSetAttribute(densify_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kABufBytes);
    if (err == cudaSuccess && segments > 0) {
        densify_kernel<<<static_cast<unsigned>(segments), 512, kABufBytes, stream>>>(layout->entries, layout->seg_ptr, x.scales,
                                                                                     row_policy ? nullptr : x.offsets,
                                                                                     row_policy ? x.offsets : nullptr, x.rows, x.cols,
                                                                                     layout->windows, layout->baked ? 1 : 0, tiles);
        count_launch();
        err = cudaGetLastError();
    }
    if (err == cudaSuccess) err = cudaStreamSynchronize(stream);
    if (err != cudaSuccess) {
        arena.give_back(tiles, bytes);
        return fail(CB200_STATUS_CUDA_ERROR, "building the dense operand tiles: %s", cudaGetErrorString(err));
    }
    arena.give_back(layout->entries, static_cast<std::uint64_t>(layout->total_entries) * 4u);
    arena.give_back(layout->seg_ptr, static_cast<std::uint64_t>(segments + 1) * 8u);
    layout->entries = nullptr;
    layout->seg_ptr = nullptr;
    layout->total_entries = 0;
    layout->dense_tiles = tiles;
    layout->bytes = bytes;
    layout->baked = false; // half_values / value_scale stay: the tiles hold what the baked words held
    layout->src_scales = x.scales;
    layout->src_offsets = x.offsets;
    *built = true;
    return CB200_STATUS_SUCCESS;
}

cb200_status launch_qcsr_forward_dense(const qcsr_view &x, const dense_args &d, std::int64_t row_begin,
                                              std::int64_t row_end, void *workspace, std::uint64_t workspace_bytes,
                                              const blocked_layout &layout, int sm_count, cudaStream_t stream, bool *taken) {
    if (d.dense_dtype != CB200_DTYPE_BF16) return CB200_STATUS_SUCCESS;
    if (d.n != 32 && d.n != 64 && d.n != 128) return CB200_STATUS_SUCCESS;
    if (row_begin % kRows != 0) return CB200_STATUS_SUCCESS; // a launch starts on a group boundary, else another kernel runs
    if (reinterpret_cast<std::uintptr_t>(d.out) % 16u != 0u || (d.out_ld * 4u) % 16u != 0u) return CB200_STATUS_SUCCESS;
    if (workspace == nullptr || workspace_bytes < qcsr_blocked_workspace_bytes(x.cols, d.n)) return CB200_STATUS_SUCCESS;
    if (reinterpret_cast<std::uintptr_t>(workspace) % 256u != 0u) return CB200_STATUS_SUCCESS;
    if (x.row_ptr != layout.src_row_ptr || x.col_idx != layout.src_col_idx || x.packed != layout.src_packed ||
        x.scales != layout.src_scales || x.offsets != layout.src_offsets)
        return fail(CB200_STATUS_STALE_STRUCTURE, "the launch's matrix is not the one the dense operand tiles were built from");
    int *status = static_cast<int *>(workspace);
    unsigned *w_absmax = reinterpret_cast<unsigned *>(workspace) + 1; // fp16 operands: float bits of the largest |W|
    unsigned char *records = static_cast<unsigned char *>(workspace) + 256;
    const bool half = layout.half_values;
    if (!half) CB200_CUDA_OK(cudaMemsetAsync(status, 0, sizeof(int), stream));
    if (half) {
        absmax_kernel<__nv_bfloat16><<<kAbsmaxParts, 1024, 0, stream>>>(static_cast<const __nv_bfloat16 *>(d.dense), d.dense_ld, x.cols, static_cast<int>(d.n),
                                                                      static_cast<unsigned *>(workspace));
        count_launch();
        CB200_CUDA_OK(cudaGetLastError());
    }
    CB200_CUDA_OK(launch_kernel(half, pack_windows_kernel<__nv_bfloat16>, dim3(static_cast<unsigned>(layout.windows), static_cast<unsigned>(d.n / kPackColumns)),
                                256, 0, stream, static_cast<const __nv_bfloat16 *>(d.dense), d.dense_ld, x.cols, static_cast<int>(d.n), 0, nullptr, nullptr, 0,
                                records, half ? w_absmax : nullptr, 0));
    count_launch();
    CB200_CUDA_OK(cudaGetLastError());
    dense_params p{};
    p.tiles = layout.dense_tiles; p.records = records; p.y = d.out; p.y_ld = d.out_ld; p.row_end = row_end;
    p.group_begin = row_begin / kRows; p.group_end = (row_end + kRows - 1) / kRows; p.windows = layout.windows;
    p.alpha = d.alpha; p.beta = d.beta; p.bias = d.bias; p.epilogue = d.epilogue; p.status = status; p.poll_limit = test_poll_limit();
    p.idesc = instr_desc(static_cast<int>(d.n), half);
    p.result_scale = half ? 1.0f / layout.value_scale : 1.0f;
    p.w_absmax = half ? w_absmax : nullptr;
    p.split = split_of_launch(x, d.n, -d.n, workspace, workspace_bytes, qcsr_blocked_workspace_bytes(x.cols, d.n), sm_count);
    *taken = true;
    cb200_status st;
    switch (d.n) {
    case 32: st = launch_dense<32>(p, sm_count, stream); break;
    case 64: st = launch_dense<64>(p, sm_count, stream); break;
    default: st = launch_dense<128>(p, sm_count, stream); break;
    }
    if (st != CB200_STATUS_SUCCESS) return st;
    return launch_add_parts(p.split, false, p.group_begin, p.group_end, row_end, static_cast<int>(d.n), d.out, d.out_ld, p.alpha, p.beta, p.bias, p.epilogue,
                            p.result_scale, p.w_absmax, stream);
}

} // namespace cb200
