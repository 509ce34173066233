// Inline PTX of the sm_100a primitives the tensor-core kernels share: mbarriers with bounded waits,
// bulk asynchronous copies into shared memory, tcgen05 MMA issue / commit, and TMEM loads.
// Every wait is bounded: after 2^22 polls the CTA's abort flag is raised and all waits of the CTA
// return at once, so a kernel always runs to its end and frees its TMEM.
#pragma once

#include <cstdint>

namespace cb200 {

__device__ __forceinline__ std::uint32_t smem_addr(const void *p) { return static_cast<std::uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void bar_init(std::uint32_t bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(std::uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_arrive_expect_tx(std::uint32_t bar, std::uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try_wait(std::uint32_t bar, std::uint32_t parity) {
    std::uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0u;
}
// Bounded wait.  Once any wait of the CTA has timed out (`*abort_flag` set) waits return at once.
// Returns true when the wait was given up (its own bound ran out, or another wait's did): the flag is
// looked at only while the barrier is not ready, so a wait that succeeds at once costs nothing extra.
constexpr int kPollLimit = 1 << 22;
__device__ __forceinline__ bool bar_wait(std::uint32_t bar, std::uint32_t parity, volatile int *abort_flag, int limit = kPollLimit) {
    int spins = 0;
    while (!bar_try_wait(bar, parity)) {
        if (*abort_flag != 0) return true;
        if (++spins > limit) {
            *abort_flag = 1;
            return true;
        }
    }
    return false;
}
// The same for a barrier that is normally microseconds away (a ring with slack, a whole row group of MMAs): the
// warp sleeps `ns` between polls, which leaves the issue slots of its scheduler to the warps that are working.
__device__ __forceinline__ bool bar_wait_sleeping(std::uint32_t bar, std::uint32_t parity, volatile int *abort_flag, unsigned ns) {
    int spins = 0;
    while (!bar_try_wait(bar, parity)) {
        if (*abort_flag != 0) return true;
        if (++spins > kPollLimit / 4) {
            *abort_flag = 1;
            return true;
        }
        __nanosleep(ns);
    }
    return false;
}
// Bounded wait that does not look at the abort flag: what a role uses, after the CTA has aborted, to let the
// copies or MMAs it still has in flight finish before the CTA gives up its shared memory and TMEM.
__device__ __forceinline__ bool bar_wait_drain(std::uint32_t bar, std::uint32_t parity, int limit = kPollLimit) {
    for (int spins = 0; spins <= limit; ++spins)
        if (bar_try_wait(bar, parity)) return true;
    return false;
}
// The same for a loader's copies, behind the barrier that ends the roles: `issued` fills of the stages in turn (every `step`-th of
// them this loader's), whose barriers receive nothing but the fills.
__device__ __forceinline__ void drain_fills(std::uint32_t bars, int stages, int issued, int step = 1) {
    for (int i = issued - 1; i >= 0 && i >= issued - stages; i -= step) bar_wait_drain(bars + i % stages * 8, static_cast<std::uint32_t>((i / stages) & 1));
}
// One contiguous global -> shared copy by the copy engine (this GPU's own memory, no multicast).
__device__ __forceinline__ void bulk_copy_g2s(std::uint32_t dst, const void *src, std::uint32_t bytes, std::uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// True in one lane of a converged warp, always the same one.  MMAs, commits and bulk copies are issued under it: inside
// `lane == 0` the compiler does not know that one thread is active, and every instruction with warp-uniform operands costs
// more.  Measured per 128 x 32 x 16 MMA: 48 to 240 cycles of its thread against the tensor pipe's 40, and more than 20 for
// each commit against none.
__device__ __forceinline__ bool elect_one() {
    std::uint32_t is;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(is) : : "memory");
    return is != 0u;
}
// the warp's number in the block, known to the compiler as the same in all its lanes
__device__ __forceinline__ int warp_of_block() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x) >> 5, 0); }
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
// Values loaded from a shared-memory buffer must be in their registers before a barrier arrival hands the buffer
// back to the copy engine; when they are only used later that is not a given: with the arrival straight after such
// loads a kernel of this library read refilled data (reproducibly).  Here the arrival's address depends on a warp vote
// over a word that depends on every loaded register (pass their OR), so it cannot be issued before those loads have
// returned; `zero` is a value that is 0 at run time without the compiler knowing it (say, the sign bit of a count
// among the kernel's arguments), which keeps the vote in the address.
__device__ __forceinline__ void arrive_when_loaded(std::uint32_t bar, std::uint32_t or_of_loaded_registers, int lane, std::uint32_t zero) {
    const unsigned seen = __ballot_sync(0xffffffffu, or_of_loaded_registers != 0u);
    if (lane == 0) bar_arrive(bar + (seen & zero));
}

// K-major operand with the 128-byte swizzle (the A tile): 8-row atoms of 1,024 bytes follow each
// other (SBO = 1,024 B), the leading offset is not used for this layout (encoded as 1), and a
// K = 16 step inside a 64-gene half moves the start address by 32 bytes.  Atoms are 1,024-byte
// aligned, so the base-offset field stays 0.
__device__ __forceinline__ std::uint64_t smem_desc_sw128(std::uint32_t addr) {
    std::uint64_t d = 0;
    d |= static_cast<std::uint64_t>((addr & 0x3ffffu) >> 4);
    d |= static_cast<std::uint64_t>(1) << 16;
    d |= static_cast<std::uint64_t>(1024u >> 4) << 32;
    d |= static_cast<std::uint64_t>(1) << 46; // descriptor version of this architecture
    d |= static_cast<std::uint64_t>(2) << 61; // 128-byte swizzle
    return d;
}
// kind::f16 instruction descriptor: D fp32, A and B both bf16 (format 1) or both fp16 (format 0), both K-major,
// M = 128.
__host__ __device__ constexpr std::uint32_t instr_desc(int n, bool fp16_operands = false) {
    return (1u << 4) | ((fp16_operands ? 0u : 1u) << 7) | ((fp16_operands ? 0u : 1u) << 10) |
           ((static_cast<std::uint32_t>(n) >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void mma_bf16(std::uint32_t tmem_d, std::uint64_t desc_a, std::uint64_t desc_b, std::uint32_t idesc,
                                         bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t}"
        :
        : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate ? 1u : 0u), "r"(0u)
        : "memory");
}
// kind::i8: D int32, A and B both signed 8-bit, both K-major, M = 128, K = 32.  Measured, A and B from shared memory, elected issuer:
// 48, 56, 64, 96, 128 cycles at n = 64, 96, 128, 192, 256; the sums are exact.
__host__ __device__ constexpr std::uint32_t instr_desc_i8(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((static_cast<std::uint32_t>(n) >> 3) << 17) | ((128u >> 4) << 24);
}
__device__ __forceinline__ void mma_i8(std::uint32_t tmem_d, std::uint64_t desc_a, std::uint64_t desc_b, std::uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}
__device__ __forceinline__ void mma_commit(std::uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// After an abort, behind the barrier that ends the roles: the MMAs this thread has issued finish.  `bar` is its own, used once.
__device__ __forceinline__ void drain_mmas(std::uint32_t bar) {
    mma_commit(bar);
    bar_wait_drain(bar, 0u);
}
__device__ __forceinline__ void tmem_ld32(std::uint32_t taddr, float (&v)[32]) {
    std::uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, %17, "
        "%18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]),
          "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]),
          "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Eight columns of this thread's lane, as integers.
__device__ __forceinline__ void tmem_ld8(std::uint32_t at, int (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&r"(v[0]), "=&r"(v[1]), "=&r"(v[2]), "=&r"(v[3]), "=&r"(v[4]), "=&r"(v[5]), "=&r"(v[6]), "=&r"(v[7])
        : "r"(at)
        : "memory");
}
// Sixteen columns of this thread's lane of tensor memory, of one, two or three places with one wait.
__device__ __forceinline__ void tmem_ld16(std::uint32_t at_v, float (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]), "=&f"(v[4]), "=&f"(v[5]), "=&f"(v[6]), "=&f"(v[7]), "=&f"(v[8]), "=&f"(v[9]),
          "=&f"(v[10]), "=&f"(v[11]), "=&f"(v[12]), "=&f"(v[13]), "=&f"(v[14]), "=&f"(v[15])
        : "r"(at_v)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(std::uint32_t at_v, std::uint32_t at_u, float (&v)[16], float (&u)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]), "=&f"(v[4]), "=&f"(v[5]), "=&f"(v[6]), "=&f"(v[7]), "=&f"(v[8]), "=&f"(v[9]),
          "=&f"(v[10]), "=&f"(v[11]), "=&f"(v[12]), "=&f"(v[13]), "=&f"(v[14]), "=&f"(v[15]), "=&f"(u[0]), "=&f"(u[1]), "=&f"(u[2]),
          "=&f"(u[3]), "=&f"(u[4]), "=&f"(u[5]), "=&f"(u[6]), "=&f"(u[7]), "=&f"(u[8]), "=&f"(u[9]), "=&f"(u[10]), "=&f"(u[11]),
          "=&f"(u[12]), "=&f"(u[13]), "=&f"(u[14]), "=&f"(u[15])
        : "r"(at_v), "r"(at_u)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(std::uint32_t at_v, std::uint32_t at_u, std::uint32_t at_t, float (&v)[16], float (&u)[16], float (&t)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%48];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%49];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47}, [%50];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(v[3]), "=&f"(v[4]), "=&f"(v[5]), "=&f"(v[6]), "=&f"(v[7]), "=&f"(v[8]), "=&f"(v[9]),
          "=&f"(v[10]), "=&f"(v[11]), "=&f"(v[12]), "=&f"(v[13]), "=&f"(v[14]), "=&f"(v[15]), "=&f"(u[0]), "=&f"(u[1]), "=&f"(u[2]),
          "=&f"(u[3]), "=&f"(u[4]), "=&f"(u[5]), "=&f"(u[6]), "=&f"(u[7]), "=&f"(u[8]), "=&f"(u[9]), "=&f"(u[10]), "=&f"(u[11]),
          "=&f"(u[12]), "=&f"(u[13]), "=&f"(u[14]), "=&f"(u[15]), "=&f"(t[0]), "=&f"(t[1]), "=&f"(t[2]), "=&f"(t[3]), "=&f"(t[4]),
          "=&f"(t[5]), "=&f"(t[6]), "=&f"(t[7]), "=&f"(t[8]), "=&f"(t[9]), "=&f"(t[10]), "=&f"(t[11]), "=&f"(t[12]), "=&f"(t[13]),
          "=&f"(t[14]), "=&f"(t[15])
        : "r"(at_v), "r"(at_u), "r"(at_t)
        : "memory");
}
// ... and the way back; tmem_wait_stores before they are read
__device__ __forceinline__ void tmem_st16(std::uint32_t at, const float (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::
                 "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]), "f"(v[10]),
                 "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "r"(at)
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_stores() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

} // namespace cb200
