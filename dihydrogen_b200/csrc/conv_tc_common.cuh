// PTX wrappers shared by the tcgen05 kernels: mbarriers with bounded waits,
// descriptors, fences, bulk tensor copies.
#pragma once

#include "common.cuh"

#include <cuda.h>

namespace dcb
{

constexpr uint32_t TC_TMEM_COLS = 512;
constexpr int TC_M = 128;
// Warps of the sweep and backward-filter kernels.
constexpr int TC_GROUPS_MAX = 3;                // converter groups of 4 warps
constexpr int TC_PRODUCERS = 4 * TC_GROUPS_MAX; // warps 0..11: warp w -> group w / 4, TMEM quadrant w % 4
constexpr int TC_MMA_WARP = TC_PRODUCERS;       // warps 12..14: one MMA issuer per converter group
constexpr int TC_TMA_WARP = TC_PRODUCERS + TC_GROUPS_MAX; // warp 15 issues the bulk tensor loads
constexpr int TC_RAW_W = TC_M + 8;              // staged raw row: 4 cells left, 4 right

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return (uint32_t) __cvta_generic_to_shared(p);
}

// fp32 -> TF32, round to nearest with ties away from zero, as cvt.rna.tf32.f32
// does, but with two integer instructions: the cvt runs on the special-function
// pipe at an eighth of the integer rate, and the converters need several
// conversions per output.  (Inf / NaN payloads are not preserved; finite
// inputs give the same bits.)
__device__ __forceinline__ uint32_t tf32_rna(float x)
{
    return (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
}

// An operand's bits rounded to TF32 (0x1000, 0xffffe000) or bf16 (0x8000, 0xffff0000), ties
// away from zero.  What is not a number stays that: the NaN that CUDA's arithmetic returns
// has all mantissa bits set and would be carried over into a zero.
__device__ __forceinline__ uint32_t round_operand(float x, uint32_t add, uint32_t mask)
{
    return x == x ? (__float_as_uint(x) + add) & mask : 0x7fc00000u;
}

// The same for converters (a comparison per value made the sweep kernel take 106 us instead of
// 70 at 128^3): the sum's upper bits.
__device__ __forceinline__ uint32_t round_fast(float x, uint32_t add)
{
    // the addition of zero makes every NaN that of arithmetic, which is positive
    return (uint32_t) min(__float_as_int(x + 0.f), 0x7fff7fff) + add;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

// Bounded parity wait.  Returns false when the budget ran out.  Every role but
// the MMA issuer backs off between polls (SLEEP_NS > 0): a hot polling loop in
// a dozen warps would take the issue slots the MMA thread needs.
template <int SLEEP_NS>
__device__ __forceinline__ bool mbar_wait_s(uint32_t addr, uint32_t parity, volatile int* abort_flag)
{
    long long t0 = 0;
#pragma unroll 1
    for (uint32_t it = 0; it < (1u << 24); ++it)
    {
        uint32_t done;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.b32 %0, 1, 0, p;\n\t"
            "}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done)
            return true;
        if (SLEEP_NS > 0)
            __nanosleep(SLEEP_NS);
        if ((it & 15) == 15 && *abort_flag)
            return false;
        if ((it & 255) == 255)
        {
            // a quarter of a second at most, whatever a poll costs
            const long long now = clock64();
            if (t0 == 0)
                t0 = now;
            else if (now - t0 > 500000000ll)
                break;
        }
    }
    *abort_flag = 1;
    return false;
}

template <int SLEEP_NS>
__device__ __forceinline__ bool mbar_wait_t(uint64_t* bar, uint32_t parity, volatile int* abort_flag)
{
    return mbar_wait_s<SLEEP_NS>(smem_u32(bar), parity, abort_flag);
}

__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag)
{
    return mbar_wait_t<20>(bar, parity, abort_flag);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// All tensor-core work this thread has issued so far arrives on `bar` when it is done.
__device__ __forceinline__ void mma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before()
{
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after()
{
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                              uint32_t layout_type)
{
    uint64_t d = 0;
    d |= (uint64_t) ((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t) ((lbo_bytes >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t) ((sbo_bytes >> 4) & 0x3FFFu) << 32;
    d |= 1ull << 46; // descriptor version for this architecture
    d |= (uint64_t) layout_type << 61;
    return d;
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_st16_zero(uint32_t taddr)
{
    const uint32_t z = 0;
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr),
        "r"(z)
        : "memory");
}

// 5-D tiled bulk copy global -> shared (no multicast), completion on an mbarrier.
__device__ __forceinline__ void tma_load_5d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            int c4, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// D[tmem] += A[tmem] * B[smem]: the A operand is read from tensor memory
// (lane = row of the tile, 8 consecutive 32-bit columns = the 8 k-rows of the
// step).  An A operand fetched through a shared-memory descriptor costs about
// 120 clocks per instruction whatever N is; from tensor memory the
// instruction time follows N.
__device__ __forceinline__ void mma_tf32_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, 1, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t"
        "}"
        :
        : "r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc)
        : "memory");
}

__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&v)[8])
{
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
                 "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}

// Eight k-rows of one output column: hi or lo TF32 part of the tap the table
// names, or zero for a padding row.
__device__ __forceinline__ uint32_t lds_u32(uint32_t saddr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(saddr));
    return v;
}

// ktab8 / raw are shared-window addresses; the loads are explicit ld.shared so
// that they are issued back to back (generic loads were serialised).  SPLIT: hi and lo
// parts, else one operand rounded as given.
template <bool SPLIT>
__device__ __forceinline__ void convert_chunk(uint32_t ktab8, uint32_t raw_lane, uint32_t (&v)[8], uint32_t rnd_add,
                                              uint32_t rnd_mask)
{
    // All loads first and unconditional (a padding row reads cell 4 and is
    // zeroed afterwards), so the eight chains run in parallel without branches.
    uint32_t tb[8], xv[8];
#pragma unroll
    for (int e = 0; e < 8; ++e)
        tb[e] = lds_u32(ktab8 + 4u * e);
#pragma unroll
    for (int e = 0; e < 8; ++e)
        xv[e] = lds_u32(raw_lane + ((tb[e] & 0xffffu) << 2));
#pragma unroll
    for (int e = 0; e < 8; ++e)
    {
        const uint32_t part = tb[e] >> 16;
        const uint32_t xe = part < 2 ? xv[e] : 0u;
        if (!SPLIT)
        {
            v[e] = round_fast(__uint_as_float(xe), rnd_add) & rnd_mask;
            continue;
        }
        const uint32_t hi = (xe + 0x1000u) & 0xffffe000u;
        const int rest = __float_as_int(__uint_as_float(xe) - __uint_as_float(hi));
        const uint32_t lo = (uint32_t) min(rest, 0x7fffefff) + 0x1000u; // the pipe reads the upper 19 bits
        v[e] = part == 0 ? hi : lo;
    }
}

} // namespace dcb
