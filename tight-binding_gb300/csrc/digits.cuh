// digits.cuh -- what the exact digit products (ozaki.cu, zgemm64.cu) share: scaled
// rounding to integers on the bit pattern, the 128-byte-swizzled K-major tile, and
// the tcgen05, bulk-copy and barrier instructions.
#pragma once
#include <cstdint>
#include "common.cuh"

namespace nrltb {

constexpr unsigned long long OZ_WAIT_NS = 2000000000ull;   // (as an argument it cost the products 2 to 3 %)
constexpr int OZ_MA = 128;                // rows of A (and of the product) per CTA: tensor-memory lanes
// instruction descriptor, kind::f16: D f32 (bits 4-5 = 1), A and B bf16
// (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bits 17-22, M >> 4 at 24-28
constexpr uint32_t OZ_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(128 >> 3) << 17) |
                              ((uint32_t)(OZ_MA >> 4) << 24);

// 2^k for -1022 <= k <= 1023, exact
__device__ __forceinline__ double pow2d(int k) { return __longlong_as_double((long long)(1023 + k) << 52); }
__device__ __forceinline__ float pow2f(int k) { return __int_as_float((127 + k) << 23); }

// v 2^k, exact: on the exponent field when the result stays a normal number
// (integer operations), else by the FP64 multiply
__device__ __forceinline__ double oz_scale2(double v, int k)
{
    const long long bits = __double_as_longlong(v);
    const int E = (int)((bits >> 52) & 0x7FF);
    if ((bits & 0x7FFFFFFFFFFFFFFFll) == 0) return v;
    if (E == 0 || E + k <= 0 || E + k >= 0x7FF) return v * pow2d(k);
    return __longlong_as_double(bits + ((long long)k << 52));
}

// rint(v 2^p) (round half to even) on the bit pattern of v, with integer
// operations only: the same integer as rounding the exactly scaled double,
// for |v 2^p| < 2^62 (no FP64-pipe multiply or conversion).
__device__ __forceinline__ long long oz_scaled_rint(double v, int p)
{
    const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
    const int E = (int)((bits >> 52) & 0x7FF);
    unsigned long long m = bits & 0xFFFFFFFFFFFFFull;
    if (E != 0) m |= 1ull << 52;
    if (m == 0) return 0;
    const int sh = (E == 0 ? 1 : E) - 1075 + p;   // |v| 2^p = m 2^sh
    unsigned long long u;
    if (sh >= 0) {
        u = m << sh;
    } else if (sh < -62) {
        u = 0;   // m 2^sh < 2^-9
    } else {
        const int r = -sh;
        const unsigned long long q = m >> r, rem = m & ((1ull << r) - 1), half = 1ull << (r - 1);
        u = q + ((rem > half || (rem == half && (q & 1ull))) ? 1ull : 0ull);
    }
    return (bits >> 63) ? -(long long)u : (long long)u;
}

// byte offset of the 16-byte chunk holding k = 8 g .. 8 g + 7 of row r in a
// 128-byte-swizzled K-major tile (chunk index XOR row mod 8)
__device__ __forceinline__ uint32_t oz_swz(int r, int g)
{
    return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((g ^ (r & 7)) << 4));
}

// ---------------------------------------------------------------------------
// tcgen05 / barrier helpers
__device__ __forceinline__ uint32_t oz_saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 B apart, descriptor version 1 (bits 46-48)
__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr)
{
    uint64_t d = (uint64_t)((saddr & 0x3FFFFu) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

__device__ __forceinline__ void oz_mma(uint32_t tmem, uint64_t da, uint64_t db, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 :: "r"(tmem), "l"(da), "l"(db), "r"(OZ_IDESC), "r"(acc));
}

__device__ __forceinline__ void oz_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar)
                 : "memory");
}

// one bounded hardware wait (the thread is suspended until the phase completes
// or about a microsecond passes)
__device__ __forceinline__ bool oz_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity), "r"(1000u) : "memory");
    return ok != 0;
}

__device__ __forceinline__ unsigned long long oz_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// wait for the phase of the given parity, at most OZ_WAIT_NS or until another
// role has given up (abort flag)
__device__ __forceinline__ bool oz_wait(uint32_t bar, uint32_t parity, volatile int *abort)
{
    if (oz_try(bar, parity)) return true;
    const unsigned long long t0 = oz_ns();
    for (;;) {
        if (oz_try(bar, parity)) return true;
        if (*abort || oz_ns() - t0 > OZ_WAIT_NS) return false;
    }
}

// the same at a kernel's end, whether or not a role has given up: a CTA that left with
// copies or MMAs of its own in flight would have them write into the next one's memory
static __device__ __noinline__ void oz_drain(uint32_t bar, uint32_t parity)
{
    if (oz_try(bar, parity)) return;
    const unsigned long long t0 = oz_ns();
    while (!oz_try(bar, parity) && oz_ns() - t0 < OZ_WAIT_NS) {}
}

__device__ __forceinline__ void oz_expect(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void oz_bulk(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// hint: bring a block of global memory into L2 ahead of its bulk copy
__device__ __forceinline__ void oz_prefetch_l2(const void *src, uint32_t bytes)
{
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" :: "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ void oz_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"(bar) : "memory");
}

__device__ __forceinline__ void oz_ld4(uint32_t taddr, float v[4])
{
    uint32_t r[4];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace nrltb
