// What the kernels that multiply digits on the tensor cores share (oz.cu, rdm_gram.cu, sym_digits.cu; opposite_tc.cu uses
// the instructions): tcgen05, mbarrier and copy instructions, and the conversion of exact 64-bit sums of digit products
// to FP64.
#pragma once

#include <cuda_fp16.h>

#include <cstdint>

#include "common.cuh"

namespace f2g {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// tcgen05 shared-memory matrix descriptor: start >> 4 [0,14), leading byte offset >> 4 [16,30), stride byte offset >> 4
// [32,46), version 1 [46,48), base offset 0, no swizzle [61,64) = 0
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// K-major with the 64-byte swizzle: rows of 64 bytes, 8 rows to an atom of 512 (sbo apart), 16-byte piece c of row r at
// place c ^ (r / 2 % 4)
__device__ __forceinline__ uint64_t smem_desc_64b(uint32_t addr, uint32_t sbo) {
    return smem_desc(addr, 16, sbo) | (4ull << 61);
}
__device__ __forceinline__ void mma_commit(uint32_t mbar, uint32_t el) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
                 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(mbar),
                 "r"(el)
                 : "memory");
}
__device__ __forceinline__ uint32_t elect_lane() {
    uint32_t el;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(el));
    return el;
}
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint32_t mbar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
// bounded wait for phase `parity`; false if it gave up or another thread of the block did
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, const volatile int* abort) {
#pragma unroll 1
    for (int it = 0; it < (1 << 26); ++it) {
        uint32_t done;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(done)
                     : "r"(mbar), "r"(parity)
                     : "memory");
        if (done)
            return true;
        if (abort && (it & 63) == 63 && *abort)
            return false;
    }
    return false;
}
// the same for a whole warp, which decides together
__device__ __forceinline__ bool mbar_wait_warp(uint32_t mbar, uint32_t parity, const volatile int* abort) {
    return __all_sync(0xffffffffu, mbar_wait(mbar, parity, abort));
}
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, uint32_t r0, uint32_t r1, uint32_t r2, uint32_t r3) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(r0), "r"(r1), "r"(r2),
                 "r"(r3)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t addr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// a * b + c on the FMA pipe. The powers of two it is used with come from registers that the compiler cannot see
// through: as shifts and adds they would go to the integer ALU, which bounds k_oz.
__device__ __forceinline__ long long mad_wide(int a, int b, long long c) {
    long long d;
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(a), "r"(b), "l"(c));
    return d;
}
__device__ __forceinline__ int opaque(int x) {
    int y;
    asm volatile("mov.b32 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}

// The FP64 value T 2^(eab - 2100), |T| < 2^63, rounded once to nearest. `base` is (eab - 1016) << 20, and
// eab - 1014 - 63 >= 1, eab - 1014 <= 2045 (no underflow or overflow whatever T is). The leading bit comes from
// a conversion of the leading word to FP32: counting leading zeros of 64 bits takes 31 clocks per warp
// of the slow integer unit, two FP64 additions or the 64-bit conversion instruction more.
__device__ __forceinline__ double oz_double(long long T, int base, int m20) { // m20: -2^20
    const uint32_t th = (uint32_t)((unsigned long long)T >> 32);
    const long long neg = (long long)((int)th >> 31);
    unsigned long long m = (unsigned long long)((T ^ neg) - neg);
    const float f = __fmaf_rz(__uint2float_rz((uint32_t)(m >> 32)), 4294967296.0f, __uint2float_rz((uint32_t)m));
    const uint32_t fe = __float_as_uint(f) >> 23;       // 127 + leading bit's place, 0 for T = 0
    const int lz1 = 189 - (int)fe;                      // leading zeros of m, less one
    m = (m << (lz1 & 63)) + 0x200u;                     // leading bit at 62, rounded at bit 10
    const uint32_t hi = (uint32_t)(m >> 42) + (uint32_t)(lz1 * m20 + base);
    const uint32_t lo = (uint32_t)(m >> 10);
    return __hiloint2double((int)(fe == 0 ? 0u : hi | (th & 0x80000000u)), (int)lo);
}
// The same for any eab: outside those bounds oz_double at kOzMid, times 2^(eab - kOzMid) in two factors
constexpr int kOzSafeLo = 1014 + 64, kOzSafeHi = 1014 + 2045, kOzMid = 2000;
__device__ __forceinline__ double oz_value(long long T, int eab) {
    const bool safe = eab >= kOzSafeLo && eab <= kOzSafeHi;
    double d = oz_double(T, ((safe ? eab : kOzMid) - 1016) << 20, -(1 << 20));
    if (!safe) {
        const int e = max(-2044, min(2046, eab - kOzMid)), h = e >> 1;
        d = d * __hiloint2double((h + 1023) << 20, 0) * __hiloint2double((e - h + 1023) << 20, 0);
    }
    return d;
}

// ---- eight digits of 62 bits ---
// x 2^(1084 - E) as an integer of 62 bits, E >= the biased exponent of x, digit offsets added: byte 7 - i is digit
// i + 128 (digit 0 in [-64, 64], the others in [-128, 127]); bits below 1 are rounded to nearest, ties away
__device__ __forceinline__ uint64_t gram_digits(double x, bool neg, int E) {
    const uint64_t bits = (uint64_t)__double_as_longlong(x);
    const int ex = (int)((bits >> 52) & 0x7ff);
    uint64_t m = (bits & 0xfffffffffffffull) | (ex ? 0x10000000000000ull : 0);
    m <<= 10; // bit 62: 2 times the integer
    const int sft = min(E - max(ex, 1), 63);
    m = ((m >> sft) + 1) >> 1;
    const uint64_t s = (bits >> 63) ^ (uint64_t)neg;
    return ((m ^ (0 - s)) + s) + 0x8080808080808080ull;
}
template <int I> __device__ __forceinline__ uint32_t gram_half2(uint64_t y0, uint64_t y1) {
    constexpr uint32_t byte = (7 - I) & 3;
    const uint32_t a = I < 4 ? (uint32_t)(y0 >> 32) : (uint32_t)y0, b = I < 4 ? (uint32_t)(y1 >> 32) : (uint32_t)y1;
    const uint32_t t = (__byte_perm(a, b, byte | (byte + 4) << 8) & 0x00ff00ffu) | 0x64006400u;
    const uint32_t off = 0xE480E480u; // -1152
    const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&t), *reinterpret_cast<const __half2*>(&off));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// D[tmem] (+)= A[smem] B[smem] like mma_ts, M = 128, N = n; major: kMajorA for an A that is contiguous along M
constexpr uint32_t kMajorA = 1u << 15;
__device__ __forceinline__ void mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t n, uint32_t accumulate, uint32_t el,
                                       uint32_t major = 0) {
    const uint32_t idesc = (1u << 4) | ((n >> 3) << 17) | (8u << 24) | major;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %4, 0;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                 :
                 : "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(el), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

} // namespace f2g
