// FP64 sigma of a C1 space on the 5th-generation tensor cores, by exact splitting of FP64 operands
// into FP16 integer digits (the scheme of Ozaki, Ogita, Oishi and Rump, Numer. Algorithms 59 (2012),
// on FP16 tensor cores as in Mukunoki et al., ISC 2020).
//
// GB300 issues 2 FP64 multiply-adds per clock and SM, 4096 FP16 ones: the FP64 terms of sigma were
// bound by that pipe. Both two-electron terms are contractions over small dense blocks:
//   same spin, per two-hole string K2 (k - 2 electrons) and column c of the other spin's strings:
//     E[K2][pr][c] = sum_{qs} <pr||qs>' D[qs][c],  D[qs][c] = <K2|a_s a_q|I> C(I, c), I = K2 + q + s,
//     sigma(J, c) += sum_{p>r in J} <J|a+_p a+_r|K2> E[J - p - r][pr][c];
//     the one-electron operator is part of it: <pr||qs>' = <pr||qs> + (h_pq d_rs - h_ps d_rq - h_rq d_ps
//     + h_rs d_pq) / (k - 1), exact on k-electron strings;
//   opposite spin, per one-hole string pair (Ka, Kb):
//     E[Ka p][Kb r] = sum_{qs} V[p][r][q][s] D[q][s], D[q][s] = sgn C(Ka + q, Kb + s),
//     sigma(Ja, Jb) += sum_{p in Ja, r in Jb} sgn E[Ja - p, p][Jb - r, r].
// The diagonal of H (every determinant's energy) is left out of both and applied as E(J) C(J) in FP64:
// it is the largest element by far and would set the digits' scale.
//
// Contraction (k_oz): a tile has 128 rows (c, or Kb; a TMEM lane each), 48 output columns (pairs pr, or
// 3 orbitals p x 16 r) and K = 16 per step (pairs qs, or one q x 16 s). Every row of D and every column
// of the integrals is scaled by its own power of two to a 57-bit integer and cut into seven signed
// base-256 digits (the first of 9 bits): A = sum_i a_i 256^(6-i), B = sum_j b_j 256^(6-j), all exact in
// FP16. The products a_i b_j with i + j = g <= 6 are summed in the accumulator of group g: integers of at
// most 2^24, so the FP32 sums are exact (see oz_lead for the bound). Digits and accumulators of neighbouring
// groups lie next to each other along N, so 11 MMAs do the 28 products of a K step. The epilogue combines
// the seven sums in a 64-bit integer T (unit: 2^-56 of the largest |a| times the largest |b|). What is
// dropped (i + j > 6) is at most six products of 2^14 in the next group: with the digits' cut, below 2^-52 of the largest
// |a| times the largest |b| per product (2^-50 with slack in both, see oz_lead), and 2^-50 (2^-48) once per output of a
// hole string for its last group's rounding and its alignment with seven others. In the norm of a row that is less than
// the roundings of an FP64 chain (figures below). It is more for an output whose own products are all far below that
// largest one: a tail of 1e-8 beside a 1 whose integral is zero is left with about half its digits.
//
// T goes to memory and a second kernel sums the terms of each sigma element, eight at a time in 64-bit
// integers aligned at their largest exponent, one conversion to FP64 per eight. One thread per element, list
// order, no atomics: sigma is bitwise the same for every grid, batch and call.
//
// Per SM one CTA of 20 warps, handing over through mbarriers (every wait bounded):
//  * 8 producer warps (two per lane quarter, alternating K steps) gather D, cut the digits and store
//    them to tensor memory as the MMAs' A operand (3 stages of 56 columns): 7 digits x 16 K. Opposite spin:
//    the integers of a tile stay in shared memory for the tile's other chunks;
//  * 8 epilogue warps (two per quarter, 24 columns each). The accumulators (7 x 48 columns) are single but
//    released in two parts, so the next chunk's MMAs follow the read-out;
//  * one warp issues the MMAs, one to three copy the integrals' digits (a ring of K steps).
//
// Bound and figures (one GB300, 2.0 GHz): sigma at CAS(16,16) 1974 ms with the FP64 kernels, 240 ms here
// (opposite spin 1510 -> 169 ms, same spin 230 -> 34 and 37 ms); CAS(14,14) 87.3 -> 14.3 ms; errors against
// 64-bit torch 6.5e-16 -> 3.5e-16 of the norm in its CSF closure. k_oz is bound by instruction issue (integer ALU 50-60 %: digits,
// read-out), the tensor pipe is 50 % busy in the opposite-spin term, 25 % in the same-spin terms. Kept: A
// from tensor memory (an MMA of N = 48 then takes N / 2 clocks; from shared memory 44); a chunk of 48
// columns (7 accumulators and 3 stages fill the 512 columns).
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "digit_mma.cuh"
#include "oz.cuh"

namespace f2g {

namespace {

constexpr int kOzS = 7;               // digits per operand
constexpr int kOzN = 48;              // output columns per chunk
constexpr int kOzM = 128;             // rows per tile
constexpr int kOzStages = 3;          // A stages in tensor memory
constexpr int kOzStageCols = kOzS * 8; // 16 halves = 8 columns per digit
constexpr int kOzProd = 8, kOzEpi = 8;
// 8 producer and 8 epilogue warps, MMA issue, B loads (registers come in units of 4 warps)
constexpr int kOzThreads = 20 * 32;
constexpr int kOzSub = 16 * 16 * 2;                      // one digit of 16 columns x 16 K
constexpr int kOzBlockBytes = kOzSub * kOzS;             // 16 columns x 16 K x 7 digits
constexpr int kOzDigitBytes = 3 * kOzSub;                // one digit of a K step of a 48-column chunk
constexpr int kOzStepBytes = kOzDigitBytes * kOzS;       // a K step of a 48-column chunk
constexpr int kOzYBytes = 16 * kOzM * 8;                 // 64-bit integers of one K step of D
constexpr int kOzMaxRing = 8;                            // K steps of B in shared memory at most
constexpr uint32_t kOzNone = 0x40000000u;                // list padding: no determinant
constexpr int kOzMinExp = 64;                            // smallest row/column exponent (denormals count as 0)
constexpr int kOzBad = 4095;                             // exponent of a row or column that holds an infinity or NaN

struct OzShared {
    alignas(8) uint64_t a_full[kOzStages], a_empty[kOzStages];
    uint64_t acc_full, acc_empty[2]; // groups 0..3, 4..6
    uint64_t b_full[kOzMaxRing], b_empty[kOzMaxRing], drain;
    uint32_t tmem_base;
    volatile int abort;
    volatile uint32_t loaded[3]; // opposite spin: K steps each loading warp has copied
};

// D[tmem] (+)= A[tmem] B[smem], kind::f16, D F32, A and B F16, K-major, M = 128, issued by the lane with
// `el` set. The whole warp runs the issue loop, so that its operands stay in uniform registers: issued
// from a branch of one thread an MMA took 45 clocks whatever its size, this way N / 2.
template <int N> __device__ __forceinline__ void mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t accumulate, uint32_t el) {
    constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kOzM >> 4) << 24);
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 q, %4, 0;\n\tsetp.ne.b32 p, %5, 0;\n\t"
                 "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
                 :
                 : "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(el), "r"(accumulate)
                 : "memory");
}
// Groups G0..G1 of one K step: digit i of A times digits G0 - i .. G1 - i of B, which lie next to each
// other along N like the groups' accumulators do, so one MMA covers up to four groups
template <int G0, int G1, int I>
__device__ __forceinline__ void mma_groups(uint32_t acc, uint32_t a, uint64_t b, uint32_t accumulate, uint32_t el) {
    if constexpr (I <= G1) {
        constexpr int g = I > G0 ? I : G0; // first group that digit I reaches
        mma_ts<(G1 - g + 1) * kOzN>(acc + g * kOzN, a + I * 8, b + (uint64_t)((g - I) * (kOzDigitBytes >> 4)), accumulate,
                                    el);
        mma_groups<G0, G1, I + 1>(acc, a, b, 1, el);
    }
}
// ---- digits --------------------------------------------------------------------------------------
// x = X 2^(e - 1078), |X| < 2^56, for the biased exponent e >= that of x (X truncated toward zero).
// Returned with the digit offsets added: bits 48..63 are the FP16 number 1280 + d0 (d0 in [-256, 256]),
// byte 5 - i is d_{i+1} + 128 (d in [-128, 127]).
constexpr unsigned long long kOzOffset = 0x6500808080808080ull;
__device__ __forceinline__ unsigned long long oz_digits(uint32_t hi, uint32_t lo, int e) {
    const int ex = (int)((hi >> 20) & 0x7ffu);
    const unsigned long long m =
        ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 3; // exponent 0 (zero): shifted out
    const unsigned long long X = m >> min(e - ex, 63);
    const long long neg = (long long)((int)hi >> 31);
    return ((X ^ (unsigned long long)neg) - (unsigned long long)neg) + kOzOffset;
}
// digit `i` of two K-neighbours as two halves
template <int I> __device__ __forceinline__ uint32_t oz_half2(unsigned long long y0, unsigned long long y1) {
    const uint32_t h0 = (uint32_t)(y0 >> 32), l0 = (uint32_t)y0, h1 = (uint32_t)(y1 >> 32), l1 = (uint32_t)y1;
    uint32_t t, off;
    if (I == 0) {
        t = __byte_perm(h0, h1, 0x7632);
        off = 0xE500E500u; // -1280
    } else {
        const uint32_t byte = I <= 2 ? 2 - I : 6 - I; // in the high word for I = 1, 2, else in the low word
        const uint32_t sel = byte | ((byte + 4) << 8);
        t = ((I <= 2 ? __byte_perm(h0, h1, sel) : __byte_perm(l0, l1, sel)) & 0x00ff00ffu) | 0x64006400u;
        off = 0xE480E480u; // -1152
    }
    const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&t), *reinterpret_cast<const __half2*>(&off));
    return *reinterpret_cast<const uint32_t*>(&r);
}

// Sum of the terms +-T[i] 2^(e[i] - 2100), i < N <= 8, |T| < 2^63: aligned at the largest exponent and added in
// 64 bits after a shift by 3, then one conversion. What the alignment cuts off is below 2^-53 of the largest
// possible term, as the roundings of a sum in FP64 would be.
template <int N> __device__ __forceinline__ double oz_sum(const long long (&T)[N], const int (&e)[N], uint32_t neg) {
    int mx = 0;
#pragma unroll
    for (int i = 0; i < N; ++i)
        mx = max(mx, e[i]);
    long long s = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const long long x = T[i] >> min(mx - e[i] + 3, 63), n = -(long long)(neg >> i & 1u);
        s += (x ^ n) - n;
    }
    return mx >= kOzBad ? __longlong_as_double(0x7ff8000000000000ll) : oz_value(s, mx + 3);
}

struct OzArgs {
    const double* C;      // vectors, cstride apart, rows of ld elements
    int64_t cstride, ld;
    long long* E;         // T of every output (see oz_double)
    int64_t ldE;          // elements per E row
    const uint16_t* rexp; // [x - x0][ldE] row exponents
    const unsigned char* b;
    const uint32_t* list; // same spin: up[K2][.]
    const uint32_t* up1;  // opposite spin: alpha one-hole lists
    const uint32_t* up1b; // opposite spin: beta one-hole lists
    const uint64_t* kstr; // opposite spin: masks of the beta one-hole strings
    int64_t x0;           // first column tile (same spin) / (v, Ka) pair (opposite spin)
    int nk;               // opposite spin: N1a
    int nt;               // same spin: column tiles; opposite spin: tiles of Kb
    int ncol;             // rows of D: columns c, or N1b
    int tpv;              // same spin: tiles per vector
    int m;                // outputs: m2, or ma
    int mb, n;
    int nchunk, ksteps;
    int tsplit;           // tile ranges per hole string
    int reuse;            // the digits' integers of a tile stay in shared memory for all chunks
    int nbuf;             // B ring: K steps held
    WaitCtl wait;
};

// Work item: a hole string, a range of tiles and (without reuse) one chunk
struct OzItem {
    int64_t K;   // hole string (same spin) or x - x0 (opposite spin)
    int64_t Ka;  // opposite spin: alpha one-hole string
    int64_t v;   // opposite spin: vector
    int nc0, nc1; // chunks
    int t0, t1;  // tiles
};

template <bool SS> __device__ __forceinline__ OzItem oz_item(const OzArgs& a, uint32_t w) {
    OzItem it;
    if (a.reuse) {
        it.nc0 = 0;
        it.nc1 = a.nchunk;
    } else {
        it.nc0 = (int)(w % (uint32_t)a.nchunk);
        it.nc1 = it.nc0 + 1;
        w /= (uint32_t)a.nchunk;
    }
    const uint32_t ts = w % (uint32_t)a.tsplit;
    w /= (uint32_t)a.tsplit;
    it.K = w;
    it.t0 = (int)((uint32_t)a.nt * ts / (uint32_t)a.tsplit);
    it.t1 = (int)((uint32_t)a.nt * (ts + 1) / (uint32_t)a.tsplit);
    it.v = it.Ka = 0;
    if (!SS) {
        const uint32_t x = (uint32_t)a.x0 + w;
        it.v = x / (uint32_t)a.nk;
        it.Ka = x - (uint32_t)it.v * (uint32_t)a.nk;
    }
    return it;
}

// digits of 8 K-neighbours (half a step) into the stage's columns of this warp's lanes
__device__ __forceinline__ void oz_store_half(uint32_t dst, const unsigned long long (&y)[8]) {
#define F2G_OZ_DIGIT(I)                                                                                               \
    tmem_st4(dst + I * 8, oz_half2<I>(y[0], y[1]), oz_half2<I>(y[2], y[3]), oz_half2<I>(y[4], y[5]),                  \
             oz_half2<I>(y[6], y[7]));
    F2G_OZ_DIGIT(0)
    F2G_OZ_DIGIT(1)
    F2G_OZ_DIGIT(2)
    F2G_OZ_DIGIT(3)
    F2G_OZ_DIGIT(4)
    F2G_OZ_DIGIT(5)
    F2G_OZ_DIGIT(6)
#undef F2G_OZ_DIGIT
}

// A producer lane's place in the sequence of K steps (same spin)
struct OzCursor {
    uint32_t w;           // work item
    int t, t1, tt, ks;    // tile, end of the item's tiles, tile within the vector, K step
    const uint32_t* list; // list of the item's hole string
    const uint16_t* rexp; // this row's exponents of it
    const double* base;   // this row's column in row 0 of its vector
};
__device__ __forceinline__ void oz_start(const OzArgs& a, OzCursor& c, int row) {
    const OzItem it = oz_item<true>(a, c.w);
    c.t = it.t0;
    c.t1 = it.t1;
    const uint32_t tg = (uint32_t)a.x0 + (uint32_t)c.t, v = tg / (uint32_t)a.tpv;
    c.tt = (int)(tg - v * (uint32_t)a.tpv);
    c.list = a.list + it.K * a.ksteps * 16;
    c.rexp = a.rexp + it.K * a.ldE + row;
    c.base = a.C + v * a.cstride + c.tt * kOzM + row;
}
__device__ __forceinline__ void oz_advance(const OzArgs& a, uint32_t nitems, OzCursor& c, int by, int row) {
    c.ks += by;
#pragma unroll 1
    while (c.ks >= a.ksteps && c.w < nitems) {
        c.ks -= a.ksteps;
        c.base += kOzM;
        if (++c.tt == a.tpv) { // next vector
            c.tt = 0;
            c.base += a.cstride - (int64_t)a.tpv * kOzM;
        }
        if (++c.t >= c.t1) {
            c.w += gridDim.x;
            if (c.w < nitems)
                oz_start(a, c, row);
        }
    }
}

} // namespace

// MB: upper bound of the beta holes per one-hole string (opposite spin)
template <bool SS, int MB>
__global__ void __launch_bounds__(kOzThreads, 1) k_oz(const __grid_constant__ OzArgs a, uint32_t nitems) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    OzShared& sh = *reinterpret_cast<OzShared*>(smem_raw);
    // opposite spin: integers of the tile's D, [K step][slot][row] ([set][slot][row] without reuse)
    unsigned long long* ybuf = reinterpret_cast<unsigned long long*>(smem_raw + 1024);
    unsigned char* bring = smem_raw + 1024 + (SS ? 0 : (a.reuse ? a.ksteps : 2) * kOzYBytes);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const volatile int* abort = &sh.abort;

    if (tid == 0) {
#pragma unroll 1
        for (int i = 0; i < kOzStages; ++i) {
            mbar_init(smem_u32(&sh.a_full[i]), 4);
            mbar_init(smem_u32(&sh.a_empty[i]), 1);
        }
        mbar_init(smem_u32(&sh.acc_full), 1);
        mbar_init(smem_u32(&sh.acc_empty[0]), kOzEpi);
        mbar_init(smem_u32(&sh.acc_empty[1]), kOzEpi);
#pragma unroll 1
        for (int i = 0; i < kOzMaxRing; ++i) {
            mbar_init(smem_u32(&sh.b_full[i]), SS ? 1 : 3);
            mbar_init(smem_u32(&sh.b_empty[i]), 1);
        }
        mbar_init(smem_u32(&sh.drain), 1);
        sh.abort = 0;
    }
    if (warp == kOzProd + kOzEpi) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_before();
    __syncthreads();
    fence_after();
    // all 512 columns are this block's: the allocation starts at column 0
    constexpr uint32_t tmem = 0;
    constexpr uint32_t acc0 = tmem, stage0 = tmem + kOzS * kOzN;
    auto give_up = [&]() {
        atomicExch(a.wait.err, 1);
        sh.abort = 1;
    };

    if (warp < kOzProd) {
        // ---- producers: digits of D, K steps alternating between the two sets
        const int quarter = warp & 3, set = warp >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        // stage of K step q: wait until its last use's MMAs are done
        auto open_stage = [&](uint32_t q) {
            const uint32_t slot = q % kOzStages, use = q / kOzStages;
            if (use > 0 && !mbar_wait_warp(smem_u32(&sh.a_empty[slot]), (use - 1) & 1, abort)) {
                give_up();
                return false;
            }
            fence_after();
            return true;
        };
        auto close_stage = [&](uint32_t q) {
            tmem_wait_st();
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&sh.a_full[q % kOzStages]));
        };
        if (SS) {
            OzCursor c;
            c.w = blockIdx.x;
            c.ks = 0;
            if (c.w < nitems) {
                oz_start(a, c, row);
                oz_advance(a, nitems, c, set, row);
            }
            uint2 x[16];
            uint32_t sg[2] = {0, 0}; // signs of x, applied at the conversion so that nothing waits for the loads
            const uint32_t ld8 = (uint32_t)a.ld * 8;
            int er = kOzMinExp;
            auto load8 = [&](bool in, int h) { // eight elements of the cursor's step
                const uint4* lp = reinterpret_cast<const uint4*>(c.list + c.ks * 16 + 8 * h);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint4 e4 = __ldg(lp + i);
                    const uint32_t e[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint2 u = make_uint2(0, 0);
                        if (in && !(e[j] & kOzNone))
                            u = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const char*>(c.base) +
                                                                     (uint64_t)(e[j] & kAddrMask) * ld8));
                        x[8 * h + 4 * i + j] = u;
                        sg[h] = __funnelshift_l(e[j], sg[h], 1);
                    }
                }
            };
            bool more = c.w < nitems;
            if (more) {
                const bool in = c.tt * kOzM + row < a.ncol;
                er = c.rexp[c.t * kOzM];
                load8(in, 0);
                load8(in, 1);
            }
#pragma unroll 1
            for (uint32_t q = (uint32_t)set; more; q += 2) {
                if (!open_stage(q))
                    break;
                const uint32_t dst = stage0 + (q % kOzStages) * kOzStageCols + lane_base;
                // the next step's loads follow the conversions that free their registers
                oz_advance(a, nitems, c, 2, row);
                more = c.w < nitems;
                const bool in = more && c.tt * kOzM + row < a.ncol;
                const int ner = more ? c.rexp[c.t * kOzM] : kOzMinExp;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    unsigned long long y[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        y[j] = oz_digits(x[8 * h + j].y ^ (sg[h] << (24 + j) & 0x80000000u), x[8 * h + j].x, er);
                    if (more)
                        load8(in, h);
                    oz_store_half(dst + 4 * h, y);
                }
                close_stage(q);
                er = ner;
            }
        } else {
            uint32_t q = 0; // K steps before this tile and chunk
            bool ok = true;
#pragma unroll 1
            for (int ks = set; ks < (a.reuse ? a.ksteps : set + 1); ks += 2)
#pragma unroll 1
                for (int sl = a.n; sl < 16; ++sl)
                    ybuf[(ks * 16 + sl) * kOzM + row] = kOzOffset;
#pragma unroll 1
            for (uint32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
                const OzItem it = oz_item<SS>(a, w);
                const double* base = a.C + it.v * a.cstride;
#pragma unroll 1
                for (int t = it.t0; t < it.t1 && ok; ++t) {
                    const int Kb = t * kOzM + row;
                    const bool valid = Kb < a.ncol;
                    const int er = valid ? a.rexp[it.K * a.ldE + Kb] : kOzMinExp;
                    const uint32_t mk = valid ? (uint32_t)a.kstr[Kb] : 0xffffu;
                    uint32_t tab[MB];
#pragma unroll
                    for (int i = 0; i < MB; ++i)
                        tab[i] = (valid && i < a.mb) ? __ldg(a.up1b + (int64_t)Kb * a.mb + i) : kOzNone;
                    // slots without a determinant hold zero (those past the orbitals always do)
                    const int nown = a.reuse ? a.ksteps : set + 1;
#pragma unroll 1
                    for (uint32_t inv = mk & ((1u << a.n) - 1u); inv; inv &= inv - 1) {
                        unsigned long long* y0 = ybuf + (__ffs((int)inv) - 1) * kOzM + row;
#pragma unroll 1
                        for (int ks = set; ks < nown; ks += 2)
                            y0[ks * 16 * kOzM] = kOzOffset;
                    }
                    uint2 x[MB];
                    uint32_t eq = 0; // alpha entry of the loaded step
                    auto load = [&](int ks) {
                        eq = __ldg(a.up1 + it.Ka * a.m + ks);
                        const double* r = base + (uint64_t)e_addr(eq) * (uint32_t)a.ld;
#pragma unroll
                        for (int i = 0; i < MB; ++i) {
                            x[i] = make_uint2(0, 0);
                            if (!(tab[i] & kOzNone))
                                x[i] = __ldg(reinterpret_cast<const uint2*>(r + (tab[i] & kAddrMask)));
                        }
                    };
#pragma unroll 1
                    for (int nc = it.nc0; nc < it.nc1 && ok; ++nc) {
                        const bool fresh = nc == it.nc0;
                        if (fresh && set < a.ksteps)
                            load(set);
#pragma unroll 1
                        for (int ks = set; ks < a.ksteps; ks += 2) {
                            unsigned long long* yk = ybuf + (a.reuse ? ks : set) * 16 * kOzM + row;
                            if (fresh) {
#pragma unroll
                                for (int i = 0; i < MB; ++i)
                                    if (valid && i < a.mb)
                                        yk[e_orb(tab[i]) * kOzM] =
                                            oz_digits(x[i].y ^ ((tab[i] ^ eq) & 0x80000000u), x[i].x, er);
                                if (ks + 2 < a.ksteps)
                                    load(ks + 2);
                            }
                            if (!open_stage(q + ks)) {
                                ok = false;
                                break;
                            }
                            const uint32_t dst = stage0 + ((q + ks) % kOzStages) * kOzStageCols + lane_base;
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                unsigned long long y[8];
#pragma unroll
                                for (int j = 0; j < 8; ++j)
                                    y[j] = yk[(8 * h + j) * kOzM];
                                oz_store_half(dst + 4 * h, y);
                            }
                            close_stage(q + ks);
                        }
                        q += a.ksteps;
                    }
                }
            }
        }
    } else if (warp < kOzProd + kOzEpi) {
        // ---- epilogue: 24 columns of 32 lanes per warp
        const int quarter = warp & 3, half = (warp - kOzProd) >> 2;
        const int row = quarter * 32 + lane;
        const uint32_t src = acc0 + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 24);
        const int c1 = opaque(1), c256 = opaque(256), c65536 = opaque(65536);
        uint32_t ntile = 0;
        bool ok = true;
#pragma unroll 1
        for (uint32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
            const OzItem it = oz_item<SS>(a, w);
#pragma unroll 1
            for (int t = it.t0; t < it.t1 && ok; ++t) {
                // this lane's row: valid outputs
                uint32_t vm = 0;
                bool valid = true;
                if (SS) {
                    const uint32_t tg = (uint32_t)a.x0 + (uint32_t)t, v = tg / (uint32_t)a.tpv;
                    valid = (int)(tg - v * (uint32_t)a.tpv) * kOzM + row < a.ncol;
                } else {
                    const int Kb = t * kOzM + row;
                    vm = Kb < a.ncol ? ~(uint32_t)a.kstr[Kb] & ((1u << a.n) - 1u) : 0u;
                }
#pragma unroll 1
                for (int nc = it.nc0; nc < it.nc1; ++nc, ++ntile) {
                    if (!mbar_wait_warp(smem_u32(&sh.acc_full), ntile & 1, abort)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    fence_after();
                    // T = sum_g S_g 256^(5-g), S_6 rounded: S_5 + S_6 / 256 in FP32 (below 2^24: rounded to an
                    // integer by the conversion), S_0 2^8 + S_1 and S_2 2^8 + S_3 in 32 bits (see oz_lead)
                    long long T[24];
                    int s4[24], s5[24];
                    auto release = [&](int set) {
                        fence_before();
                        __syncwarp();
                        if (lane == 0)
                            mbar_arrive(smem_u32(&sh.acc_empty[set]));
                    };
                    auto whole = [](uint32_t x) { return __float2int_rn(__uint_as_float(x)); };
#pragma unroll
                    for (int b = 0; b < 24; b += 8) {
                        uint32_t r6[8], r5[8], r4[8];
                        tmem_ld8(src + 6 * kOzN + b, r6);
                        tmem_ld8(src + 5 * kOzN + b, r5);
                        tmem_ld8(src + 4 * kOzN + b, r4);
                        tmem_wait_ld();
                        if (b == 16)
                            release(1);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            s4[b + j] = whole(r4[j]);
                            s5[b + j] = __float2int_rn(fmaf(__uint_as_float(r6[j]), 0.00390625f, __uint_as_float(r5[j])));
                        }
                    }
#pragma unroll
                    for (int b = 0; b < 24; b += 8) {
                        uint32_t r3[8], r2[8], r1[8], r0[8];
                        tmem_ld8(src + 3 * kOzN + b, r3);
                        tmem_ld8(src + 2 * kOzN + b, r2);
                        tmem_ld8(src + 1 * kOzN + b, r1);
                        tmem_ld8(src + 0 * kOzN + b, r0);
                        tmem_wait_ld();
                        if (b == 16)
                            release(0);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const int m = whole(r2[j]) * c256 + whole(r3[j]), h = whole(r0[j]) * c256 + whole(r1[j]);
                            T[b + j] = mad_wide(s5[b + j], c1,
                                                mad_wide(s4[b + j], c256, mad_wide(m, c65536, (long long)h << 32)));
                        }
                    }
                    if (SS) {
                        const int c0 = nc * kOzN + half * 24, left = valid ? a.m - c0 : 0;
                        long long* out = a.E + (it.K * a.m + c0) * a.ldE + t * kOzM + row;
#pragma unroll
                        for (int j = 0; j < 24; ++j) {
                            if (j < left)
                                *out = T[j];
                            out += a.ldE;
                        }
                    } else {
#pragma unroll
                        for (int blk = 0; blk < 3; ++blk) {
                            const int col = half * 24 + blk * 8, r0 = col & 15, pl = nc * 3 + (col >> 4);
                            long long* o = a.E + ((it.K * a.m + pl) * a.mb + __popc(vm & ((1u << r0) - 1u))) * a.ldE +
                                           t * kOzM + row;
                            const uint32_t v8 = pl < a.m ? vm >> r0 : 0u;
#pragma unroll
                            for (int j = 0; j < 8; ++j)
                                if (v8 >> j & 1u) {
                                    *o = T[blk * 8 + j];
                                    o += a.ldE;
                                }
                        }
                    }
                }
            }
        }
    } else if (warp == kOzProd + kOzEpi) {
        // ---- MMA issue (all lanes run the loop, one issues)
        const uint32_t el = elect_lane();
        const uint32_t lbo = 128, sbo = 256;
        uint32_t slot = 0, suse = 0, ntile = 0, bslot = 0, buse = 0;
        bool ok = a.wait.polls == 0; // with a limit on the tries (for tests) the first wait counts as given up
#pragma unroll 1
        for (uint32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
            const OzItem it = oz_item<SS>(a, w);
            const int ntc = (it.t1 - it.t0) * (it.nc1 - it.nc0);
#pragma unroll 1
            for (int t = 0; t < ntc && ok; ++t, ++ntile) {
#pragma unroll 1
                for (int ks = 0; ks < a.ksteps; ++ks) {
                    if (!mbar_wait_warp(smem_u32(&sh.b_full[bslot]), buse & 1, abort) ||
                        !mbar_wait_warp(smem_u32(&sh.a_full[slot]), suse & 1, abort)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t as = stage0 + slot * kOzStageCols;
                    const uint64_t bd = smem_desc(smem_u32(bring) + bslot * kOzStepBytes, lbo, sbo);
                    // the two sets of groups follow the epilogue's read-out of the previous tile
                    const uint32_t more = ks > 0;
                    if (!more && ntile > 0 && !mbar_wait_warp(smem_u32(&sh.acc_empty[1]), (ntile - 1) & 1, abort)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    mma_groups<4, 6, 0>(acc0, as, bd, more, el);
                    if (!more && ntile > 0 && !mbar_wait_warp(smem_u32(&sh.acc_empty[0]), (ntile - 1) & 1, abort)) {
                        ok = false;
                        break;
                    }
                    fence_after();
                    mma_groups<0, 3, 0>(acc0, as, bd, more, el);
                    mma_commit(smem_u32(&sh.a_empty[slot]), el);
                    mma_commit(smem_u32(&sh.b_empty[bslot]), el);
                    if (++slot == kOzStages) {
                        slot = 0;
                        ++suse;
                    }
                    if (++bslot == (uint32_t)a.nbuf) {
                        bslot = 0;
                        ++buse;
                    }
                }
                if (ok)
                    mma_commit(smem_u32(&sh.acc_full), el);
            }
        }
        if (!ok)
            give_up();
        // the MMAs in flight end before the block leaves
        mma_commit(smem_u32(&sh.drain), el);
        mbar_wait_warp(smem_u32(&sh.drain), 0, nullptr);
    } else if (!SS || warp == kOzProd + kOzEpi + 1) {
        // ---- integrals' digits, one K step per ring slot: same spin one copy by one warp; opposite spin the
        // seven digits of the block (p, q) of orbital pl go to [digit][pl], a warp per pl (issued by the lanes
        // of one warp the 21 copies took 1900 clocks, three steps' MMAs)
        const uint32_t el = elect_lane();
        const int pl = warp - (kOzProd + kOzEpi + 1);
        uint32_t bslot = 0, buse = 0, total = 0;
        bool ok = true;
#pragma unroll 1
        for (uint32_t w = blockIdx.x; w < nitems && ok; w += gridDim.x) {
            const OzItem it = oz_item<SS>(a, w);
            const uint32_t* up = a.up1 + it.Ka * a.m;
#pragma unroll 1
            for (int t = it.t0; t < it.t1 && ok; ++t)
#pragma unroll 1
                for (int nc = it.nc0; nc < it.nc1 && ok; ++nc) {
                    // past the last orbital: any finite values
                    const unsigned char* bp =
                        SS ? a.b + (it.K * a.nchunk + nc) * a.ksteps * (int64_t)kOzStepBytes
                           : a.b + (int64_t)e_orb(__ldg(up + min(nc * 3 + pl, a.m - 1))) * a.n * kOzBlockBytes;
#pragma unroll 1
                    for (int ks = 0; ks < a.ksteps; ++ks) {
                        const unsigned char* src =
                            SS ? bp + ks * (int64_t)kOzStepBytes : bp + (int64_t)e_orb(__ldg(up + ks)) * kOzBlockBytes;
                        const uint32_t bar = smem_u32(&sh.b_full[bslot]);
                        if (buse > 0 && !mbar_wait_warp(smem_u32(&sh.b_empty[bslot]), (buse - 1) & 1, abort)) {
                            ok = false;
                            break;
                        }
                        const uint32_t dst = smem_u32(bring) + bslot * kOzStepBytes;
                        if (el) {
                            mbar_expect(bar, SS ? kOzStepBytes : kOzBlockBytes);
                            if (SS) {
                                bulk_load(dst, src, kOzStepBytes, bar);
                            } else {
#pragma unroll
                                for (int d = 0; d < kOzS; ++d)
                                    bulk_load(dst + d * kOzDigitBytes + pl * kOzSub, src + d * kOzSub, kOzSub, bar);
                            }
                        }
                        __syncwarp();
                        ++total;
                        if (++bslot == (uint32_t)a.nbuf) {
                            bslot = 0;
                            ++buse;
                        }
                    }
                }
        }
        if (!ok)
            give_up();
        if (!SS) {
            // A slot's barrier completes with the copies of all three warps. After an abort one may have stopped
            // before the others: it arrives in the steps that they have copied and it has not (a step is copied
            // once its slot's last use is complete, so every arrival counts for its own step), or the waits below
            // would not end.
            if (el)
                sh.loaded[pl] = total;
            __syncwarp();
            asm volatile("bar.sync 1, 96;" ::: "memory");
            const uint32_t most = max(sh.loaded[0], max(sh.loaded[1], sh.loaded[2]));
            for (; total < most; ++total)
                if (el)
                    mbar_arrive(smem_u32(&sh.b_full[total % a.nbuf]));
            __syncwarp();
        }
        // the copies in flight end before the block leaves: the last of every slot
#pragma unroll 1
        for (uint32_t i = 0; i < (uint32_t)a.nbuf && i < total; ++i) {
            const uint32_t c = total - 1 - i;
            mbar_wait_warp(smem_u32(&sh.b_full[c % a.nbuf]), (c / a.nbuf) & 1, nullptr);
        }
    }
    __syncwarp();
    __syncthreads();
    if (warp == kOzProd + kOzEpi) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

namespace {

// ---- row exponents -------------------------------------------------------------------------------
__device__ __forceinline__ int oz_row_exp(uint32_t hi, int slack) {
    const int e = (int)(hi >> 20);
    return e == 0x7ff ? kOzBad : max(e, kOzMinExp) + slack;
}

// largest exponent over the pairs of K2 (blockIdx.x), per column x of the chunk
__global__ void k_oz_rexp_ss(const double* __restrict__ C, int64_t cstride, int64_t ld, const uint32_t* __restrict__ list,
                             int width, int m2, int tpv, int64_t ncol, int64_t t0, int64_t nx, int slack,
                             uint16_t* __restrict__ rexp) {
    const int64_t x = blockIdx.y * (int64_t)blockDim.x + threadIdx.x, K = blockIdx.x;
    if (x >= nx)
        return;
    const int64_t tg = t0 + x / kOzM, v = tg / tpv, c = (tg - v * tpv) * kOzM + x % kOzM;
    uint32_t mx = 0;
    if (c < ncol) {
        const uint32_t* base = reinterpret_cast<const uint32_t*>(C + v * cstride + c) + 1;
        const uint32_t* l = list + K * width;
#pragma unroll 8
        for (int i = 0; i < m2; ++i)
            mx = max(mx, __ldg(base + 2 * (int64_t)(__ldg(l + i) & kAddrMask) * ld) & 0x7fffffffu);
    }
    rexp[K * nx + x] = (uint16_t)oz_row_exp(mx, slack);
}

// opposite spin: largest exponent over (q, s) for every Kb of one (v, Ka); a maximum over q for every
// beta string first (shared memory), then over s
__global__ void k_oz_rexp_ab(const double* __restrict__ C, int64_t nd, int64_t N0b, const uint32_t* __restrict__ up_a,
                             int ma, int64_t N1a, const uint32_t* __restrict__ up_b, int mb, int64_t N1b, int64_t x0,
                             int64_t ldE, int slack, uint16_t* __restrict__ rexp) {
    extern __shared__ uint16_t m1[];
    const int64_t x = x0 + blockIdx.x, v = x / N1a, Ka = x - v * N1a;
    const uint32_t* base = reinterpret_cast<const uint32_t*>(C + v * nd) + 1;
    for (int64_t c = threadIdx.x; c < N0b; c += blockDim.x) {
        uint32_t mx = 0;
#pragma unroll 4
        for (int i = 0; i < ma; ++i)
            mx = max(mx, __ldg(base + 2 * ((int64_t)e_addr(__ldg(up_a + Ka * ma + i)) * N0b + c)) & 0x7fffffffu);
        m1[c] = (uint16_t)(mx >> 20);
    }
    __syncthreads();
    for (int64_t k = threadIdx.x; k < N1b; k += blockDim.x) {
        uint32_t e = 0;
        for (int i = 0; i < mb; ++i)
            e = max(e, (uint32_t)m1[e_addr(__ldg(up_b + k * mb + i))]);
        rexp[blockIdx.x * ldE + k] = (uint16_t)oz_row_exp(e << 20, slack);
    }
}

// ---- sums of E into sigma ------------------------------------------------------------------------
// sigma = E_det C: es[0] per alpha string (scalar energy included), es[1] per beta string, coul[Ja][q]
__global__ void k_oz_diag(int64_t N0a, int64_t N0b, int n, const double* __restrict__ ea, const double* __restrict__ eb,
                          const double* __restrict__ coul, const uint64_t* __restrict__ strb,
                          const double* __restrict__ C, double* __restrict__ S) {
    const int64_t Jb = blockIdx.y * (int64_t)blockDim.x + threadIdx.x;
    const int64_t row = blockIdx.x, Ja = row % N0a;
    if (Jb >= N0b)
        return;
    double e = ea[Ja] + eb[Jb];
    for (uint64_t m = strb[Jb]; m; m &= m - 1)
        e += __ldg(coul + Ja * n + (__ffsll((long long)m) - 1));
    const int64_t i = row * N0b + Jb;
    S[i] = e * C[i];
}

// the pairs of string J at column x: sum over its two-hole strings, eight at a time
__device__ __forceinline__ double oz_pairs_sum(const long long* __restrict__ E, const uint16_t* __restrict__ rexp,
                                               int64_t nx, int m2, const uint32_t* __restrict__ down,
                                               const uint16_t* __restrict__ dpair, const int* __restrict__ bexp, int np,
                                               int64_t J, int64_t x) {
    double acc = 0.0;
#pragma unroll 1
    for (int i0 = 0; i0 < np; i0 += 8) {
        long long T[8];
        int e[8];
        uint32_t neg = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            T[i] = 0;
            e[i] = 0;
            if (i0 + i < np) {
                const uint32_t d = __ldg(down + J * np + i0 + i);
                const int64_t K = d & kAddrMask;
                T[i] = __ldg(E + (K * m2 + ((d >> 24) & 127u)) * nx + x);
                e[i] = (int)__ldg(rexp + K * nx + x) + __ldg(bexp + __ldg(dpair + J * np + i0 + i));
                neg |= (d >> 31) << i;
            }
        }
        acc += oz_sum<8>(T, e, neg);
    }
    return acc;
}

// alpha: sigma(J, c) += sum of J's pairs, columns of the chunk
__global__ void __launch_bounds__(256) k_oz_sum_a(const long long* __restrict__ E, const uint16_t* __restrict__ rexp,
                                                  int64_t nx, int m2, const uint32_t* __restrict__ down,
                                                  const uint16_t* __restrict__ dpair, const int* __restrict__ bexp,
                                                  int np, int tpv, int64_t ncol, int64_t t0, int64_t nd,
                                                  double* __restrict__ S, const WaitCtl wait) {
    const int64_t x = blockIdx.y * (int64_t)blockDim.x + threadIdx.x, J = blockIdx.x;
    const int64_t tg = t0 + x / kOzM, v = tg / tpv, c = (tg - v * tpv) * kOzM + x % kOzM;
    if (x >= nx || c >= ncol)
        return;
    const double sum = oz_pairs_sum(E, rexp, nx, m2, down, dpair, bexp, np, J, x);
    S[v * nd + J * ncol + c] += waited(sum, wait);
}

// beta: the chunk's columns are alpha strings; 32 x 32 tiles turned in shared memory
__global__ void __launch_bounds__(256) k_oz_sum_b(const long long* __restrict__ E, const uint16_t* __restrict__ rexp,
                                                  int64_t nx, int m2, const uint32_t* __restrict__ down,
                                                  const uint16_t* __restrict__ dpair, const int* __restrict__ bexp,
                                                  int np, int64_t N0b, int tpv, int64_t ncol, int64_t t0, int64_t nd,
                                                  double* __restrict__ S, const WaitCtl wait) {
    __shared__ double tile[32][33];
    const int64_t x0 = blockIdx.y * 32, j0 = blockIdx.x * (int64_t)32;
    const int64_t tg = t0 + x0 / kOzM, v = tg / tpv, c0 = (tg - v * tpv) * kOzM + x0 % kOzM;
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
#pragma unroll 1
    for (int j = ty; j < 32; j += 8) {
        double acc = 0.0;
        if (j0 + j < N0b && c0 + tx < ncol)
            acc = oz_pairs_sum(E, rexp, nx, m2, down, dpair, bexp, np, j0 + j, x0 + tx);
        tile[j][tx] = acc;
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8)
        if (c0 + j < ncol && j0 + tx < N0b)
            S[v * nd + (c0 + j) * N0b + j0 + tx] += waited(tile[tx][j], wait);
}

// opposite spin: sigma(Ja, Jb) += sum over the p of Ja with Ja - p in the range, r of Jb
template <int NB>
__global__ void __launch_bounds__(256) k_oz_sum_ab(const long long* __restrict__ E, const uint16_t* __restrict__ rexp,
                                                   int64_t ldE, int ma, int mb, int na, int nb, int n,
                                                   const int* __restrict__ vexp, const uint32_t* __restrict__ rows,
                                                   int64_t v0, int64_t N0a, int64_t N0b, int64_t N1a, int64_t x0,
                                                   int64_t x1, const uint32_t* __restrict__ down_a,
                                                   const uint32_t* __restrict__ down_b,
                                                   const uint64_t* __restrict__ stra, double* __restrict__ S,
                                                   const WaitCtl wait) {
    __shared__ int ve[16 * 16];
    for (int i = threadIdx.x; i < n * 16; i += blockDim.x)
        ve[i] = vexp[i];
    __syncthreads();
    const int64_t Jb = blockIdx.y * (int64_t)blockDim.x + threadIdx.x;
    int64_t v = v0, Ja;
    if (rows) {
        Ja = rows[blockIdx.x];
    } else {
        v = v0 + blockIdx.x / N0a;
        Ja = blockIdx.x % N0a;
    }
    if (Jb >= N0b)
        return;
    uint32_t kb[NB], sg = 0; // Kb = Jb - r | r << 24; sign bits
#pragma unroll
    for (int j = 0; j < NB; ++j) {
        kb[j] = 0;
        if (j < nb) {
            const uint32_t e = __ldg(down_b + Jb * nb + j);
            kb[j] = e & 0x3fffffffu;
            sg |= (e >> 31) << j;
        }
    }
    const uint64_t mJ = stra[Ja];
    double* out = S + (v * N0a + Ja) * N0b + Jb;
    double acc = *out;
#pragma unroll 1
    for (int i = 0; i < na; ++i) {
        const uint32_t ep = __ldg(down_a + Ja * na + i);
        const int64_t x = v * N1a + e_addr(ep);
        if (x < x0 || x >= x1)
            continue;
        const int p = e_orb(ep), ps = (n - 1 - p) - popc64(mJ >> (p + 1)); // slot of p: unoccupied orbitals above it
        const long long* ex = E + ((x - x0) * ma + ps) * mb * ldE;
        const uint16_t* rx = rexp + (x - x0) * ldE;
        const int* vp = ve + p * 16;
        const uint32_t s = (ep >> 31) ? ~sg : sg;
#pragma unroll
        for (int h = 0; h < NB; h += 8) {
            constexpr int M = NB < 8 ? NB : 8;
            long long T[M];
            int e[M];
#pragma unroll
            for (int j = 0; j < M; ++j) {
                T[j] = 0;
                e[j] = 0;
                if (h + j < nb) {
                    const uint32_t k = kb[h + j] & kAddrMask, r = kb[h + j] >> 24;
                    // r - j unoccupied orbitals of Jb - r below r
                    T[j] = __ldg(ex + (uint64_t)(r - (uint32_t)(h + j)) * (uint32_t)ldE + k);
                    e[j] = (int)__ldg(rx + k) + vp[r];
                }
            }
            acc += oz_sum<M>(T, e, s >> h);
        }
    }
    *out = waited(acc, wait);
}

// ---- set-up ----------------------------------------------------------------------------------------
__global__ void k_oz_lists(int64_t N2, int m2, int per, int width, int np, const uint64_t* __restrict__ up2,
                           const uint64_t* __restrict__ str, uint32_t* __restrict__ up, uint32_t* __restrict__ down,
                           int cols, uint16_t* __restrict__ pair, uint16_t* __restrict__ dpair) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, K = t / per;
    const int i = (int)(t % per);
    if (K >= N2)
        return;
    uint32_t e = kOzNone;
    int id = 0;
    if (i < m2) {
        const uint64_t u = up2[K * m2 + i];
        const uint32_t I = (uint32_t)u, neg = (uint32_t)(u >> 48) & 1u;
        const int p = (int)(u >> 32) & 255, q = (int)(u >> 40) & 255; // p > q
        const uint64_t m = str[I];
        const int ip = popc64(m & ((uint64_t(1) << p) - 1)), iq = popc64(m & ((uint64_t(1) << q) - 1));
        e = I | (neg << 31);
        id = p * (p - 1) / 2 + q;
        down[(int64_t)I * np + ip * (ip - 1) / 2 + iq] = (uint32_t)K | ((uint32_t)i << 24) | (neg << 31);
        dpair[(int64_t)I * np + ip * (ip - 1) / 2 + iq] = (uint16_t)id;
    }
    if (i < width)
        up[K * width + i] = e;
    if (i < cols)
        pair[K * cols + i] = (uint16_t)id;
}

// pair integrals g[pr][qs] = <pr||qs> + one-electron part / (k - 1), zero on the diagonal, and the
// exponent of every row pr (one block per row)
__global__ void k_oz_pairs(int n, double inv, const double* __restrict__ h, const double* __restrict__ V, int slack,
                           double* __restrict__ g, int* __restrict__ bexp) {
    const int P = n * (n - 1) / 2, pr = blockIdx.x;
    int p = 1;
    while (p * (p + 1) / 2 <= pr)
        ++p;
    const int r = pr - p * (p - 1) / 2;
    uint32_t mx = 0;
    for (int qs = threadIdx.x; qs < P; qs += blockDim.x) {
        int q = 1;
        while (q * (q + 1) / 2 <= qs)
            ++q;
        const int s = qs - q * (q - 1) / 2;
        double x = 0.0;
        if (pr != qs) {
            double o = 0.0;
            if (r == s)
                o += h[p * n + q];
            if (r == q)
                o -= h[p * n + s];
            if (p == s)
                o -= h[r * n + q];
            if (p == q)
                o += h[r * n + s];
            x = V[((p * n + r) * n + q) * n + s] - V[((p * n + r) * n + s) * n + q] + o * inv;
        }
        g[pr * P + qs] = x;
        mx = max(mx, (uint32_t)(__double_as_longlong(x) >> 32) & 0x7fffffffu);
    }
    mx = __reduce_max_sync(0xffffffffu, mx);
    __shared__ uint32_t w[32];
    if ((threadIdx.x & 31) == 0)
        w[threadIdx.x >> 5] = mx;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < (int)(blockDim.x >> 5); ++i)
            mx = max(mx, w[i]);
        bexp[pr] = oz_row_exp(mx, slack);
    }
}

// 8 K-neighbours of one output column: their digits, one 16-byte row of a core matrix each
template <int DIGIT> __device__ __forceinline__ void oz_store8(const double (&x)[8], int e, unsigned char* dst) {
    unsigned long long y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const unsigned long long u = (unsigned long long)__double_as_longlong(x[j]);
        y[j] = oz_digits((uint32_t)(u >> 32), (uint32_t)u, e);
    }
#define F2G_OZ_ROW(I)                                                                                                 \
    *reinterpret_cast<uint4*>(dst + I * DIGIT) = make_uint4(oz_half2<I>(y[0], y[1]), oz_half2<I>(y[2], y[3]),         \
                                                            oz_half2<I>(y[4], y[5]), oz_half2<I>(y[6], y[7]));
    F2G_OZ_ROW(0)
    F2G_OZ_ROW(1)
    F2G_OZ_ROW(2)
    F2G_OZ_ROW(3)
    F2G_OZ_ROW(4)
    F2G_OZ_ROW(5)
    F2G_OZ_ROW(6)
#undef F2G_OZ_ROW
}

// digits of the pair integrals of one (K2, chunk, K step): block of 96 threads, (column, K half) each
__global__ void __launch_bounds__(96) k_oz_b_ss(int P, int m2, int nchunk, int ksteps, int width,
                                                const uint16_t* __restrict__ pair, const double* __restrict__ g,
                                                const int* __restrict__ bexp, unsigned char* __restrict__ b) {
    const int64_t K = blockIdx.x;
    const int nc = blockIdx.y, cols = nchunk * kOzN;
    const int col = threadIdx.x >> 1, kh = threadIdx.x & 1;
    const int slot = nc * kOzN + col;
    const uint16_t* pk = pair + K * cols;
    const int pr = slot < m2 ? pk[slot] : -1;
    const int e = pr >= 0 ? bexp[pr] : kOzMinExp;
    for (int ks = 0; ks < ksteps; ++ks) {
        double x[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = ks * 16 + kh * 8 + j;
            x[j] = (pr >= 0 && k < m2) ? g[pr * P + pk[k]] : 0.0;
        }
        unsigned char* dst = b + ((K * nchunk + nc) * ksteps + ks) * (int64_t)kOzStepBytes +
                             (col >> 3) * 256 + kh * 128 + (col & 7) * 16;
        oz_store8<kOzDigitBytes>(x, e, dst);
    }
}

// digits of V[p][r][q][s], block (p, q); exponents per (p, r)
__global__ void k_oz_vexp(int n, const double* __restrict__ V, int slack, int* __restrict__ vexp) {
    const int p = blockIdx.x / 16, r = blockIdx.x % 16;
    uint32_t mx = 0;
    if (r < n)
        for (int t = threadIdx.x; t < n * n; t += 32) {
            const int q = t / n, s = t % n;
            if (!(p == q && r == s))
                mx = max(mx, (uint32_t)(__double_as_longlong(V[((p * n + r) * n + q) * n + s]) >> 32) & 0x7fffffffu);
        }
    mx = __reduce_max_sync(0xffffffffu, mx);
    if (threadIdx.x == 0)
        vexp[blockIdx.x] = oz_row_exp(mx, slack);
}
__global__ void __launch_bounds__(32) k_oz_b_ab(int n, const double* __restrict__ V, const int* __restrict__ vexp,
                                                unsigned char* __restrict__ b) {
    const int p = blockIdx.x / n, q = blockIdx.x % n;
    const int r = threadIdx.x >> 1, kh = threadIdx.x & 1;
    double x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const int s = kh * 8 + j;
        x[j] = (r < n && s < n && !(p == q && r == s)) ? V[((p * n + r) * n + q) * n + s] : 0.0;
    }
    oz_store8<kOzSub>(x, vexp[p * 16 + r],
                      b + (int64_t)blockIdx.x * kOzBlockBytes + (r >> 3) * 256 + kh * 128 + (r & 7) * 16);
}

// same-spin energy of every string (+ e0), Coulomb row of every alpha string (coul may be null)
__global__ void k_oz_energies(int n, int64_t N0, const uint64_t* __restrict__ str, const double* __restrict__ h,
                              const double* __restrict__ V, double e0, double* __restrict__ es,
                              double* __restrict__ coul) {
    const int64_t I = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (I >= N0)
        return;
    const uint64_t m = str[I];
    double e = e0;
    for (int p = 0; p < n; ++p) {
        if (!(m >> p & 1))
            continue;
        e += h[p * n + p];
        for (int q = 0; q < p; ++q)
            if (m >> q & 1)
                e += V[((p * n + q) * n + p) * n + q] - V[((p * n + q) * n + q) * n + p];
    }
    es[I] = e;
    if (coul)
        for (int q = 0; q < n; ++q) {
            double j = 0.0;
            for (int p = 0; p < n; ++p)
                if (m >> p & 1)
                    j += V[((p * n + q) * n + p) * n + q];
            coul[I * n + q] = j;
        }
}

int oz_sms() {
    int dev = 0, sms = 0;
    F2G_CUDA(cudaGetDevice(&dev));
    F2G_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return sms;
}

// The FP32 sums of k_oz are exact while the products of one group sum to at most 2^24 in magnitude. Of
// nk non-zero rows of D per output, with |d_0| <= 2^8 (2^7 with slack 1) and |d_i| <= 2^7 otherwise, group
// 6 is the largest: nk (2 2^15 + 5 2^14) <= 2^24 for nk <= 113, nk (2^15 + 6 2^14) for nk <= 128 (slack in
// B), nk 7 2^14 for nk <= 146 (slack in A and B). The epilogue's S_2 2^8 + S_3 also fits 32 bits, |S_2| 2^8
// <= 2^31 - 2^24: nk 5 2^22 without slack for nk <= 101, nk 4 2^22 with slack in B for nk <= 126, nk 3 2^22
// with both for all 146. -1: too many.
int oz_lead(int nk) { return nk <= 101 ? 0 : nk <= 126 ? 1 : nk <= 146 ? 2 : -1; }
int oz_slack_a(int lead) { return lead >= 2; }
int oz_slack_b(int lead) { return lead >= 1; }

} // namespace

bool oz_supported(const CIStrings* s, bool* fast) {
    const int na = s->na, nb = s->nb, n = s->norb;
    if (n > 16 || na < 2 || nb < 2 || s->a.N0 == 0 || s->b.N0 == 0)
        return false;
    if (oz_lead(std::max({s->a.m1 * s->b.m1, s->a.m2, s->b.m2})) < 0)
        return false;
    if (fast) {
        // Up to 8,192 determinants one launch of small.cu: 4,900 determinants 29 us (89 us here), 15,876 determinants 102
        // us (90 us), four vectors 324 us (113 us). A beta spin with two or three holes leaves 3 or 4 of the 16 places of a
        // K step and a column block in use; where the alpha spin too has few electrons or holes, the FP64 kernels are
        // faster: (14, 2, 12) 113 and 181 us, (16, 14, 14) 292 and 357 us, (13, 10, 11) 270 and 313 us, but 329 and 262
        // us with the 33,124 determinants of (14, 3, 12); three holes: (11, 2, 8) 110 and 135 us, (12, 2, 9) 138 and 148
        // us (282 and 218 us for four vectors). With four electrons or holes of alpha: (10, 4, 8) 132 and 119 us.
        const int few = std::min(na, n - na), holes = n - nb;
        const bool sparse = few >= 2 && few <= 3 && (holes == 2 || holes == 3);
        *fast = s->nfull > (!sparse ? 8192 : holes == 2 ? 24000 : 10000);
    }
    return true;
}

void oz_build(const CIStrings* s, std::shared_ptr<OzSigma>& ozp, const double* H, const double* V, double E,
              int64_t bytes, cudaStream_t st) {
    const int n = s->norb, P = n * (n - 1) / 2;
    if (!ozp) {
        ozp = std::make_shared<OzSigma>();
        OzSigma& o = *ozp;
        o.s = s;
        o.max_elems = bytes / (int64_t)sizeof(long long);
        o.lead = oz_lead(std::max({s->a.m1 * s->b.m1, s->a.m2, s->b.m2}));
        for (int sp = 0; sp < 2; ++sp) {
            const SpinStrings& ss = s->spin(sp);
            OzSpin& t = o.spin[sp];
            t.m2 = ss.m2;
            t.nchunk = (ss.m2 + kOzN - 1) / kOzN;
            t.ksteps = (ss.m2 + 15) / 16;
            const int np = ss.k * (ss.k - 1) / 2, width = t.ksteps * 16, cols = t.nchunk * kOzN;
            TmpBuf<uint64_t> up2((size_t)ss.N2 * ss.m2, st);
            strings_up2(ss, s->binom.get(), up2.get(), st);
            t.up.reserve((size_t)ss.N2 * width);
            t.down.reserve((size_t)ss.N0 * np);
            t.pair.reserve((size_t)ss.N2 * cols);
            t.dpair.reserve((size_t)ss.N0 * np);
            t.b.reserve((size_t)ss.N2 * t.nchunk * t.ksteps * kOzStepBytes);
            t.bexp.reserve(P);
            t.diag.reserve(ss.N0);
            const int w = std::max(width, cols);
            k_oz_lists<<<ceil_div(ss.N2 * w, 256), 256, 0, st>>>(ss.N2, ss.m2, w, width, np, up2.get(), ss.str.get(),
                                                                t.up.get(), t.down.get(), cols, t.pair.get(),
                                                                t.dpair.get());
            F2G_LAUNCH("k_oz_lists");
        }
        o.kstr.reserve(s->b.N1);
        strings_masks(n, s->nb - 1, s->b.N1, s->binom.get(), o.kstr.get(), st);
        o.vb.reserve((size_t)n * n * kOzBlockBytes);
        o.vexp.reserve((size_t)n * 16);
        o.coul.reserve((size_t)s->a.N0 * n);
        o.plan(st);
    }
    OzSigma& o = *ozp;
    const int sb = oz_slack_b(o.lead);
    TmpBuf<double> g((size_t)P * P, st);
    for (int sp = 0; sp < 2; ++sp) {
        const SpinStrings& ss = s->spin(sp);
        OzSpin& t = o.spin[sp];
        k_oz_pairs<<<P, 128, 0, st>>>(n, 1.0 / (ss.k - 1), H, V, sb, g.get(), t.bexp.get());
        F2G_LAUNCH("k_oz_pairs");
        k_oz_b_ss<<<dim3((unsigned)ss.N2, (unsigned)t.nchunk), 96, 0, st>>>(P, t.m2, t.nchunk, t.ksteps, t.ksteps * 16,
                                                                           t.pair.get(), g.get(), t.bexp.get(),
                                                                           t.b.get());
        F2G_LAUNCH("k_oz_b_ss");
        k_oz_energies<<<ceil_div(ss.N0, 128), 128, 0, st>>>(n, ss.N0, ss.str.get(), H, V, sp == 0 ? E : 0.0,
                                                           t.diag.get(), sp == 0 ? o.coul.get() : nullptr);
        F2G_LAUNCH("k_oz_energies");
    }
    k_oz_vexp<<<n * 16, 32, 0, st>>>(n, V, sb, o.vexp.get());
    k_oz_b_ab<<<n * n, 32, 0, st>>>(n, V, o.vexp.get(), o.vb.get());
    F2G_LAUNCH("k_oz_b_ab");
}

// Ranges of alpha one-hole strings whose E fits the buffer, and the sigma rows each reaches
void OzSigma::plan(cudaStream_t st) {
    const int64_t N1a = s->a.N1, N1b = s->b.N1;
    ldE = (N1b + 15) / 16 * 16;
    const int64_t per = (int64_t)s->a.m1 * s->b.m1 * ldE;
    range_strings = std::max<int64_t>(1, max_elems / per);
    ranges.clear();
    if (range_strings >= N1a)
        return;
    const int ma = s->a.m1;
    std::vector<uint32_t> up((size_t)N1a * ma), list;
    F2G_CUDA(cudaMemcpyAsync(up.data(), s->a.up1.get(), up.size() * 4, cudaMemcpyDeviceToHost, st));
    F2G_CUDA(cudaStreamSynchronize(st));
    for (int64_t k0 = 0; k0 < N1a; k0 += range_strings) {
        OzRange r;
        r.k0 = k0;
        r.k1 = std::min(N1a, k0 + range_strings);
        r.j0 = (int64_t)list.size();
        for (size_t i = (size_t)r.k0 * ma; i < (size_t)r.k1 * ma; ++i)
            list.push_back(e_addr(up[i]));
        std::sort(list.begin() + r.j0, list.end());
        list.erase(std::unique(list.begin() + r.j0, list.end()), list.end());
        r.nrows = (int)((int64_t)list.size() - r.j0);
        ranges.push_back(r);
    }
    rows.reserve(list.size());
    F2G_CUDA(cudaMemcpyAsync(rows.get(), list.data(), list.size() * 4, cudaMemcpyHostToDevice, st));
    F2G_CUDA(cudaStreamSynchronize(st));
}

// Same spin: column tiles at a time, of `per` elements of E each; k_oz_sum_b takes four blocks of a grid's second
// dimension (65,535 at most) for one
static int64_t oz_tiles(const OzSigma& o, int64_t tiles, int64_t per) {
    return std::min({tiles, std::max<int64_t>(1, o.max_elems / per), int64_t(16383)});
}

void oz_limit(OzSigma& o, int64_t bytes, cudaStream_t st) {
    o.max_elems = bytes / (int64_t)sizeof(long long);
    for (OzScratch& w : o.scr)
        w.nvec = 0; // reserved again by the new plan
    o.plan(st);
}

void oz_reserve(OzSigma& o, int set, int nvec) {
    OzScratch& w = o.scr[set];
    nvec = std::max(1, nvec);
    if (nvec <= w.nvec)
        return;
    size_t e = 0, r = 0;
    for (int sp = 0; sp < 2; ++sp) {
        const SpinStrings& ss = o.s->spin(sp);
        const int64_t ncol = o.s->spin(1 - sp).N0, tiles = (ncol + kOzM - 1) / kOzM * nvec;
        const int64_t per = ss.N2 * ss.m2 * kOzM;
        const int64_t nt = oz_tiles(o, tiles, per);
        e = std::max<size_t>(e, (size_t)(nt * per));
        r = std::max<size_t>(r, (size_t)(nt * kOzM * ss.N2));
    }
    const int64_t nx = std::min<int64_t>(o.s->a.N1 * nvec, o.range_strings);
    e = std::max<size_t>(e, (size_t)(nx * o.s->a.m1 * o.s->b.m1 * o.ldE));
    r = std::max<size_t>(r, (size_t)(nx * o.ldE));
    w.E.reserve(e);
    w.rexp.reserve(r);
    w.nvec = nvec;
}

void oz_diag(const OzSigma& o, const double* C, double* S, int nvec, cudaStream_t st) {
    const CIStrings* s = o.s;
    k_oz_diag<<<dim3((unsigned)(s->a.N0 * nvec), (unsigned)ceil_div(s->b.N0, 256)), 256, 0, st>>>(
        s->a.N0, s->b.N0, s->norb, o.spin[0].diag.get(), o.spin[1].diag.get(), o.coul.get(), s->b.str.get(), C, S);
    F2G_LAUNCH("k_oz_diag");
}

template <bool SS, int MB>
static void oz_launch(OzArgs& a, int64_t nk, int64_t tiles, int max_ctas, cudaStream_t st) {
    const int sms = oz_sms();
    const int64_t room = 227 * 1024 - 1024;
    a.nt = (int)tiles;
    // the integers of a tile's D are kept for all its chunks while they and three K steps of B fit
    a.reuse = !SS && (int64_t)a.ksteps * kOzYBytes + 3 * kOzStepBytes <= room;
    const int64_t ybytes = SS ? 0 : (int64_t)(a.reuse ? a.ksteps : 2) * kOzYBytes;
    a.nbuf = (int)std::min<int64_t>(SS ? 6 : kOzMaxRing, (room - ybytes) / kOzStepBytes);
    const int64_t per = nk * (a.reuse ? 1 : a.nchunk);
    // tile ranges per hole string: six waves of work items where the tiles allow it
    a.tsplit = (int)std::max<int64_t>(1, std::min<int64_t>(tiles, 6 * (int64_t)sms / std::max<int64_t>(1, per)));
    const int64_t items = per * a.tsplit;
    const size_t smem = 1024 + ybytes + (size_t)a.nbuf * kOzStepBytes;
    F2G_CUDA(cudaFuncSetAttribute(k_oz<SS, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int64_t grid = std::min<int64_t>(items, max_ctas > 0 ? std::min(max_ctas, sms) : sms);
    k_oz<SS, MB><<<(unsigned)grid, kOzThreads, smem, st>>>(a, (uint32_t)items);
    F2G_LAUNCH("k_oz");
}

void oz_same_spin(OzSigma& o, int set, int spin, const double* C, double* S, int nvec, int max_ctas, const WaitCtl& wait,
                  cudaStream_t st) {
    const CIStrings* s = o.s;
    const SpinStrings& ss = s->spin(spin);
    OzSpin& t = o.spin[spin];
    OzScratch& w = o.scr[set];
    const int64_t ncol = s->spin(1 - spin).N0, nd = s->nfull, tpv = (ncol + kOzM - 1) / kOzM, tiles = tpv * nvec;
    const int64_t per = ss.N2 * ss.m2 * kOzM, step = oz_tiles(o, tiles, per);
    const int np = ss.k * (ss.k - 1) / 2;
    for (int64_t t0 = 0; t0 < tiles; t0 += step) {
        const int64_t nt = std::min(step, tiles - t0), nx = nt * kOzM;
        k_oz_rexp_ss<<<dim3((unsigned)ss.N2, (unsigned)ceil_div(nx, 256)), 256, 0, st>>>(
            C, nd, ncol, t.up.get(), t.ksteps * 16, t.m2, (int)tpv, ncol, t0, nx, oz_slack_a(o.lead), w.rexp.get());
        F2G_LAUNCH("k_oz_rexp_ss");
        OzArgs a{};
        a.C = C;
        a.cstride = nd;
        a.ld = ncol;
        a.E = w.E.get();
        a.ldE = nx;
        a.rexp = w.rexp.get();
        a.b = t.b.get();
        a.list = t.up.get();
        a.x0 = t0;
        a.ncol = (int)ncol;
        a.tpv = (int)tpv;
        a.m = t.m2;
        a.n = s->norb;
        a.nchunk = t.nchunk;
        a.ksteps = t.ksteps;
        a.wait = wait;
        oz_launch<true, 8>(a, ss.N2, nt, max_ctas, st);
        if (spin == 0) {
            k_oz_sum_a<<<dim3((unsigned)ss.N0, (unsigned)ceil_div(nx, 256)), 256, 0, st>>>(
                w.E.get(), w.rexp.get(), nx, t.m2, t.down.get(), t.dpair.get(), t.bexp.get(), np, (int)tpv, ncol, t0, nd, S,
                wait);
            F2G_LAUNCH("k_oz_sum_a");
        } else {
            k_oz_sum_b<<<dim3((unsigned)ceil_div(ss.N0, 32), (unsigned)(nx / 32)), 256, 0, st>>>(
                w.E.get(), w.rexp.get(), nx, t.m2, t.down.get(), t.dpair.get(), t.bexp.get(), np, ss.N0, (int)tpv, ncol, t0,
                nd, S, wait);
            F2G_LAUNCH("k_oz_sum_b");
        }
    }
}

template <int NB>
static void oz_sum_ab(const OzSigma& o, const OzScratch& w, const uint32_t* rows, int64_t nrows, int64_t v0, int64_t x0,
                      int64_t x1, double* S, const WaitCtl& wait, cudaStream_t st) {
    const CIStrings* s = o.s;
    k_oz_sum_ab<NB><<<dim3((unsigned)nrows, (unsigned)ceil_div(s->b.N0, 256)), 256, 0, st>>>(
        w.E.get(), w.rexp.get(), o.ldE, s->a.m1, s->b.m1, s->na, s->nb, s->norb, o.vexp.get(), rows, v0, s->a.N0,
        s->b.N0, s->a.N1, x0, x1,
        s->a.down1.get(), s->b.down1.get(), s->a.str.get(), S, wait);
    F2G_LAUNCH("k_oz_sum_ab");
}

void oz_opposite(OzSigma& o, int set, const double* C, double* S, int nvec, int max_ctas, const WaitCtl& wait,
                 cudaStream_t st) {
    const CIStrings* s = o.s;
    OzScratch& w = o.scr[set];
    const int64_t N1a = s->a.N1, N1b = s->b.N1, N0b = s->b.N0;
    auto part = [&](int64_t x0, int64_t x1, const uint32_t* rows, int64_t nrows, int64_t v0) {
        const size_t sm = (size_t)N0b * 2;
        if (sm > 48 * 1024)
            F2G_CUDA(cudaFuncSetAttribute(k_oz_rexp_ab, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
        k_oz_rexp_ab<<<(unsigned)(x1 - x0), 512, sm, st>>>(C, s->nfull, N0b, s->a.up1.get(), s->a.m1, N1a,
                                                           s->b.up1.get(), s->b.m1, N1b, x0, o.ldE,
                                                           oz_slack_a(o.lead), w.rexp.get());
        F2G_LAUNCH("k_oz_rexp_ab");
        OzArgs a{};
        a.C = C;
        a.cstride = s->nfull;
        a.ld = N0b;
        a.E = w.E.get();
        a.ldE = o.ldE;
        a.rexp = w.rexp.get();
        a.b = o.vb.get();
        a.up1 = s->a.up1.get();
        a.up1b = s->b.up1.get();
        a.kstr = o.kstr.get();
        a.nk = (int)N1a;
        a.x0 = x0;
        a.ncol = (int)N1b;
        a.m = s->a.m1;
        a.mb = s->b.m1;
        a.n = s->norb;
        a.nchunk = (s->a.m1 + 2) / 3;
        a.ksteps = s->a.m1;
        a.wait = wait;
        const int tiles = ceil_div(N1b, kOzM);
        if (a.mb <= 8)
            oz_launch<false, 8>(a, x1 - x0, tiles, max_ctas, st);
        else if (a.mb <= 10)
            oz_launch<false, 10>(a, x1 - x0, tiles, max_ctas, st);
        else
            oz_launch<false, 16>(a, x1 - x0, tiles, max_ctas, st);
        if (s->nb <= 4)
            oz_sum_ab<4>(o, w, rows, nrows, v0, x0, x1, S, wait, st);
        else if (s->nb <= 8)
            oz_sum_ab<8>(o, w, rows, nrows, v0, x0, x1, S, wait, st);
        else
            oz_sum_ab<16>(o, w, rows, nrows, v0, x0, x1, S, wait, st);
    };
    if (o.ranges.empty()) { // whole vectors per range
        const int64_t vs = std::max<int64_t>(1, o.range_strings / N1a);
        for (int64_t v = 0; v < nvec; v += vs) {
            const int64_t v1 = std::min<int64_t>(nvec, v + vs);
            part(v * N1a, v1 * N1a, nullptr, (v1 - v) * s->a.N0, v);
        }
        return;
    }
    for (int64_t v = 0; v < nvec; ++v)
        for (const OzRange& r : o.ranges)
            part(v * N1a + r.k0, v * N1a + r.k1, o.rows.get() + r.j0, r.nrows, v);
}

} // namespace f2g
