// Opposite-spin sigma (FP64) of a point-group-blocked space on the tensor cores, exact in digits.
//
// For an alpha 1-hole string Ka and the beta 1-hole strings Kb of irrep c,
//   E[Kb][(p, r)] = sum_(q, s) V[p, r, q, s] sgn C(Ka + q, Kb + s)
// over the orbital pairs of irrep(q) ^ irrep(s) = t = S ^ irrep(Ka) ^ c with q not in Ka; p, r run over the same pairs,
// 14 of them (16 with padding) for 14 orbitals in 8 irreps. That is a GEMM with K = N = 16 per Ka and c, 128 strings
// Kb to a tile: nearly free on the tensor cores, while the FP64 pipe (2 multiply-adds per clock and SM; it takes
// the pairs with s or r occupied in Kb along, 196 products for 64 that count) needs 3.0 ms for the 9 million hole
// pairs of CAS(14,14) and took 5.8 ms.
//
// The rows of the vector, scaled by their largest exponents e(Ia) to integers of 62 bits, are cut into eight FP16 digits
// once (k_sy_expand: rows (Ia, s) over the Kb of the one irrep that Ia and s leave). The integrals take the rows' scales
// along: those of a Ka and an output pair (p, r) are the V[p, r, q, s] 2^e(Ka + q), scaled by the largest of them
// (k_sy_integrals, in the order of each Ka's pairs, sgn(Ka, q) included). k_sy_gemm's A operand is contiguous along
// M = Kb, so a row's digits go from there to core matrices by 16-byte copies. Products of digits i, j with i + j <= 7 are
// kept, sums of at most 64 rows of eight products are exact in FP32, and an element of E is their 96-bit sum rounded
// once. k_sy_sum adds sgn E into sigma, a thread per determinant in a fixed order.
//
// Accuracy. A product of E[Kb][(p, r)] loses less than 2^-56 of the largest |V[p, r, q, s]| max_Ib |C(Ka + q, Ib)| in its
// sum: 2^-61 each from the element and the integral, at most 2^-57.2 from the digit products left out. Compared with a
// sum in FP64 that is less in the norm of the rows that meet in a Ka, and more for an element whose own products are
// all 2^-6 and less of that largest one. (With one scale for the whole vector that held for its norm alone: rows at 1e-12
// of the largest were left with 22 bits.)
//
// Bound: operand copies and drains by turns. CAS(14,14) in 8 irreps (1,472,512 determinants), opposite-spin term: 5.82 ->
// 1.7 ms (k_sy_gemm 1.15 ms; 1.09 ms with one scale for all output pairs; 0.15 ms more with unswizzled core matrices,
// whose 16-byte copies take a wavefront each; k_sy_sum 0.34 ms, k_sy_expand 0.10 ms).
#include <algorithm>

#include "common.cuh"
#include "digit_mma.cuh"
#include "sym_digits.cuh"

namespace f2g {

namespace {

constexpr int kYM = 128;
constexpr int kYProd = 4, kYEpi = 16;
constexpr int kYThreads = (kYProd + kYEpi + 1) * 32;
constexpr int kYA = 8 * kYM * 16 * 2;               // digits of a K step's 16 pairs x 128 strings
constexpr int kYStagesMax = 6;
constexpr int kYSmem = 216 * 1024;
constexpr int64_t kYBytes = int64_t(1) << 31;       // digits of 128 strings Kb and of the integrals at most
constexpr int kYUnit = 88 - 68;                     // exponent of the digits' sums, see below
constexpr int kYBadRow = 1 << 15; // with a row's exponent: it holds an infinity or NaN
constexpr int kYSlow = 1 << 16; // with the first exponent of four: some need the general conversion
constexpr int kYBad = 1 << 14;    // exponent of an output pair with an integral that is not finite

struct SymShared {
    alignas(8) uint64_t full[kYStagesMax], empty[kYStagesMax], acc_full[4], acc_empty[4], drain;
    uint32_t tmem_base;
    volatile int abort;
    uint32_t row[kYProd][kSymSlots]; // [copy warp][pair]: its digits in z, in 16 bytes; ~0: none
};

struct SymArgs {
    const uint4 *z, *b;
    double* e;
    const int* ecol;
    WaitCtl wait;
    const uint32_t* up_a;
    const int8_t* hka;
    int64_t ka0; // first Ka
    int ma, n, most, slots, ksteps, tiles, chunk, nirrep, nbuf, stages, stage_bytes;
    OrbSym os;
};

// ec[Ia]: largest biased exponent of the finite elements of row Ia of the vector, at least 1, with kYBadRow if there are
// others (then ec[N0a] is set: k_sy_not_finite adds their products); a block per row
__global__ void __launch_bounds__(256) k_sy_rowexp(int64_t N0a, int64_t N0b, const double* __restrict__ C, int* __restrict__ ec) {
    const uint32_t* hi = reinterpret_cast<const uint32_t*>(C + blockIdx.x * N0b) + 1;
    uint32_t m = 0;
    bool bad = false;
#pragma unroll 4
    for (int64_t i = threadIdx.x; i < N0b; i += 256) {
        const uint32_t x = __ldg(hi + 2 * i) & 0x7fffffffu;
        bad |= x >= 0x7ff00000u;
        m = max(m, x < 0x7ff00000u ? x : 0u);
    }
    m = __reduce_max_sync(0xffffffffu, m);
    bad = __syncthreads_or(bad);
    __shared__ uint32_t w[8];
    if ((threadIdx.x & 31) == 0)
        w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i)
            m = max(m, w[i]);
        ec[blockIdx.x] = max((int)(m >> 20), 1) | (bad ? kYBadRow : 0);
        if (bad)
            atomicExch(ec + N0a, 1);
    }
}

__global__ void k_sy_tab(const uint32_t* __restrict__ up_b, int mb, int64_t N1b, int n, int lmax,
                         const int32_t* __restrict__ kpos, uint32_t* __restrict__ tab) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= N1b * mb)
        return;
    const int32_t p = kpos[t / mb];
    const uint32_t e = up_b[t];
    tab[((int64_t)(p >> 24) * n + e_orb(e)) * lmax + (p & 0xffffff)] = e_addr(e) | (uint32_t)e_neg(e) << 31;
}

__device__ __forceinline__ void digits8(const uint64_t (&y)[8], uint4* dst, int stride) {
#define F2G_DIGIT(D)                                                                                               \
    dst[D * stride] = make_uint4(gram_half2<D>(y[0], y[1]), gram_half2<D>(y[2], y[3]), gram_half2<D>(y[4], y[5]),   \
                                 gram_half2<D>(y[6], y[7]))
    F2G_DIGIT(0);
    F2G_DIGIT(1);
    F2G_DIGIT(2);
    F2G_DIGIT(3);
    F2G_DIGIT(4);
    F2G_DIGIT(5);
    F2G_DIGIT(6);
    F2G_DIGIT(7);
#undef F2G_DIGIT
}

// z[(Ia, s)][64 positions][digit][64]: C(Ia, Kb + s) sgn for the Kb of irrep S ^ irrep(Ia) ^ irrep(s), positions
// pos0 .. pos0 + chunk
__global__ void __launch_bounds__(256) k_sy_expand(const double* __restrict__ C, int64_t N0a, int64_t N0b, int n, int lmax,
                                                   int pos0, int chunk, const int8_t* __restrict__ hja, const __grid_constant__ OrbSym os,
                                                   const uint32_t* __restrict__ tab, const int* __restrict__ ec,
                                                   uint4* __restrict__ z) {
    __shared__ uint4 sm[8][256]; // a warp's digits, written from here in whole lines
    const int g8 = chunk >> 3, lane = threadIdx.x & 31; // g8 and with it the total: multiples of 16
    uint4* my = sm[threadIdx.x >> 5];
    const int64_t total = N0a * n * g8;
    for (int64_t t0 = blockIdx.x * (int64_t)256 + (threadIdx.x & ~31); t0 < total; t0 += (int64_t)gridDim.x * 256) {
        const int64_t t = min(t0 + lane, total - 1);
        const int g = (int)(t % g8);
        const int64_t r = t / g8, Ia = r / n;
        const int s = (int)(r - Ia * n), e = __ldg(ec + Ia), E = e & (kYBadRow - 1);
        const uint4* src = reinterpret_cast<const uint4*>(tab + ((int64_t)(os.S ^ hja[Ia] ^ os.h[s]) * n + s) * lmax + pos0 + g * 8);
        const uint4 a0 = __ldg(src), a1 = __ldg(src + 1);
        const uint32_t a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        uint64_t y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            double x = a[j] == ~0u ? 0.0 : __ldg(C + Ia * N0b + (a[j] & 0x7fffffffu));
            if (e >= kYBadRow && !isfinite(x))
                x = 0.0;
            y[j] = gram_digits(x, a[j] >> 31, E);
        }
        uint4 q[8];
        digits8(y, q, 1);
#pragma unroll
        for (int d = 0; d < 8; ++d)
            my[lane * 8 + (d ^ (lane & 7))] = q[d];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int o = (i & 3) * 8 + (lane & 7), d = (i >> 2) * 4 + (lane >> 3); // eight lanes: 128 bytes
            if (t0 + o < total)
                z[((t0 + o) >> 3) * 64 + d * 8 + ((t0 + o) & 7)] = my[o * 8 + (d ^ (o & 7))];
        }
        __syncwarp();
    }
}

// b[(Ka, t)][K step][group of 8 (q, s)][digit][(p, r)][8]: sgn(Ka, q) V[p, r, q, s] 2^ec(Ka + q) below 2^ecol;
// ecol[(Ka, t)][(p, r)]: the largest exponent of these products, kYBad if one is not finite (and kYSlow); a block per Ka
__global__ void __launch_bounds__(256) k_sy_integrals(const double* __restrict__ V, int n, int ma, const uint32_t* __restrict__ up_a,
                                                      const __grid_constant__ OrbSym os, int slots, const int* __restrict__ ec,
                                                      int* __restrict__ ecol, uint4* __restrict__ b) {
    __shared__ uint8_t q_of[8][kSymSlots], s_of[8][kSymSlots], neg_of[8][kSymSlots];
    __shared__ int16_t ec_of[8][kSymSlots];
    __shared__ int cnt[8], col[8 * kSymSlots];
    const int64_t Ka = blockIdx.x;
    if (threadIdx.x < os.nirrep) {
        const int t = threadIdx.x;
        int c = 0;
        for (int i = 0; i < ma; ++i) {
            const uint32_t e = up_a[Ka * ma + i];
            const int q = e_orb(e), h = t ^ os.h[q], x = ec[e_addr(e)] & (kYBadRow - 1);
            for (int j = 0; j < os.cnt[h]; ++j, ++c) {
                q_of[t][c] = (uint8_t)q;
                s_of[t][c] = (uint8_t)os.list[h][j];
                neg_of[t][c] = (uint8_t)e_neg(e);
                ec_of[t][c] = (int16_t)x;
            }
        }
        cnt[t] = c;
    }
    __syncthreads();
    const int groups = slots >> 3, items = os.nirrep * groups * slots, stride = os.nirrep * slots;
    for (int i = threadIdx.x; i < stride; i += 256)
        col[i] = 2; // of a zero below the smallest scale
    __syncthreads();
    double x[8];
    auto load = [&](int i, int& o, int& t, int& g) { // eight integrals of one output pair
        o = i % slots;
        g = i / slots % groups;
        t = i / (slots * groups);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = g * 8 + j;
            x[j] = o < cnt[t] && k < cnt[t]
                       ? __ldg(V + (((int64_t)q_of[t][o] * n + s_of[t][o]) * n + q_of[t][k]) * n + s_of[t][k])
                       : 0.0;
        }
    };
    int o, t, g;
    for (int i = threadIdx.x; i < items; i += 256) {
        load(i, o, t, g);
        int m = 2;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = g * 8 + j, ev = (int)((__double_as_longlong(x[j]) >> 52) & 0x7ff);
            if (o < cnt[t] && k < cnt[t])
                m = max(m, ev == 0x7ff ? kYBad : max(ev, 1) + ec_of[t][k]);
        }
        atomicMax(col + t * slots + o, m);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < stride; i += 256) {
        int x = col[i];
        if ((i & 3) == 0) {
            const int lo = min(min(x, col[i + 1]), min(col[i + 2], col[i + 3]));
            const int hi = max(max(x, col[i + 1]), max(col[i + 2], col[i + 3]));
            if (lo + kYUnit - 32 < kOzSafeLo || hi + kYUnit > kOzSafeHi)
                x |= kYSlow;
        }
        ecol[Ka * stride + i] = x;
    }
    for (int i = threadIdx.x; i < items; i += 256) {
        if (items > 256)
            load(i, o, t, g); // with 16 pairs in 8 irreps every thread still has its own
        uint64_t y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int k = g * 8 + j;
            y[j] = gram_digits(x[j], neg_of[t][k], o < cnt[t] && k < cnt[t] ? col[t * slots + o] - ec_of[t][k] : 1);
        }
        digits8(y, b + ((Ka * os.nirrep + t) * groups + g) * 8 * slots + o, slots);
    }
}

// item: Ka, irrep of Kb, tile of 128 positions
__device__ __forceinline__ void sym_item(const SymArgs& a, int64_t w, int64_t& Ka, int& c, int& tile) {
    tile = (int)(w % a.tiles);
    const int64_t r = w / a.tiles;
    c = (int)(r % a.nirrep);
    Ka = a.ka0 + r / a.nirrep;
}

__device__ __forceinline__ void sym_next(const SymArgs& a, int64_t& Ka, int& c, int& tile) { // the item after it
    if (++tile < a.tiles)
        return;
    tile = 0;
    if (++c < a.nirrep)
        return;
    c = 0;
    ++Ka;
}

__global__ void __launch_bounds__(kYThreads, 1) k_sy_gemm(const __grid_constant__ SymArgs a, int64_t nitems) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SymShared& sh = *reinterpret_cast<SymShared*>(smem_raw);
    const uint32_t ring = smem_u32(smem_raw) + ((sizeof(SymShared) + 1023) / 1024) * 1024;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const volatile int* abort = &sh.abort;
    if (tid == 0) {
        for (int i = 0; i < kYStagesMax; ++i) {
            mbar_init(smem_u32(&sh.full[i]), kYProd * 32);
            mbar_init(smem_u32(&sh.empty[i]), 1);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(smem_u32(&sh.acc_full[i]), 1);
            mbar_init(smem_u32(&sh.acc_empty[i]), kYEpi);
        }
        mbar_init(smem_u32(&sh.drain), 1);
        sh.abort = 0;
    }
    if (warp == kYProd + kYEpi) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.tmem_base)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_before();
    __syncthreads();
    fence_after();
    constexpr uint32_t tmem = 0; // all 512 columns are this block's
    auto give_up = [&]() {
        atomicExch(a.wait.err, 1);
        sh.abort = 1;
    };
    const uint32_t cols = 8u * a.slots; // accumulators of an item: eight groups
    // neighbouring items, so that a Ka's list is read once per block, not once per item and waited for
    const int64_t w0 = blockIdx.x * nitems / gridDim.x, w1 = (blockIdx.x + 1) * nitems / gridDim.x;

    if (warp < kYProd) {
        // ---- copies: a K step (16 pairs) per stage, four pairs per warp; eight lanes take 64 strings of a digit
        uint32_t slot = 0, phase = 1, e = 0;
        int64_t last = -1;
        int hk = 0;
        bool ok = true;
        int64_t Ka;
        int c, tile;
        sym_item(a, min(w0, nitems - 1), Ka, c, tile);
        for (int64_t w = w0; ok && w < w1; ++w, sym_next(a, Ka, c, tile)) {
            if (Ka != last) {
                last = Ka;
                hk = a.hka[Ka];
                if (lane < a.ma)
                    e = __ldg(a.up_a + Ka * a.ma + lane);
            }
            const int t = a.os.S ^ hk ^ c;
            __syncwarp();
            for (int i = lane; i < kSymSlots; i += 32)
                sh.row[warp][i] = ~0u;
            __syncwarp();
            int at = 0, h = 0, cn = 0;
            if (lane < a.ma) {
                h = t ^ a.os.h[e_orb(e)];
                cn = a.os.cnt[h];
            }
            int incl = cn;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o)
                    incl += y;
            }
            at = incl - cn;
            for (int j = 0; j < cn; ++j)
                sh.row[warp][at + j] = (uint32_t)((e_addr(e) * (uint32_t)a.n + a.os.list[h][j]) * (uint32_t)a.chunk);
            __syncwarp();
            const uint4* zt = a.z + tile * kYM + (lane & 7);
            const uint4* bt = a.b + (Ka * a.nirrep + t) * (int64_t)(a.slots * a.slots) + tid;
            for (int ks = 0; ks < a.ksteps; ++ks) {
                if (!mbar_wait_warp(smem_u32(&sh.empty[slot]), phase, abort)) {
                    give_up();
                    ok = false;
                    break;
                }
                const uint32_t dst = ring + slot * a.stage_bytes;
                const int pair = warp * 4 + (lane >> 3), piece = lane & 7;
                const uint32_t r = sh.row[warp][ks * 16 + pair];
                const uint4* src = zt + (r == ~0u ? 0 : r);
                const uint32_t to = dst + pair * 128 + ((piece ^ pair) & 7) * 16, bytes = r == ~0u ? 0 : 16;
#pragma unroll
                for (int d = 0; d < 8; ++d)
#pragma unroll
                    for (int mb = 0; mb < 2; ++mb)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to + d * (kYM * 32) + mb * 2048),
                                     "l"(src + (mb * 8 + d) * 8), "r"(bytes));
                for (int i = 0; i < a.slots / 8; ++i) // 16 slots pieces in all, contiguous
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + kYA + (i * 128 + tid) * 16),
                                 "l"(bt + ks * 16 * a.slots + i * 128));
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&sh.full[slot]))
                             : "memory");
                if (++slot == (uint32_t)a.stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < kYProd + kYEpi) {
        // ---- drains: a row's eight groups into one FP64 number, four columns at a time
        const int quarter = warp & 3, part = (warp - kYProd) >> 2;
        uint32_t buf = 0, phase = 0;
        auto exponents = [&](int64_t Ka, int c) { // of an item's output pairs, four to a vector
            return reinterpret_cast<const int4*>(a.ecol + (Ka * a.nirrep + (a.os.S ^ __ldg(a.hka + Ka) ^ c)) * a.slots);
        };
        const int last4 = a.slots / 4 - 1;
        int64_t nKa; // the next item: its exponents are loaded an item ahead, so that nothing waits for them
        int nc, ntile;
        sym_item(a, min(w0, nitems - 1), nKa, nc, ntile);
        const int4* ecol_next = exponents(nKa, nc);
        int4 ev_next = __ldg(ecol_next + min(part, last4));
        for (int64_t w = w0; w < w1; ++w) {
            const int64_t Ka = nKa;
            const int c = nc, tile = ntile;
            const int4* ecol = ecol_next;
            int4 ev = ev_next;
            if (w + 1 < w1) {
                sym_next(a, nKa, nc, ntile);
                if (nc != c || nKa != Ka) {
                    ecol_next = exponents(nKa, nc);
                    ev_next = __ldg(ecol_next + min(part, last4));
                }
            }
            if (!mbar_wait_warp(smem_u32(&sh.acc_full[buf]), phase, abort)) {
                give_up();
                break;
            }
            fence_after();
            const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + buf * cols;
            const int64_t pitch = (int64_t)a.nirrep * a.chunk;
            double* out = a.e + (Ka - a.ka0) * a.most * pitch + (int64_t)c * a.chunk + tile * kYM + quarter * 32 + lane;
            for (int b = part; b * 4 < a.most; b += kYEpi / 4) {
                uint32_t r[32];
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    tmem_ld4(at + g * a.slots + b * 4, r + 4 * g);
                const bool safe = !(ev.x & kYSlow);
                const int col[4] = {ev.x & (kYSlow - 1), ev.y, ev.z, ev.w};
                if (b + kYEpi / 4 < a.most / 4)
                    ev = __ldg(ecol + b + kYEpi / 4);
                tmem_wait_ld();
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    int G[8], P[4];
#pragma unroll
                    for (int g = 0; g < 8; ++g)
                        G[g] = __float2int_rn(__uint_as_float(r[4 * g + j]));
#pragma unroll
                    for (int g = 0; g < 4; ++g) // at most 64 rows of 6 products of 2^14 in the leading one: below 2^31
                        P[g] = G[2 * g] * 256 + G[2 * g + 1];
                    long long hi = mad_wide(P[0], 65536, P[1]), lo = mad_wide(P[2], 65536, P[3]);
                    // hi 2^32 + lo, |hi| < 2^47: its leading 64 bits, then one rounding
                    hi += lo >> 32;
                    uint32_t low = (uint32_t)lo;
                    const bool neg = hi < 0;
                    if (neg) {
                        low = 0u - low;
                        hi = ~hi + (low == 0);
                    }
                    const int sft = min(32, __clz((uint32_t)((unsigned long long)hi >> 16)) + 14);
                    long long T = (hi << sft) | (long long)((unsigned long long)low >> (32 - sft));
                    T = neg ? -T : T;
                    // units of T: 2^(32 - sft) 2^56 2^(col - 2 1084)
                    const int e = col[j] + kYUnit - sft;
                    out[(b * 4 + j) * pitch] = safe ? oz_double(T, (e - 1016) << 20, -(1 << 20))
                                               : col[j] >= kYBad ? __longlong_as_double(0x7ff8000000000000ll)
                                                                 : oz_value(T, e);
                }
            }
            fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(smem_u32(&sh.acc_empty[buf]));
            if (++buf == (uint32_t)a.nbuf) {
                buf = 0;
                phase ^= 1;
            }
        }
    } else {
        // ---- MMAs
        const uint32_t el = elect_lane();
        const uint32_t ns = (uint32_t)a.slots, lbo_b = 8 * ns * 16;
        uint32_t slot = 0, phase = 0, buf = 0, buf_phase = 1;
        bool ok = a.wait.polls == 0; // with a limit on the tries (for tests) the first wait counts as given up
        for (int64_t w = w0; ok && w < w1; ++w) {
            if (!mbar_wait_warp(smem_u32(&sh.acc_empty[buf]), buf_phase, abort)) {
                ok = false;
                break;
            }
            const uint32_t acc = tmem + buf * cols;
            for (int ks = 0; ks < a.ksteps; ++ks) {
                if (!mbar_wait_warp(smem_u32(&sh.full[slot]), phase, abort)) {
                    ok = false;
                    break;
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic copies, read by the MMAs
                fence_after();
                // A: atoms of 8 pairs x 64 strings (rows of 128 bytes, swizzled), next 64 strings 2,048 bytes on, next
                // 8 pairs 1,024
                const uint64_t ad = smem_desc(ring + slot * a.stage_bytes, 2048, 1024) | (2ull << 61);
                const uint64_t bd = smem_desc(ring + slot * a.stage_bytes + kYA, lbo_b, 128);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    uint32_t n = (uint32_t)(8 - i) * ns, dcol = acc + i * ns;
                    uint64_t b = bd;
                    if (n > 256) {
                        mma_ss(dcol, ad + i * (kYM * 32 / 16), b, 256, ks > 0 || i > 0, el, kMajorA);
                        n -= 256, dcol += 256, b += 256;
                    }
                    mma_ss(dcol, ad + i * (kYM * 32 / 16), b, n, ks > 0 || i > 0, el, kMajorA);
                }
                mma_commit(smem_u32(&sh.empty[slot]), el);
                if (++slot == (uint32_t)a.stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
            if (ok)
                mma_commit(smem_u32(&sh.acc_full[buf]), el);
            if (++buf == (uint32_t)a.nbuf) {
                buf = 0;
                buf_phase ^= 1;
            }
        }
        if (!ok)
            give_up();
        mma_commit(smem_u32(&sh.drain), el); // the instructions in flight end before the block leaves
        mbar_wait_warp(smem_u32(&sh.drain), 0, nullptr);
    }
    __syncwarp();
    __syncthreads();
    if (warp == kYProd + kYEpi) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// sigma(Ja, Jb) += sum over p in Ja, r in Jb with Ja - p and Jb - r in this chunk; a block per Ja and 256 strings Jb
__global__ void __launch_bounds__(256) k_sy_sum(int64_t N0b, int n, int na, int nb, int ma, int most, int64_t ka0, int64_t ka1, int pos0, int chunk,
                                                const __grid_constant__ OrbSym os, const uint32_t* __restrict__ down_a,
                                                const uint32_t* __restrict__ up_a, const uint32_t* __restrict__ down_b,
                                                const int32_t* __restrict__ kpos, const int8_t* __restrict__ hja,
                                                const int32_t* __restrict__ jb, const int32_t* __restrict__ njb_of, int64_t njb,
                                                const double* __restrict__ E, double* __restrict__ sig, const WaitCtl wait) {
    __shared__ int off[32][8]; // [p of Ja][t]: the first pair of p
    const int64_t Ja = blockIdx.x;
    const int h = os.S ^ hja[Ja], cnt = njb_of[h];
    if ((int64_t)blockIdx.y * 256 >= cnt)
        return;
    for (int i = threadIdx.x; i < na * os.nirrep; i += 256) {
        const int pi = i / os.nirrep, t = i % os.nirrep;
        const uint32_t ep = down_a[Ja * na + pi];
        int o = 0;
        for (int q = 0; q < ma; ++q) { // pairs in the order of Ka's list
            const int oq = e_orb(up_a[(int64_t)e_addr(ep) * ma + q]);
            if (oq == e_orb(ep))
                break;
            o += os.cnt[t ^ os.h[oq]];
        }
        off[pi][t] = o;
    }
    bool any = false;
    for (int pi = 0; pi < na; ++pi) {
        const int64_t Ka = e_addr(down_a[Ja * na + pi]);
        any |= Ka >= ka0 && Ka < ka1;
    }
    if (!any)
        return;
    __syncthreads();
    const int64_t at = (int64_t)blockIdx.y * 256 + threadIdx.x;
    if (at >= cnt)
        return;
    const int64_t Jb = jb[h * njb + at], pitch = (int64_t)os.nirrep * chunk;
    double* out = sig + Ja * N0b + Jb;
    double acc = *out;
    for (int pi = 0; pi < na; ++pi) {
        const uint32_t ep = __ldg(down_a + Ja * na + pi);
        const int hp = os.h[e_orb(ep)];
        const int64_t Ka = e_addr(ep);
        if (Ka < ka0 || Ka >= ka1)
            continue;
        const double* e0 = E + (Ka - ka0) * most * pitch;
#pragma unroll 8
        for (int j = 0; j < nb; ++j) {
            const uint32_t er = __ldg(down_b + Jb * nb + j);
            const int r = e_orb(er), kp = __ldg(kpos + e_addr(er)), pos = (kp & 0xffffff) - pos0;
            if (pos >= 0 && pos < chunk) {
                const double x = __ldg(e0 + (off[pi][hp ^ os.h[r]] + os.pos[r]) * pitch + (int64_t)(kp >> 24) * chunk + pos);
                acc += (e_neg(ep) ^ e_neg(er)) ? -x : x;
            }
        }
    }
    *out = waited(acc, wait);
}

// Elements of the vector that are not finite count as zero in E. If there are any, their products are added here, as a
// sum in FP64 would have them.
__global__ void __launch_bounds__(256) k_sy_not_finite(int64_t N0a, int64_t N0b, int n, int na, int nb, int ma, const __grid_constant__ OrbSym os,
                                                       const uint32_t* __restrict__ down_a, const uint32_t* __restrict__ up_a,
                                                       const uint32_t* __restrict__ down_b, const int32_t* __restrict__ kpos,
                                                       const int8_t* __restrict__ hja, const int32_t* __restrict__ jb,
                                                       const int32_t* __restrict__ njb_of, int64_t njb, const uint32_t* __restrict__ tab,
                                                       int lmax, const int* __restrict__ ec, const double* __restrict__ C,
                                                       const double* __restrict__ V, double* __restrict__ sig) {
    if (!ec[N0a])
        return;
    for (int64_t Ja = blockIdx.x; Ja < N0a; Ja += gridDim.x)
        for (int i = 0; i < na * ma; ++i) {
            const uint32_t ep = down_a[Ja * na + i / ma], eq = up_a[(int64_t)e_addr(ep) * ma + i % ma];
            const int64_t Ia = e_addr(eq);
            if (ec[Ia] < kYBadRow)
                continue;
            const int p = e_orb(ep), q = e_orb(eq), h = os.S ^ hja[Ja], cnt = njb_of[h];
            for (int at = threadIdx.x; at < cnt; at += 256) {
                const int64_t Jb = jb[h * njb + at];
                double acc = 0.0;
                for (int j = 0; j < nb; ++j) {
                    const uint32_t er = down_b[Jb * nb + j];
                    const int kp = kpos[e_addr(er)], hb = kp >> 24, hs = os.S ^ hja[Ia] ^ hb;
                    for (int l = 0; l < os.cnt[hs]; ++l) {
                        const int s = os.list[hs][l];
                        const uint32_t es = tab[((int64_t)hb * n + s) * lmax + (kp & 0xffffff)];
                        if (es == ~0u)
                            continue;
                        const double x = C[Ia * N0b + (es & 0x7fffffffu)];
                        if (!isfinite(x)) {
                            const double y = V[(((int64_t)p * n + e_orb(er)) * n + q) * n + s] * x;
                            acc += (e_neg(ep) ^ e_neg(er) ^ e_neg(eq) ^ (es >> 31)) ? -y : y;
                        }
                    }
                }
                if (acc != 0.0)
                    sig[Ja * N0b + Jb] += acc;
            }
        }
}

int sm_total() {
    int dev = 0, sms = 0;
    F2G_CUDA(cudaGetDevice(&dev));
    F2G_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return sms;
}

} // namespace

std::shared_ptr<SymDigits> sym_digits_build(const CIStrings* s, const OppositeSym& t) {
    const int n = s->norb;
    int nir = 1; // closed under products, whatever irreps occur
    while (nir < t.os.nirrep || nir <= t.os.S)
        nir *= 2;
    const int64_t N1a = s->a.N1, N1b = s->b.N1, N0a = s->a.N0, N0b = s->b.N0;
    if (N1a == 0 || N1b == 0 || s->a.m1 > 32 || s->na > 32 || nir > 8 || N0a * n * 16 * 128 > kYBytes)
        return nullptr;
    auto d = std::make_shared<SymDigits>();
    d->os = t.os;
    d->os.nirrep = nir;
    std::vector<uint64_t> bt(kBinomLd * kBinomLd);
    for (int a = 0; a < kBinomLd; ++a)
        for (int b = 0; b < kBinomLd; ++b)
            bt[a * kBinomLd + b] = host_binom(a, b);
    auto irrep = [&](uint64_t m) {
        int h = 0;
        for (; m; m &= m - 1)
            h ^= t.os.h[__builtin_ctzll(m)];
        return h;
    };
    // pairs per (Ka, t)
    std::vector<int8_t> hka(N1a), hja(N0a);
    int most = 0;
    for (int64_t K = 0; K < N1a; ++K) {
        const uint64_t m = string_unrank((uint64_t)K, n, s->na - 1, bt.data());
        hka[K] = (int8_t)irrep(m);
        for (int u = 0; u < nir; ++u) {
            int c = 0;
            for (int q = 0; q < n; ++q)
                if (!(m >> q & 1))
                    c += t.os.cnt[u ^ t.os.h[q]];
            most = std::max(most, c);
        }
    }
    // Below some 2e7 products the FP64 kernel's one launch is the faster one: sigma of (10 orbitals, 5, 5) in 8 and 4 irreps
    // (5e6 and 1.4e7 products) 35 and 13 us faster, in 2 (4e7) 246 and 162 us, of (12, 6, 6) in 8 (1.2e8) 637 and 341 us
    if (most > kSymSlots || (double)N1a * (double)N1b * most * most < 2e7)
        return nullptr;
    d->slots = (most + 15) / 16 * 16;
    for (int64_t I = 0; I < N0a; ++I)
        hja[I] = (int8_t)irrep(string_unrank((uint64_t)I, n, s->na, bt.data()));
    std::vector<int32_t> kpos(N1b), count(8, 0);
    for (int64_t K = 0; K < N1b; ++K) {
        const int h = irrep(string_unrank((uint64_t)K, n, s->nb - 1, bt.data()));
        kpos[K] = h << 24 | count[h]++;
    }
    d->lmax = (*std::max_element(count.begin(), count.end()) + 127) / 128 * 128;
    std::vector<std::vector<int32_t>> jb(8);
    for (int64_t J = 0; J < N0b; ++J)
        jb[irrep(string_unrank((uint64_t)J, n, s->nb, bt.data()))].push_back((int32_t)J);
    for (const auto& x : jb)
        d->njb = std::max<int64_t>(d->njb, (int64_t)x.size());
    std::vector<int32_t> flat((size_t)(8 * d->njb), 0), nj(8);
    for (int h = 0; h < 8; ++h) {
        nj[h] = (int32_t)jb[h].size();
        std::copy(jb[h].begin(), jb[h].end(), flat.begin() + h * d->njb);
    }
    d->most = (most + 3) / 4 * 4; // stored four at a time
    if (N1a * nir * (int64_t)d->slots * d->slots * 16 > kYBytes)
        return nullptr;
    sym_digits_plan(*d, s, kYBytes);
    auto put = [](auto& buf, const auto& v) {
        buf.reserve(v.size());
        F2G_CUDA(cudaMemcpy(buf.get(), v.data(), v.size() * sizeof(v[0]), cudaMemcpyHostToDevice));
    };
    put(d->hka, hka);
    put(d->hja, hja);
    put(d->kpos, kpos);
    put(d->jb, flat);
    put(d->njb_of, nj);
    const size_t nt = (size_t)8 * n * d->lmax;
    d->tab.reserve(nt);
    F2G_CUDA(cudaMemset(d->tab.get(), 0xff, nt * sizeof(uint32_t)));
    k_sy_tab<<<(unsigned)ceil_div(N1b * s->b.m1, 256), 256>>>(s->b.up1.get(), s->b.m1, N1b, n, d->lmax, d->kpos.get(),
                                                              d->tab.get());
    F2G_LAUNCH("k_sy_tab");
    F2G_CUDA(cudaStreamSynchronize(0));
    return d;
}

// positions at a time: the vector's digits within `bytes`; then hole strings Ka at a time: E within twice that
void sym_digits_plan(SymDigits& d, const CIStrings* s, int64_t bytes) {
    const int64_t N0a = s->a.N0, N1a = s->a.N1, n = s->norb;
    const int64_t most128 = std::max<int64_t>(1, bytes / (N0a * n * 16 * 128)), all128 = d.lmax / 128;
    const int64_t parts = (all128 + most128 - 1) / most128;
    d.chunk = (int)((all128 + parts - 1) / parts * 128);
    const int64_t mostka = std::max<int64_t>(1, 2 * bytes / ((int64_t)d.most * d.os.nirrep * d.chunk * 8));
    const int64_t kparts = (N1a + mostka - 1) / mostka;
    d.ka = (N1a + kparts - 1) / kparts;
}

void sym_digits_reserve(SymDigits& d, const CIStrings* s, int set) {
    SymDigits::Scratch& w = d.set[set];
    const int nir = d.os.nirrep;
    w.z.reserve((size_t)(s->a.N0 * s->norb * d.chunk));
    w.b.reserve((size_t)(s->a.N1 * nir * d.slots * d.slots));
    w.e.reserve((size_t)(d.ka * d.most * nir * d.chunk));
    w.ec.reserve((size_t)s->a.N0 + 1);
    w.ecol.reserve((size_t)(s->a.N1 * nir * d.slots));
}

void sym_digits_run(SymDigits& d, const CIStrings* s, int set, const double* V, const double* C, double* sig, int nvec,
                    int max_ctas, const WaitCtl& wait, cudaStream_t st) {
    if (set == 0)
        sym_digits_reserve(d, s, 0);
    SymDigits::Scratch& w = d.set[set];
    const int n = s->norb, nir = d.os.nirrep;
    const int64_t N0a = s->a.N0, N0b = s->b.N0;
    const int sms = sm_total(), ctas = max_ctas > 0 ? std::min(max_ctas, sms) : sms;
    SymArgs a{};
    a.z = w.z.get();
    a.b = w.b.get();
    a.e = w.e.get();
    a.ecol = w.ecol.get();
    a.wait = wait;
    a.up_a = s->a.up1.get();
    a.hka = d.hka.get();
    a.ma = s->a.m1;
    a.n = n;
    a.most = d.most;
    a.slots = d.slots;
    a.ksteps = d.slots / 16;
    a.nirrep = nir;
    a.chunk = d.chunk;
    a.nbuf = std::min(4, 512 / (8 * d.slots));
    a.stage_bytes = kYA + d.slots * 256;
    a.stages = std::min<int>(kYStagesMax, (kYSmem - (int)((sizeof(SymShared) + 1023) / 1024 * 1024)) / a.stage_bytes);
    a.os = d.os;
    F2G_CUDA(cudaFuncSetAttribute(k_sy_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, kYSmem));
    for (int v = 0; v < nvec; ++v) {
        const double* x = C + v * N0a * N0b;
        F2G_CUDA(cudaMemsetAsync(w.ec.get() + N0a, 0, sizeof(int), st));
        k_sy_rowexp<<<(unsigned)N0a, 256, 0, st>>>(N0a, N0b, x, w.ec.get());
        F2G_LAUNCH("k_sy_rowexp");
        k_sy_integrals<<<(unsigned)s->a.N1, 256, 0, st>>>(V, n, s->a.m1, s->a.up1.get(), d.os, d.slots, w.ec.get(),
                                                          w.ecol.get(), w.b.get());
        F2G_LAUNCH("k_sy_integrals");
        for (int pos0 = 0; pos0 < d.lmax; pos0 += d.chunk) {
            // the last part may be shorter than the others: positions past lmax do not exist
            const int now = std::min(d.chunk, d.lmax - pos0);
            a.chunk = now;
            a.tiles = now / kYM;
            const int64_t work = N0a * n * (now / 8);
            k_sy_expand<<<(unsigned)std::min<int64_t>(ceil_div(work, 256), (int64_t)sms * 32), 256, 0, st>>>(
                x, N0a, N0b, n, d.lmax, pos0, now, d.hja.get(), d.os, d.tab.get(), w.ec.get(), w.z.get());
            F2G_LAUNCH("k_sy_expand");
            for (int64_t ka0 = 0; ka0 < s->a.N1; ka0 += d.ka) {
                const int64_t ka1 = std::min(ka0 + d.ka, s->a.N1), items = (ka1 - ka0) * nir * a.tiles;
                a.ka0 = ka0;
                k_sy_gemm<<<(unsigned)std::min<int64_t>(items, ctas), kYThreads, kYSmem, st>>>(a, items);
                F2G_LAUNCH("k_sy_gemm");
                k_sy_sum<<<dim3((unsigned)N0a, (unsigned)ceil_div(d.njb, 256)), 256, 0, st>>>(
                    N0b, n, s->na, s->nb, s->a.m1, d.most, ka0, ka1, pos0, now, d.os, s->a.down1.get(), s->a.up1.get(),
                    s->b.down1.get(), d.kpos.get(), d.hja.get(), d.jb.get(), d.njb_of.get(), d.njb, w.e.get(),
                    sig + v * N0a * N0b, wait);
                F2G_LAUNCH("k_sy_sum");
            }
        }
        k_sy_not_finite<<<(unsigned)std::min<int64_t>(N0a, sms), 256, 0, st>>>(
            N0a, N0b, n, s->na, s->nb, s->a.m1, d.os, s->a.down1.get(), s->a.up1.get(), s->b.down1.get(), d.kpos.get(),
            d.hja.get(), d.jb.get(), d.njb_of.get(), d.njb, d.tab.get(), d.lmax, w.ec.get(), x, V, sig + v * N0a * N0b);
        F2G_LAUNCH("k_sy_not_finite");
    }
}

} // namespace f2g
