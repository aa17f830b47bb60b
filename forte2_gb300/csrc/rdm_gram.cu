// Reduced density matrices as Gram matrices on the tensor cores, exact in digits.
//
// Every spin block of the 1-, 2- and 3-RDMs is a sum over hole strings K of one spin of Gram matrices
//   sum_R x(K + o, R + v) x'(K + o', R + v')
// over the other spin's strings R (same-spin blocks: no hole v) or its 1-hole strings (mixed blocks). The slots
// (o, v) of one K, 8 x 14 for the mixed 2-RDM of CAS(14,14), are the rows and columns of the matrix and R is the
// contraction: a GEMM per K whose operands are rows of the vector. 9/14 of the mixed blocks' products have a factor
// of zero (v occupied in R); the tensor cores do them all the same.
//
// Arithmetic. A source row is scaled by its largest exponent to integers of 62 bits and cut into eight signed digits
// of base 256, which are exact FP16 numbers. Products of digits i and j belong to group i + j; the groups 0..7 are
// kept. A group's sum over 128 rows (256 for groups 0..3, which have half the products) is an
// integer below 2^24: exact in the FP32 accumulators. Then it is added into a 64-bit integer in a register, so a
// K's whole sum is exact; it is rounded once per K and added in FP64.
//
// k_rg_expand writes the digits once per vector, 16 bytes per element, K-major. k_rg_gram copies a K's rows from
// there into swizzled core matrices with 16-byte asynchronous copies and no register work. Groups 0..3 need digits
// 0..3 only: they and groups 4..7 are separate work items, so that a tile of 128 x 128 fits the accumulators (4 x 128
// columns) and operands are loaded 1.5 times, not twice as by column halves. Where a tile has at most 64 slots, M = 128 holds
// the slots of q = 128 / nt adjacent digits: digit i's and the next ones' products with a digit of B come from one
// instruction (the accumulator rows then belong to groups one apart).
//
// Bound, for the mixed block of CAS(14,14): the tensor cores (36 digit pairs, 4.0 ms), then the drains and the operands
// (24 GB from L2). At 112 slots the accumulators take 448 of 512 columns: one buffer, whose two halves are drained and
// refilled in turn, so that the MMAs of one overlap with the drain of the other (as one piece 6.64 ms, so 5.75 ms).
// Rows of a digit lie 64 bytes together in shared memory (64-byte swizzle): with unswizzled core matrices, 16 bytes
// together, every 16-byte copy was a wavefront of its own and the copies bound the kernel (7.75 ms, then 6.64). One
// vector, FP64 kernels -> this file: mixed block 56.4 -> 6.5 ms, same spin 8.5 -> 1.7 ms and 1-RDM 1.33 -> 1.08 ms per
// spin; CAS(10,10) mixed 3-RDM block 1,406 -> 142 us, same-spin 3-RDM 146 -> 47 us (whole calls).
//
// Accuracy: a product loses less than 2^-56 of the product of its two source rows' largest elements (2^-62 of each from
// the digits' cut, at most 2^-57.2 from the groups left out).
#include <cuda_fp16.h>

#include <algorithm>

#include "digit_mma.cuh"
#include "rdm.cuh"

namespace f2g {

namespace {

constexpr int kGM = 128;                          // rows of a tile
constexpr int kGProd = 2, kGEpi = 16;             // warps: copies, drains; one more issues the MMAs
constexpr int kGThreads = (kGProd + kGEpi + 1) * 32;
constexpr int kGCols = kGM / 4;                   // columns per drain thread at most
constexpr int kGMaxStages = 8;
constexpr int kGBad = 0x7ff;                      // exponent of a row that holds an infinity or NaN
constexpr int kGSmem = 227 * 1024;

struct GramArgs {
    const uint4 *zl, *zr;   // [row][32 rows R][digit][4 groups of 8 rows R]
    const int *el, *er;
    const void* list;
    double* out;
    WaitCtl wait;
    int64_t d, ko, kv, nK;
    int64_t pstride;        // elements of one partial result
    int parts;              // K goes to partial result K % parts
    uint32_t k8, nsteps;    // groups of 8 rows R per row (a multiple of 4), double K steps of 32 rows
    int m, nv, S, nt, ntile, ntp, q, sym, stages, nbuf, colsbuf, stage_bytes, spt, per_lo, per_hi;
};

struct GramShared {
    alignas(8) uint64_t full[kGMaxStages], empty[kGMaxStages], acc_full[2], acc_empty[2], drain;
    uint32_t tmem_base;
    volatile int abort;
    uint32_t row[kGProd][2][kGM]; // [copy warp][bra, ket][slot]: its digits in zl or zr, in 16 bytes
};

struct GramItem {
    int64_t K;
    int ta, tb, lo;
};
__device__ __forceinline__ GramItem gram_item(const GramArgs& a, int64_t w) {
    GramItem it;
    const int64_t half = a.nK * a.ntp;
    it.lo = w < half; // the longer items first
    if (!it.lo)
        w -= half;
    it.K = w / a.ntp;
    int tp = (int)(w - it.K * a.ntp);
    it.ta = 0;
    if (a.sym) {
        while (tp >= a.ntile - it.ta) {
            tp -= a.ntile - it.ta;
            ++it.ta;
        }
        it.tb = it.ta + tp;
    } else {
        it.ta = tp / a.ntile;
        it.tb = tp % a.ntile;
    }
    return it;
}

// slot s of K: source row, hole v, output offset, sign
template <int LIST>
__device__ __forceinline__ void gram_slot(const GramArgs& a, int64_t K, int s, int64_t& I, int& v, int& off, int& neg) {
    const int e = s / a.nv;
    int o;
    v = s - e * a.nv;
    hole_entry<LIST>(a.list, K * a.m + e, I, o, neg);
    off = (int)(o * a.ko + v * a.kv);
}

template <int LIST>
__global__ void __launch_bounds__(kGThreads, 1) k_rg_gram(const __grid_constant__ GramArgs a, int64_t nitems) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    GramShared& sh = *reinterpret_cast<GramShared*>(smem_raw);
    const uint32_t ring = smem_u32(smem_raw) + ((sizeof(GramShared) + 1023) / 1024) * 1024;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const volatile int* abort = &sh.abort;
    if (tid == 0) {
        for (int i = 0; i < kGMaxStages; ++i) {
            mbar_init(smem_u32(&sh.full[i]), kGProd * 32);
            mbar_init(smem_u32(&sh.empty[i]), 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(smem_u32(&sh.acc_full[i]), 1);
            mbar_init(smem_u32(&sh.acc_empty[i]), kGEpi);
        }
        mbar_init(smem_u32(&sh.drain), 1);
        sh.abort = 0;
    }
    if (warp == kGProd + kGEpi) {
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
    const uint32_t a_bytes = (uint32_t)a.nt * 512; // a double K step of eight digits (32 rows R) of a tile

    if (warp < kGProd) {
        // ---- copies: spt double K steps per stage. Four lanes take a row's 64 bytes of a digit, eight rows to an
        // instruction (16-byte pieces that land apart take a wavefront each: 16 bytes per clock); the warps take every
        // other digit. What is left of a tile past its last slot keeps any value: those rows and columns are not used
        uint32_t slot = 0, phase = 1; // of the stage's `empty`: the first round finds every stage free
        bool ok = true;
        const uint32_t row_pitch = a.k8 * 8;
        for (int64_t w = blockIdx.x; ok && w < nitems; w += gridDim.x) {
            const GramItem it = gram_item(a, w);
            const bool two = !(a.sym && it.ta == it.tb);
            __syncwarp();
            for (int side = 0; side < (two ? 2 : 1); ++side)
                for (int t = lane; t < a.nt; t += 32) {
                    int64_t I;
                    int v, off, neg;
                    gram_slot<LIST>(a, it.K, min((side ? it.tb : it.ta) * a.nt + t, a.S - 1), I, v, off, neg);
                    sh.row[warp][side][t] = (uint32_t)(I * a.nv + v) * row_pitch;
                }
            __syncwarp();
            const int nd = it.lo ? 8 : 4, row = lane >> 2, piece = lane & 3;
            const uint32_t side_bytes = it.lo ? a_bytes : a_bytes / 2, step_bytes = two ? 2 * side_bytes : side_bytes;
            const uint32_t dst0 = (uint32_t)row * 64 + ((piece ^ (row >> 1)) & 3) * 16;
            const uint32_t spt = it.lo ? a.spt : 2 * a.spt, digit_bytes = (uint32_t)a.nt * 64;
            for (uint32_t ks = 0; ks < a.nsteps;) {
                if (!mbar_wait_warp(smem_u32(&sh.empty[slot]), phase, abort)) {
                    give_up();
                    ok = false;
                    break;
                }
                const uint32_t k0 = ks, ke = min(ks + spt, a.nsteps), dst = ring + slot * a.stage_bytes + dst0;
                ks = ke;
                for (int side = 0; side < (two ? 2 : 1); ++side) {
                    const int ng = (min(a.nt, a.S - (side ? it.tb : it.ta) * a.nt) + 7) >> 3;
                    uint32_t r[kGM / 8];
#pragma unroll
                    for (int g = 0; g < kGM / 8; ++g)
                        r[g] = sh.row[warp][side][g * 8 + row];
                    const uint4* z = (side ? a.zr : a.zl) + k0 * 32 + piece;
                    uint32_t to = dst + side * side_bytes;
                    for (uint32_t k = k0; k < ke; ++k, z += 32, to += step_bytes)
                        for (int d = warp; d < nd; d += kGProd)
#pragma unroll
                            for (int g = 0; g < kGM / 8; ++g) {
                                if (g >= ng)
                                    break;
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + d * digit_bytes + g * 512),
                                             "l"(z + d * 4 + r[g]));
                            }
                }
                // this thread's arrival, once its copies have landed
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&sh.full[slot]))
                             : "memory");
                if (++slot == (uint32_t)a.stages) {
                    slot = 0;
                    phase ^= 1;
                }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < kGProd + kGEpi) {
        // ---- drains: groups into 64-bit integers in registers, at the end of the item into the output
        const int ew = warp - kGProd, quarter = warp & 3, part = ew >> 2;
        const int row = quarter * 32 + lane;
        const int w4 = (a.nt / 4 + 3) / 4;             // blocks of four columns per warp
        const int c0 = part * w4 * 4, nb = max(0, min(w4, a.nt / 4 - part * w4));
        const int di = row / a.nt, rs = row - di * a.nt;
        uint32_t buf = 0, phase = 0;
        bool ok = true;
        for (int64_t w = blockIdx.x; ok && w < nitems; w += gridDim.x) {
            const GramItem it = gram_item(a, w);
            const int base = it.lo ? 4 : 0, cl = it.lo ? max(0, 5 - a.q) : 0, nc = it.lo ? 8 - cl : 4;
            const uint32_t per = it.lo ? a.per_lo : a.per_hi;
            long long T[kGCols];
#pragma unroll
            for (int j = 0; j < kGCols; ++j)
                T[j] = 0;
            for (uint32_t k = 0; ok && k < a.nsteps; k += per) {
                // one buffer: the first half of its column blocks and the second are handed over by themselves
                for (int half = 0; half < (a.nbuf == 1 ? 2 : 1); ++half) {
                    const uint32_t bar = a.nbuf == 1 ? half : buf;
                    if (!mbar_wait_warp(smem_u32(&sh.acc_full[bar]), phase, abort)) {
                        give_up();
                        ok = false;
                        break;
                    }
                    fence_after();
                    const uint32_t at = tmem + ((uint32_t)(quarter * 32) << 16) + (a.nbuf == 1 ? 0 : buf * a.colsbuf) + c0;
                    const int lo = half ? nc / 2 : 0, hi = a.nbuf == 1 && !half ? nc / 2 : nc;
                    for (int cc = lo; cc < hi; cc += 2) {
                        int mul[2];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int g = cl + cc + u + di - base; // this row's group in column block cc + u
                            mul[u] = cc + u < hi && g >= 0 && g < 4 ? 1 << (8 * (3 - g)) : 0;
                        }
#pragma unroll
                        for (int b = 0; b < kGCols / 4; ++b)
                            if (b < nb) {
                                uint32_t r[8];
#pragma unroll
                                for (int u = 0; u < 2; ++u)
                                    tmem_ld4(at + min(cc + u, hi - 1) * a.nt + b * 4, r + 4 * u);
                                tmem_wait_ld();
#pragma unroll
                                for (int u = 0; u < 2; ++u)
#pragma unroll
                                    for (int j = 0; j < 4; ++j)
                                        T[b * 4 + j] = mad_wide(__float2int_rn(__uint_as_float(r[4 * u + j])), mul[u],
                                                                T[b * 4 + j]);
                            }
                    }
                    fence_before();
                    __syncwarp();
                    if (lane == 0)
                        mbar_arrive(smem_u32(&sh.acc_empty[bar]));
                }
                if (a.nbuf == 1 || (buf ^= 1) == 0)
                    phase ^= 1;
            }
            // lane j: offset in the output, exponent and sign of column c0 + j
            int coff = -1, ce = 0, cneg = 0;
            if (c0 + lane < a.nt && it.tb * a.nt + c0 + lane < a.S) {
                int64_t I;
                int v;
                gram_slot<LIST>(a, it.K, it.tb * a.nt + c0 + lane, I, v, coff, cneg);
                ce = max(a.er[I], 1);
            }
            const int s = it.ta * a.nt + rs;
            double* out = a.out + (it.K % a.parts) * a.pstride;
            const bool mine = ok && di < a.q && s < a.S, mirror = a.sym && it.ta != it.tb;
            int64_t I;
            int v, off = 0, neg = 0, ea = 1;
            if (mine) {
                gram_slot<LIST>(a, it.K, s, I, v, off, neg);
                ea = max(a.el[I], 1);
            }
            const bool abad = ea >= kGBad;
            ea += it.lo ? 56 - 68 : 88 - 68; // units of T: 2^(56 or 88) 2^(ea - 1084) 2^(eb - 1084)
#pragma unroll
            for (int j = 0; j < kGCols; ++j)
                if (j < nb * 4) {
                    const int o = __shfl_sync(0xffffffffu, coff, j), eb = __shfl_sync(0xffffffffu, ce, j),
                              nn = __shfl_sync(0xffffffffu, cneg, j) ^ neg;
                    const bool bad = eb >= kGBad || abad;
                    if (!mine || o < 0 || (T[j] == 0 && !bad))
                        continue;
                    double x = bad ? __longlong_as_double(0x7ff8000000000000ll) : oz_value(T[j], ea + eb);
                    if (nn)
                        x = -x;
                    atomicAdd(out + (int64_t)off * a.d + o, x);
                    if (mirror)
                        atomicAdd(out + (int64_t)o * a.d + off, x);
                }
        }
    } else {
        // ---- MMAs
        const uint32_t el = elect_lane();
        const uint32_t nt = (uint32_t)a.nt;
        uint32_t slot = 0, phase = 0, buf = 0, buf_phase = 1;
        bool ok = a.wait.polls == 0; // with a limit on the tries (for tests) the first wait counts as given up
        for (int64_t w = blockIdx.x; ok && w < nitems; w += gridDim.x) {
            const GramItem it = gram_item(a, w);
            const bool two = !(a.sym && it.ta == it.tb);
            const int cm = it.lo ? 7 : 3, cl = it.lo ? max(0, 5 - a.q) : 0;
            const uint32_t spt = it.lo ? a.spt : 2 * a.spt, per = it.lo ? a.per_lo : a.per_hi;
            const uint32_t side16 = (it.lo ? 8 : 4) * nt * 4, step16 = two ? 2 * side16 : side16; // descriptors count 16 bytes
            const int split = cl + (cm - cl + 1) / 2; // one buffer: column blocks before it are the first half
            for (uint32_t k = 0; ok && k < a.nsteps;) {
                if (!mbar_wait_warp(smem_u32(&sh.acc_empty[a.nbuf == 1 ? 0 : buf]), buf_phase, abort)) {
                    ok = false;
                    break;
                }
                const uint32_t acc = tmem + (a.nbuf == 1 ? 0 : buf * a.colsbuf), k0 = k, kend = min(k + per, a.nsteps);
                while (k < kend) {
                    if (!mbar_wait_warp(smem_u32(&sh.full[slot]), phase, abort)) {
                        ok = false;
                        break;
                    }
                    // the copies were made by the generic proxy. This warp fences, not the copying ones: there the
                    // fence waits for all copies in flight (1,100 clocks per K step)
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    fence_after();
                    const uint64_t ad0 = smem_desc_64b(ring + slot * a.stage_bytes, 512);
                    const uint32_t ks = k, ke = min(k + spt, kend);
                    // column blocks c0 <= c < c1 of the stage's double K steps
                    auto issue = [&](int c0, int c1) {
                        uint64_t ad = ad0;
                        uint32_t add = ks > k0;
                        for (uint32_t s = ks; s < ke; ++s, ad += step16)
                            for (int h = 0; h < 2; ++h) { // 16 of the 32 rows R: 32 bytes on in every row of 64
                                const uint64_t bd = ad + (two ? side16 : 0) + 2 * h;
                                for (int i = 0; i < c1; i += a.q) {
                                    const int c = max(i, c0); // digit i reaches column block i and those after it
                                    uint32_t n = (uint32_t)(c1 - c) * nt, dcol = acc + (uint32_t)(c - cl) * nt;
                                    uint64_t b = bd + (c - i) * nt * 4;
                                    const uint64_t ai = ad + 2 * h + i * nt * 4;
                                    if (n > 256) {
                                        mma_ss(dcol, ai, b, 256, add, el);
                                        n -= 256, dcol += 256, b += 1024;
                                    }
                                    mma_ss(dcol, ai, b, n, add, el);
                                    add = 1;
                                }
                            }
                    };
                    if (a.nbuf == 1) {
                        issue(cl, split);
                        if (ke == kend)
                            mma_commit(smem_u32(&sh.acc_full[0]), el);
                        if (ks == k0 && !mbar_wait_warp(smem_u32(&sh.acc_empty[1]), buf_phase, abort)) {
                            ok = false;
                            break;
                        }
                        fence_after();
                        issue(split, cm + 1);
                    } else {
                        issue(cl, cm + 1);
                    }
                    k = ke;
                    mma_commit(smem_u32(&sh.empty[slot]), el);
                    if (++slot == (uint32_t)a.stages) {
                        slot = 0;
                        phase ^= 1;
                    }
                }
                if (ok)
                    mma_commit(smem_u32(&sh.acc_full[a.nbuf == 1 ? 1 : buf]), el);
                if (a.nbuf == 1 || (buf ^= 1) == 0)
                    buf_phase ^= 1;
            }
        }
        if (!ok)
            give_up();
        // the instructions in flight end before the block leaves
        mma_commit(smem_u32(&sh.drain), el);
        mbar_wait_warp(smem_u32(&sh.drain), 0, nullptr);
    }
    __syncwarp();
    __syncthreads();
    if (warp == kGProd + kGEpi) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---- operands --------------------------------------------------------------------------------------

// largest biased exponent of every source row (element (r, k) at C[r sr + k sk]), by atomic maximum
__global__ void __launch_bounds__(256) k_rg_rowexp(const double* __restrict__ C, int64_t sr, int64_t sk, int64_t nrow,
                                                   int64_t ncol, int* __restrict__ e) {
    uint32_t mx = 0;
    const uint32_t* hi = reinterpret_cast<const uint32_t*>(C) + 1;
    if (sk == 1) { // a block per row
        for (int64_t r = blockIdx.x; r < nrow; r += gridDim.x) {
            mx = 0;
            for (int64_t k = threadIdx.x; k < ncol; k += blockDim.x)
                mx = max(mx, hi[2 * (r * sr + k)] & 0x7fffffffu);
            mx = __reduce_max_sync(0xffffffffu, mx);
            if ((threadIdx.x & 31) == 0 && mx)
                atomicMax(e + r, (int)(mx >> 20));
        }
    } else { // a thread per row and 64 columns
        const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, k0 = blockIdx.y * (int64_t)64;
        if (r >= nrow)
            return;
#pragma unroll 8
        for (int64_t k = k0; k < min(k0 + 64, ncol); ++k)
            mx = max(mx, hi[2 * (r * sr + k * sk)] & 0x7fffffffu);
        if (mx)
            atomicMax(e + r, (int)(mx >> 20));
    }
}

// tab[v][K] = address | negative << 31 of K + v, ~0 where v is occupied in K
__global__ void k_rg_tab(const uint32_t* __restrict__ up1, int m, int64_t nK, uint32_t* __restrict__ tab) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= nK * m)
        return;
    const uint32_t e = up1[t];
    tab[e_orb(e) * nK + t / m] = e_addr(e) | (uint32_t)e_neg(e) << 31;
}

// digits of rows (I, v) (element (I, R + v) of the source, v = 0 without a table) for the rows R k0 .. k0 + 8 k8 of
// nR: a thread makes 8 neighbours in R (128 bytes, written through shared memory in whole lines). Lanes run along R
// where the source is contiguous there, else along I.
__global__ void __launch_bounds__(256) k_rg_expand(const double* __restrict__ C, int64_t sr, int64_t sk, int64_t nI, int nv,
                                                   const uint32_t* __restrict__ tab, int64_t nR, int64_t k0, uint32_t k8,
                                                   const int* __restrict__ e, uint4* __restrict__ z) {
    __shared__ uint4 sm[8][256];
    const int lane = threadIdx.x & 31;
    uint4* my = sm[threadIdx.x >> 5];
    const int64_t total = nI * nv * k8, stride = (int64_t)gridDim.x * 256;
    for (int64_t t0 = blockIdx.x * (int64_t)256 + (threadIdx.x & ~31); t0 < total; t0 += stride) {
        const int64_t t = min(t0 + lane, total - 1); // the last warp repeats the last thread's work
        int64_t I, zi;
        int v;
        uint32_t g;
        if (sk == 1) {
            zi = t;
            g = (uint32_t)(t % k8);
            const int64_t r = t / k8;
            I = r / nv;
            v = (int)(r - I * nv);
        } else {
            I = t % nI;
            const int64_t r = t / nI;
            v = (int)(r % nv);
            g = (uint32_t)(r / nv);
            zi = (I * nv + v) * k8 + g;
        }
        const int E = max(e[I], 1);
        uint64_t y[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const int64_t k = k0 + (int64_t)g * 8 + j;
            uint32_t a = ~0u;
            if (k < nR)
                a = tab ? __ldg(tab + v * nR + k) : (uint32_t)k;
            y[j] = gram_digits(a == ~0u ? 0.0 : __ldg(C + I * sr + (int64_t)(a & 0x7fffffffu) * sk), a >> 31, E);
        }
        auto put = [&](int d, uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3) {
            my[lane * 8 + (d ^ (lane & 7))] = make_uint4(x0, x1, x2, x3);
        };
#define F2G_DIGIT(D)                                                                                               \
    put(D, gram_half2<D>(y[0], y[1]), gram_half2<D>(y[2], y[3]), gram_half2<D>(y[4], y[5]), gram_half2<D>(y[6], y[7]))
        F2G_DIGIT(0);
        F2G_DIGIT(1);
        F2G_DIGIT(2);
        F2G_DIGIT(3);
        F2G_DIGIT(4);
        F2G_DIGIT(5);
        F2G_DIGIT(6);
        F2G_DIGIT(7);
#undef F2G_DIGIT
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int o = i * 4 + (lane & 3), d = lane >> 2; // 512 bytes in the order of the lanes
            const int64_t at = __shfl_sync(0xffffffffu, zi, o);
            // [32 rows R][digit][group of 8]
            if (t0 + o < total)
                z[(at >> 2) * 32 + d * 4 + (at & 3)] = my[o * 8 + (d ^ (o & 7))];
        }
        __syncwarp();
    }
}

// out += the partial results, added as a tree over eight of them at a time; NaN once a wait has given up
__global__ void k_rg_reduce(int64_t size, int parts, const double* __restrict__ part, double* __restrict__ out,
                            const WaitCtl wait) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < size; i += (int64_t)gridDim.x * blockDim.x) {
        double sum = 0.0;
        for (int p = 0; p < parts; p += 8) {
            double x[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                x[j] = p + j < parts ? part[(p + j) * size + i] : 0.0;
            sum += ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));
        }
        out[i] += waited(sum, wait);
    }
}

// bra or ket: row exponents
void gram_exponents(const double* C, int64_t sr, int64_t sk, int64_t nI, int64_t ncol, DevBuf<int>& e, cudaStream_t st) {
    e.reserve((size_t)nI);
    F2G_CUDA(cudaMemsetAsync(e.get(), 0, (size_t)nI * sizeof(int), st));
    if (sk == 1)
        k_rg_rowexp<<<(unsigned)std::min<int64_t>(nI, 4096), 256, 0, st>>>(C, sr, sk, nI, ncol, e.get());
    else
        k_rg_rowexp<<<dim3((unsigned)((nI + 255) / 256), (unsigned)((ncol + 63) / 64)), 256, 0, st>>>(C, sr, sk, nI, ncol,
                                                                                                    e.get());
    F2G_LAUNCH("k_rg_rowexp");
}

template <int LIST> void gram_launch(const GramArgs& a, int64_t items, int sms, cudaStream_t st) {
    F2G_CUDA(cudaFuncSetAttribute(k_rg_gram<LIST>, cudaFuncAttributeMaxDynamicSharedMemorySize, kGSmem));
    k_rg_gram<LIST><<<(unsigned)std::min<int64_t>(items, sms), kGThreads, kGSmem, st>>>(a, items);
    F2G_LAUNCH("k_rg_gram");
}

} // namespace

// Is this kernel the faster one? Times of a call from Python on the device's vectors, FP64 kernel and this one.
static bool gram_pays(const CIStrings& s, int spin, int holes, bool inner, bool sym, int m, int64_t nR) {
    // Same-spin blocks of two and three holes where a K is worth a tile: from m^2 nR = 1.2e5 (1.1e5: 30 and 37 us; 2.0e5:
    // 73 and 23 us; 3.9e5: 74 and 24 us). One hole, where a K has few slots: from 2,048 rows R (924 rows: 113 and 181 us)
    // and for one vector from 8 slots (7: 989 and 1,059 us at (14, 8, 6); 8: 1,327 and 1,073 us at (14, 7, 7); 13: 2,067
    // and 1,006 us at (16, 4, 8)), for two, whose digits are written twice, from 12 (8: 1,333 and 2,071 us; 11: 1,060 and
    // 1,082 us at (15, 5, 5); 12: 6,896 and 5,725 us at (16, 5, 8)).
    if (!inner)
        return holes == 1 ? nR >= 2048 && m >= (sym ? 8 : 12) : (double)m * m * (double)nR >= 1.2e5;
    // Mixed blocks: the FP64 kernel takes a launch and, for every pair of alpha hole sets, a pass over the beta spin's
    // pairs per alpha hole string, this one seven launches (ten for two vectors): FP64 where those passes are few. One
    // hole each: 6 of them 36 and 37 us (one vector, (5, 3, 3)), 7 40 and 38 us, 10 59 and 37 us (6, 4, 3); two vectors
    // 8 45 and 46 us (9, 8, 7), 9 50 and 45 us, 20 79 and 46 us (7, 4, 3). Two alpha holes, where there are more pairs:
    // 4 32 and 36 us (6, 3, 3), 5 60 and 42 us (7, 3, 2); two vectors 6 43 and 49 us (8, 7, 4), 53 and 47 us (6, 4, 2). Two
    // beta holes, longer passes: 4 32 and 37 us (5, 4, 2), 5 42 and 38 us (6, 5, 4); two vectors 5 38 and 50 us, 6 60 and
    // 52 us (7, 6, 5). A single pass is the whole FP64 kernel, and a single hole string here few blocks' work: (16, 1, 12)
    // 51 and 396 us, (13, 13, 6) 43 and 49 us.
    const bool aab = spin == 0 && holes == 2, abb = spin == 1;
    const int ha = aab ? 2 : 1, hb = abb ? 2 : 1, n = s.norb;
    const double passes = (double)host_binom(n - ha, s.na - ha);
    const double ma = (double)host_binom(n - s.na + ha, ha), alpha = host_binom(n, s.na - ha) * ma * ma;
    const double mb = (double)host_binom(n - s.nb + hb, hb), beta = host_binom(n, s.nb - hb) * mb * mb;
    const int few = aab ? (sym || alpha > 520 ? 4 : 6) : abb ? (sym ? 4 : 5) : sym ? 6 : 8;
    return !(passes <= few && alpha <= 800 && passes * beta <= (passes == 1 ? 131072 : 16384));
}

bool rdm_gram(SigmaBuilder& sb, GramScratch& g, int spin, int holes, bool inner, const double* CL, const double* CR,
              int64_t d, int64_t ko, int64_t kv, double* out, cudaStream_t st) {
    if (!sb.use_oz)
        return false;
    const CIStrings& s = *sb.s;
    SpinStrings& so = sb.s->spin(spin);
    SpinStrings& si = sb.s->spin(1 - spin);
    if (so.k < holes || (inner && si.k < 1))
        return true; // nothing to add
    const int64_t nK = holes == 1 ? so.N1 : holes == 2 ? so.N2 : so.N3;
    const int m = holes == 1 ? so.m1 : holes == 2 ? so.m2 : so.m3;
    const int64_t nI = so.N0, nR = inner ? si.N1 : si.N0;
    const int nv = inner ? s.norb : 1;
    if (nK == 0 || m == 0 || nR == 0)
        return true;
    if (!sb.digits_always && !gram_pays(s, spin, holes, inner, CL == CR, m, nR))
        return false;
    // rows R at a time: digits of a vector within the limit, whole drains of 128
    const int64_t rows = nI * nv, all8 = (nR + 31) / 32 * 4;
    int64_t k8 = all8;
    if (rows * 128 * std::min<int64_t>(all8, 16) > int64_t(1) << 31)
        return false;
    if (rows * 128 * all8 > sb.digit_limit()) {
        const int64_t most = std::max<int64_t>(1, sb.digit_limit() / (rows * 128 * 16)) * 16;
        const int64_t parts = (all8 + most - 1) / most;
        k8 = std::min(most, ((all8 + parts - 1) / parts + 15) / 16 * 16);
    }
    if (rows >= int64_t(0xffffffff))
        return false;
    int sms = 0, dev = 0;
    F2G_CUDA(cudaGetDevice(&dev));
    F2G_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const bool sym = CL == CR;
    const int64_t NB = s.b.N0;
    const int64_t sr = spin == 0 ? NB : 1, sk = spin == 0 ? 1 : NB;

    GramArgs a{};
    if (holes == 2)
        so.build_up2(sb.s->binom.get(), st);
    if (holes == 3)
        so.build_up3(sb.s->binom.get(), st);
    a.list = holes == 1 ? (const void*)so.up1.get() : holes == 2 ? (const void*)so.up2.get() : (const void*)so.up3.get();
    const uint32_t* tab = nullptr;
    if (inner) {
        DevBuf<uint32_t>& t = g.tab[1 - spin];
        if (!t.get()) {
            t.reserve((size_t)(nR * nv));
            F2G_CUDA(cudaMemsetAsync(t.get(), 0xff, (size_t)(nR * nv) * sizeof(uint32_t), st));
            k_rg_tab<<<(unsigned)((nR * si.m1 + 255) / 256), 256, 0, st>>>(si.up1.get(), si.m1, nR, t.get());
            F2G_LAUNCH("k_rg_tab");
        }
        tab = t.get();
    }
    gram_exponents(CL, sr, sk, nI, s.spin(1 - spin).N0, g.el, st);
    if (!sym)
        gram_exponents(CR, sr, sk, nI, s.spin(1 - spin).N0, g.er, st);
    a.el = g.el.get();
    a.er = sym ? a.el : g.er.get();
    // many K added one after the other to an element would cost it digits (3,003 K: 3.1e-15 of the largest element
    // against 1.0e-15 of the FP64 kernel; 56 K: 9e-16 against 2e-16): partial results of few K each, added as a tree
    const int64_t size = d * d;
    const bool many = nK >= 768;
    a.parts = (int)std::min<int64_t>({nK, many ? 128 : 16, std::max<int64_t>(4, (int64_t(1) << (many ? 25 : 20)) / size)});
    a.pstride = size;
    a.out = g.part.reserve((size_t)(a.parts * size));
    F2G_CUDA(cudaMemsetAsync(a.out, 0, (size_t)(a.parts * size) * sizeof(double), st));
    a.wait = sb.wait_ctl();
    a.d = d;
    a.ko = ko;
    a.kv = kv;
    a.nK = nK;
    a.m = m;
    a.nv = nv;
    a.S = m * nv;
    // slots per tile: 128 with one operand, 112 with two (two stages of 2 x 112 x 512 bytes just fit)
    a.ntile = sym && a.S <= kGM ? 1 : (a.S + 111) / 112;
    a.nt = ((a.S + a.ntile - 1) / a.ntile + 15) / 16 * 16;
    a.ntile = (a.S + a.nt - 1) / a.nt;
    a.sym = sym;
    a.ntp = sym ? a.ntile * (a.ntile + 1) / 2 : a.ntile * a.ntile;
    a.q = std::min(8, kGM / a.nt);
    a.colsbuf = std::max(4, 8 - std::max(0, 5 - a.q)) * a.nt;
    // double K steps per drain: 2^24 / 2^14 products of digits, the i q-th digits of A's side in every accumulator
    // (digit 0 is at most 64, so that q = 1 has 7 times and 3 times 2^14 per row)
    a.per_lo = a.q == 1 ? 4 : 32 / ((8 + a.q - 1) / a.q);
    a.per_hi = a.q == 1 ? 8 : 32 / ((4 + a.q - 1) / a.q);
    a.nbuf = 2 * a.colsbuf <= 512 ? 2 : 1;
    a.stage_bytes = a.nt * 512 * (sym && a.ntile == 1 ? 1 : 2);
    const int ring = kGSmem - (int)((sizeof(GramShared) + 1023) / 1024 * 1024) -
                     (sym && a.ntile == 1 ? 8192 : 0); // a tile's last digits are read as 128 rows of 64 bytes; behind the
                                                       // first of two operands lies the second
    static_assert(kGSmem - (sizeof(GramShared) + 1023) / 1024 * 1024 >= 2 * 2 * 112 * 512);
    // stages as large as leave two (seven of one K step: same spin 1.99 against 1.73 ms without drains); spt double
    // K steps of 8 digits (twice that of 4), a divisor of per_lo
    a.spt = a.per_lo;
    while (a.spt > 1 && 2 * a.spt * a.stage_bytes > ring)
        a.spt /= 2;
    a.stage_bytes *= a.spt;
    a.stages = std::min(kGMaxStages, ring / a.stage_bytes);
    const int64_t items = a.nK * a.ntp * 2;
    for (int64_t at = 0; at < all8; at += k8) {
        const int64_t now = std::min(k8, all8 - at);
        a.k8 = (uint32_t)now;
        a.nsteps = (uint32_t)(now / 4);
        const int64_t work = rows * now;
        const unsigned grid = (unsigned)std::min<int64_t>((work + 255) / 256, (int64_t)sms * 32);
        g.zl.reserve((size_t)(rows * k8 * 8));
        k_rg_expand<<<grid, 256, 0, st>>>(CL, sr, sk, nI, nv, tab, nR, at * 8, (uint32_t)now, a.el, g.zl.get());
        F2G_LAUNCH("k_rg_expand");
        if (!sym) {
            g.zr.reserve((size_t)(rows * k8 * 8));
            k_rg_expand<<<grid, 256, 0, st>>>(CR, sr, sk, nI, nv, tab, nR, at * 8, (uint32_t)now, a.er, g.zr.get());
            F2G_LAUNCH("k_rg_expand");
        }
        a.zl = g.zl.get();
        a.zr = sym ? a.zl : g.zr.get();
        if (holes == 1)
            gram_launch<1>(a, items, sms, st);
        else if (holes == 2)
            gram_launch<2>(a, items, sms, st);
        else
            gram_launch<3>(a, items, sms, st);
    }
    k_rg_reduce<<<(unsigned)std::min<int64_t>((size + 255) / 256, 4096), 256, 0, st>>>(size, a.parts, a.out, out,
                                                                                       a.wait);
    F2G_LAUNCH("k_rg_reduce");
    return true;
}

} // namespace f2g
