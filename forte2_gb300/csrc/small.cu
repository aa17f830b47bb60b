// FP64 sigma of a small C1 space in one launch.
//
// A small space is bound by launches and latency: the separate kernels (two transposes, two same-spin
// products, opposite spin) took 33 us of device time for the 400 determinants of (6e,6o), 84 us for the
// 4,900 of (8e,8o). Here a block keeps the whole vector and the opposite-spin integrals in shared memory
// and four lanes form one sigma element: the same-spin string-Hamiltonian rows of its alpha and its beta
// string and all products of an alpha with a beta excitation,
//   sigma(Ja, Jb) = sum_k Haa(Ja, I_k) C(I_k, Jb) + sum_k Hbb(Jb, I_k) C(Ja, I_k)
//                   + sum_{a = (p,q), b = (r,s)} sgn_a sgn_b V[p][r][q][s] C(Ia, Ib),
// every lane every fourth entry of the lists, added in lane order: bitwise the same for every batch.
// Bound: the FP64 pipe (4,900 x 506 multiply-adds: 4 us of the chip's) and the loads of the vector per block.
#include "sigma.cuh"

namespace f2g {

namespace {

constexpr int kSmallBlock = 128, kSmallLanes = 4;
constexpr int64_t kSmallSmem = 200 * 1024;

// excitations of every string J: entry = address of I (14 bits) | (p * n + q) << 14 | negative << 31 for
// J <- I = J - p + q, p ascending, then q in list order
__global__ void k_small_exc(int64_t N0, int n, int k, int m1, const uint32_t* __restrict__ down,
                            const uint32_t* __restrict__ up, uint32_t* __restrict__ exc) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, J = t / (k * m1);
    if (J >= N0)
        return;
    const int i = (int)(t % (k * m1));
    const uint32_t ep = down[J * k + i / m1], eq = up[(int64_t)e_addr(ep) * m1 + i % m1];
    exc[t] = e_addr(eq) | (uint32_t)(e_orb(ep) * n + e_orb(eq)) << 14 | ((ep ^ eq) & 0x80000000u);
}

__device__ __forceinline__ double sgn(double x, uint32_t e) { // x with its sign flipped by the top bit of e
    return __longlong_as_double(__double_as_longlong(x) ^ ((long long)(e & 0x80000000u) << 32));
}

__global__ void __launch_bounds__(kSmallBlock)
    k_small_sigma(int nd, int N0b, int n, int nnza, const int32_t* __restrict__ cola, const double* __restrict__ vala,
                  int nnzb, const int32_t* __restrict__ colb, const double* __restrict__ valb, int nea,
                  const uint32_t* __restrict__ exa, int neb, const uint32_t* __restrict__ exb,
                  const double* __restrict__ V, const double* __restrict__ C, double* __restrict__ S) {
    extern __shared__ double sm[];
    double* c = sm;       // the vector
    double* w = sm + nd;  // w[(p q)][(r s)] = V[p][r][q][s]
    C += blockIdx.y * (int64_t)nd;
    S += blockIdx.y * (int64_t)nd;
    for (int i = threadIdx.x; i < nd; i += kSmallBlock)
        c[i] = C[i];
    const int n2 = n * n;
    for (int i = threadIdx.x; i < n2 * n2; i += kSmallBlock) {
        const int q = i / n % n, s = i % n, r = i / n2 % n, p = i / (n2 * n); // i = ((p n + r) n + q) n + s
        w[(p * n + q) * n2 + r * n + s] = V[i];
    }
    __syncthreads();
    const int lane = threadIdx.x & (kSmallLanes - 1);
    const int J = (blockIdx.x * kSmallBlock + threadIdx.x) / kSmallLanes;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    if (J < nd) {
        const int Ja = J / N0b, Jb = J - Ja * N0b;
        const int32_t* ca = cola + (int64_t)Ja * nnza;
        const double* va = vala + (int64_t)Ja * nnza;
#pragma unroll 4
        for (int k = lane; k < nnza; k += kSmallLanes)
            acc[0] += va[k] * c[ca[k] * N0b + Jb];
        const int32_t* cb = colb + (int64_t)Jb * nnzb;
        const double* vb = valb + (int64_t)Jb * nnzb;
#pragma unroll 4
        for (int k = lane; k < nnzb; k += kSmallLanes)
            acc[1] += vb[k] * c[Ja * N0b + cb[k]];
        for (int a = lane; a < nea; a += kSmallLanes) {
            const uint32_t ea = exa[Ja * nea + a];
            const double* row = c + (ea & 0x3fffu) * N0b;
            const double* wr = w + ((ea >> 14) & 0xffffu) * n2;
            double x[4] = {0.0, 0.0, 0.0, 0.0};
            int b = 0;
            for (; b + 4 <= neb; b += 4)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t eb = __ldg(exb + Jb * neb + b + i);
                    x[i] += sgn(wr[(eb >> 14) & 0xffffu], eb) * row[eb & 0x3fffu];
                }
            for (; b < neb; ++b) {
                const uint32_t eb = __ldg(exb + Jb * neb + b);
                x[0] += sgn(wr[(eb >> 14) & 0xffffu], eb) * row[eb & 0x3fffu];
            }
            acc[2] += sgn((x[0] + x[1]) + (x[2] + x[3]), ea);
        }
    }
    double s = (acc[0] + acc[1]) + acc[2];
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    if (J < nd && lane == 0)
        S[J] = s;
}

} // namespace

// The space's vector and integrals fit a block's shared memory (and the addresses the packed lists)
bool small_supported(const CIStrings* s) {
    const int64_t n4 = (int64_t)s->norb * s->norb * s->norb * s->norb;
    return s->norb <= 16 && s->na >= 1 && s->nb >= 1 && s->a.N0 < (1 << 14) && s->b.N0 < (1 << 14) && s->nfull > 0 &&
           (s->nfull + n4) * 8 <= kSmallSmem;
}

void small_lists(const CIStrings* s, DevBuf<uint32_t> (&exc)[2], cudaStream_t st) {
    for (int sp = 0; sp < 2; ++sp) {
        const SpinStrings& ss = s->spin(sp);
        const int64_t ne = ss.N0 * ss.k * ss.m1;
        exc[sp].reserve((size_t)ne);
        k_small_exc<<<ceil_div(ne, 256), 256, 0, st>>>(ss.N0, s->norb, ss.k, ss.m1, ss.down1.get(), ss.up1.get(),
                                                       exc[sp].get());
        F2G_LAUNCH("k_small_exc");
    }
}

void launch_small_sigma(const CIStrings* s, const StringHamiltonian& ha, const StringHamiltonian& hb,
                        const DevBuf<uint32_t> (&exc)[2], const double* V, const double* C, double* sig, int nvec,
                        cudaStream_t st) {
    const int n = s->norb, nd = (int)s->nfull;
    const size_t smem = ((size_t)nd + (size_t)n * n * n * n) * sizeof(double);
    F2G_CUDA(cudaFuncSetAttribute(k_small_sigma, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_small_sigma<<<dim3((unsigned)ceil_div((int64_t)nd * kSmallLanes, kSmallBlock), (unsigned)nvec), kSmallBlock, smem,
                    st>>>(nd, (int)s->b.N0, n, ha.nnz, ha.col.get(), ha.val.get(), hb.nnz, hb.col.get(), hb.val.get(),
                          s->na * s->a.m1, exc[0].get(), s->nb * s->b.m1, exc[1].get(), V, C, sig);
    F2G_LAUNCH("k_small_sigma");
}

} // namespace f2g
