// FP64 sigma of a C1 space on the tensor cores (see oz.cu).
#pragma once

#include <memory>
#include <vector>

#include "strings.cuh"

namespace f2g {

// One spin's two-hole lists and integral digits for the same-spin term
struct OzSpin {
    int m2 = 0, nchunk = 0, ksteps = 0; // pairs per two-hole string, 48-column chunks, K steps of 16
    DevBuf<uint32_t> up;     // [N2][ksteps * 16] I | negative << 31 of K + pair, kOzNone padding
    DevBuf<uint32_t> down;   // [N0][C(k, 2)] K | slot << 24 | negative << 31
    DevBuf<uint16_t> pair;   // [N2][nchunk * 48] index of the slot's pair (p (p - 1) / 2 + q)
    DevBuf<uint16_t> dpair;  // [N0][C(k, 2)] pair of every entry of `down`
    DevBuf<unsigned char> b; // [N2][nchunk][ksteps][kOzStepBytes] digits of the pair integrals
    DevBuf<int> bexp;        // [n (n - 1) / 2] exponent of every output pair's integrals
    DevBuf<double> diag;     // [N0] same-spin energy of every string
};

// Alpha one-hole strings [k0, k1) and the sigma rows they reach
struct OzRange {
    int64_t k0 = 0, k1 = 0;
    int64_t j0 = 0; // first entry of its rows in OzSigma::rows
    int nrows = 0;
};

// Work buffers of one stream of calls
struct OzScratch {
    int nvec = 0; // vectors per call they suffice for
    DevBuf<long long> E;
    DevBuf<uint16_t> rexp;
};

struct OzSigma {
    const CIStrings* s = nullptr;
    OzSpin spin[2];
    DevBuf<uint64_t> kstr;    // [N1b] masks of the beta one-hole strings
    DevBuf<unsigned char> vb; // [n][n][kOzBlockBytes] digits of V[p][r][q][s] per (p, q)
    DevBuf<int> vexp;         // [n][16] exponent of V[p][r][..][..]
    DevBuf<double> coul;      // [N0a][n] Coulomb energy of beta orbital q with the alpha string
    int64_t ldE = 0;          // opposite spin: elements per E row
    int64_t max_elems = 0;     // elements of the E buffer
    int64_t range_strings = 0; // alpha one-hole strings whose E fits the buffer
    std::vector<OzRange> ranges; // empty: whole vectors fit
    DevBuf<uint32_t> rows;
    OzScratch scr[2];         // [0] direct calls, [1] captured graphs
    int lead = 0;             // exponent slack that keeps the digit sums exact (see oz_lead)
    void plan(cudaStream_t st);
};

// The space's sizes fit the digit sums and the tile shapes; `fast` (optional) tells whether it is large
// enough to gain from it
bool oz_supported(const CIStrings* s, bool* fast = nullptr);
// lists of the strings (once, with at most `bytes` of E at a time where one tile or one alpha hole string allows it),
// then the digits of the integrals (stream order)
void oz_build(const CIStrings* s, std::shared_ptr<OzSigma>& oz, const double* H, const double* V, double E,
              int64_t bytes, cudaStream_t st);
// another limit for the E buffers of later calls
void oz_limit(OzSigma& oz, int64_t bytes, cudaStream_t st);
// buffers of set 0 (direct calls) or 1 (captured graphs) for calls with up to nvec vectors
// (never smaller than before)
void oz_reserve(OzSigma& oz, int set, int nvec);
// sigma = diagonal of H times C (overwrites), then the same-spin terms and the opposite-spin term, added
void oz_diag(const OzSigma& oz, const double* C, double* S, int nvec, cudaStream_t st);
void oz_same_spin(OzSigma& oz, int set, int spin, const double* C, double* S, int nvec, int max_ctas, const WaitCtl& wait,
                  cudaStream_t st);
void oz_opposite(OzSigma& oz, int set, const double* C, double* S, int nvec, int max_ctas, const WaitCtl& wait,
                 cudaStream_t st);

} // namespace f2g
