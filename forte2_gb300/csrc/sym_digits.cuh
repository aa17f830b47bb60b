// Opposite-spin sigma of a point-group-blocked space on the tensor cores (see sym_digits.cu).
#pragma once

#include <memory>

#include "opposite_sym.cuh"

namespace f2g {

constexpr int kSymSlots = 64; // orbital pairs (q, s) of one irrep per hole pair at most

struct SymDigits {
    OrbSym os{};
    int most = 0;     // pairs per hole pair at most, padded to 4
    int slots = 0;    // padded to 16
    int lmax = 0;     // beta 1-hole strings of one irrep at most, padded to 128
    int chunk = 0;    // of them at a time, a multiple of 128
    int64_t ka = 0;   // alpha 1-hole strings at a time
    int64_t njb = 0;  // beta strings of one irrep at most
    DevBuf<int8_t> hka, hja;      // irreps of the alpha 1-hole strings and strings
    DevBuf<int32_t> kpos;         // beta 1-hole string -> irrep << 24 | position among its irrep's
    DevBuf<uint32_t> tab;         // [irrep][s][position]: address | negative << 31 of K + s, ~0 without
    DevBuf<int32_t> jb, njb_of;   // [irrep][njb] beta strings, their number
    struct Scratch {
        DevBuf<uint4> z, b;       // digits of the vector and of the integrals
        DevBuf<double> e;
        DevBuf<int> ec, ecol;     // exponents of the vector's rows and a mark behind them; of every output pair of (Ka, t)
    } set[2];                     // direct calls, captured graphs
};

// null if the space is left to the FP64 kernel (opposite_sym.cu)
std::shared_ptr<SymDigits> sym_digits_build(const CIStrings* s, const OppositeSym& t);
void sym_digits_plan(SymDigits& d, const CIStrings* s, int64_t bytes); // parts for work buffers of that size
void sym_digits_reserve(SymDigits& d, const CIStrings* s, int set);
// sigma += the opposite-spin term for nvec C1-embedded vectors back to back
void sym_digits_run(SymDigits& d, const CIStrings* s, int set, const double* V, const double* C, double* sig, int nvec,
                    int max_ctas, const WaitCtl& wait, cudaStream_t st);

} // namespace f2g
