// Can a foreign label that a vertex sees once never have a positive gain?
//
// With d_in = 1 the terms A and B of the model (gain.cuh) are 0 (their numerators hold
// d_in - 1), and the gain is (r - 1) C with
//   C = -(r-1)(r-2) p_in^3 (q + t) alpha / den,
//   den = ((r-1)(r-2) p_in^3 + t (t-1) p_ext + t (r-1) p_in p_ext)
//         (q + t + alpha (r - q)) (q + t + alpha (r - q - 1))
// for q = (r-1) p_in and t = (ext - 1) / r. Every factor of den is >= 0 if
//   t is 0 or at least 1 (t (t - 1) is negative between), and
//   p_in is in [0, 1]: then r - q - 1 = (r-1)(1 - p_in) >= 0.
// (r-1)(r-2) does not wrap up to r = 46340; for r <= 2 the numerator is 0 whatever den is.
// Rounding to nearest keeps all these signs, so the FP64 gain is <= 0 and the label is never
// chosen.
//
// p_in is above 1 where rows list an edge more than once or hold loops, which a transferred
// graph's may; there the last factor of den can be negative (r = 3, ext = 1, p_in = 4/3,
// alpha = 7.5: a gain of +3.3), and the label's gain has to be looked at.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SCD_RULE __host__ __device__ __forceinline__
#else
#define SCD_RULE inline
#endif

namespace scd {

// r, ext: the community's size and external edges; [pin_lo, pin_hi] encloses its p_in; alpha
// and p_ext are >= 0
SCD_RULE bool seen_once_never_gains(int r, int ext, float pin_lo, float pin_hi) {
    return r >= 1 && r <= 46340 && ext >= 1 && pin_lo >= 0.f && pin_hi <= 1.f && (r <= 2 || ext == 1 || ext - 1 >= r);
}

}  // namespace scd
