// The comb's index at a running weight, apart from the kernels so that it also
// compiles for the host.
#pragma once
#include <cmath>
#include <cstdint>

#ifdef __CUDACC__
#define STORM_HD __host__ __device__ __forceinline__
#else
#define STORM_HD inline
#endif

namespace storm {

// A combed cell's teeth: tooth k lies at the weight (k + r) e.
struct CombTeeth {
    double r, e;
    double scale, perE;   // a running weight P is near tooth P * scale * perE
    double top;           // above every index (below)
};

// perE is a reciprocal of e lifted out of the smallest numbers, where 1 / e would
// be infinite.  A combed cell holds more than nin particles, so its weight is above
// nin of the smallest double, and e, that weight over nin, rounds to no less than
// 2/3 of the quotient: the index stays below 1.5 nin + 2.
STORM_HD CombTeeth comb_teeth(double r, double e, uint64_t nin) {
    const double scale = e < 0x1p-900 ? 0x1p600 : 1.0;
    return CombTeeth{r, e, scale, 1.0 / (e * scale), 2.0 * static_cast<double>(nin) + 2.0};
}

// #{k >= 0 : (k + r) e < P} for P > 0 from the guess P * scale * perE, with the
// index as a whole number in FP64: the index follows from the comparisons, not from
// the guess, and costs neither a division nor 64-bit integer conversions.  Both
// walks stay inside [0, top], so they end whatever the numbers are.
STORM_HD double teeth_index(const CombTeeth &t, double P) {
    double k = fmin(fmax(ceil(P * t.scale * t.perE - t.r), 0.0), t.top);
    while (k > 0.0 && ((k - 1.0) + t.r) * t.e >= P) k -= 1.0;
    while (k < t.top && (k + t.r) * t.e < P) k += 1.0;
    return k;
}

}  // namespace storm
