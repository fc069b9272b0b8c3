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
    double perE;   // 1 / e, or zero where that is not finite
    double top;    // above every index (below)
};

// A combed cell holds more than nin particles, so its weight is above
// nin of the smallest double, and e, that weight over nin, rounds to no less than
// 2/3 of the quotient: the index stays below 1.5 nin + 2.
STORM_HD CombTeeth comb_teeth(double r, double e, uint64_t nin) {
    return CombTeeth{r, e, e < 0x1p-1000 ? 0.0 : 1.0 / e, 2.0 * static_cast<double>(nin) + 2.0};
}

// #{k >= 0 : (k + r) e < P} for P > 0 from the guess P / e, with the index as a whole
// number in FP64: the index follows from the comparisons, not from the guess, and
// costs neither a division (but for the smallest numbers) nor 64-bit integer
// conversions.  Both walks stay inside [0, top], so they end whatever the numbers are.
STORM_HD double teeth_index(const CombTeeth &t, double P) {
    double k = fmin(fmax(ceil((t.perE > 0.0 ? P * t.perE : P / t.e) - t.r), 0.0), t.top);
    while (k > 0.0 && ((k - 1.0) + t.r) * t.e >= P) k -= 1.0;
    while (k < t.top && (k + t.r) * t.e < P) k += 1.0;
    return k;
}

}  // namespace storm
