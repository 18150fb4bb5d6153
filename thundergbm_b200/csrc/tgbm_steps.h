// Loops that step through stored values.
#pragma once
#ifdef __CUDACC__
#define TGBM_HD __host__ __device__ __forceinline__
#else
#define TGBM_HD inline
#endif

namespace tgbm {

// f(begin + first), f(begin + first + step), ... for all positions before `end`.  Positions run up to INT_MAX and the last step
// goes beyond them: counted as an int it would come out below zero, which is before the end as well.  f takes an unsigned, and so
// does what it adds to it.
template <typename F>
TGBM_HD void each_step(int begin, int end, unsigned first, unsigned step, F f) {
    for (unsigned j = (unsigned)begin + first; j < (unsigned)end; j += step) f(j);
}

}  // namespace tgbm
