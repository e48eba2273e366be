// FP32 hi / lo split of the FP64 duals of a mixed pass, on a grid that all duals
// of the pass share: g = 2^(floor(log2 max |dual|) - 21).
#pragma once

#include <cuda_runtime.h>

namespace regot {

struct SplitGrid {
    double g = 1.0, inv_g = 1.0;
    // of *maxabs (null: the unit grid)
    __device__ explicit SplitGrid(const double* maxabs) {
        if (!maxabs) return;
        const double mx = *maxabs;
        if (mx > 0.0 && isfinite(mx)) {
            const int e = ilogb(mx) - 21;
            g = ldexp(1.0, e);
            inv_g = ldexp(1.0, -e);
        }
    }
    __device__ __forceinline__ void split(double v, float& hi, float& lo) const {
        if (!isfinite(v)) {
            hi = (float)v;
            lo = 0.f;
            return;
        }
        const double h = rint(v * inv_g) * g;
        hi = (float)h;
        lo = (float)(v - h);
    }
};

}  // namespace regot
