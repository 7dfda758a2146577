// pm_div.h -- integer quotients by a float reciprocal (device code; plain C++ for
// the host).
#pragma once

#ifdef __CUDACC__
#define PM_DIV_FN __host__ __device__ __forceinline__
#else
#define PM_DIV_FN inline
#endif

namespace pm {

// u / d for 0 <= u < 2^30, 0 < d < 2^20, inv = 1 / d to within 2 ulp: a float estimate,
// then steps of one.  The estimate is off by at most one for quotients below 2^21
// (all but maps of millions of rows of sub-cells), and by about q 2^-21 beyond.
PM_DIV_FN int small_div(int u, int d, float inv) {
    int q = (int)(((float)u + 0.5f) * inv), r = u - q * d;
    while (r < 0) { r += d; q--; }
    while (r >= d) { r -= d; q++; }
    return q;
}

}  // namespace pm
