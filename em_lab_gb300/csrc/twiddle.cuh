// twiddle.cuh - e^{j k r p} of a direction component r at lattice positions p, for the pattern kernels.
#pragma once

namespace emlab {

// sin and cos of 2 pi (a p) for the position p (exact in float): a = hi + lo in turns per cell, formed
// in FP64, so the product with p is reduced to [-1/2, 1/2] turns without losing the phase's low bits
// (a float phase of 60 rad is off by up to 4e-6). Then the nearest quarter turn is taken out and sin and
// cos of the rest, |r| <= pi/4, are their Taylor polynomials to r^9 and r^8 (truncation below 3e-8).
struct Turns {
    float hi, lo;
};

__device__ __forceinline__ Turns turns_per_cell(double k, float r) {
    const double t = k * (double)r * 0.15915494309189535;
    const float hi = (float)t;
    return {hi, (float)(t - (double)hi)};
}

__device__ __forceinline__ void twiddle(Turns a, float p, float& s, float& c) {
    const float n = rintf(a.hi * p);
    const float f = fmaf(a.lo, p, fmaf(a.hi, p, -n));
    const float m = rintf(4.0f * f);
    const float r = fmaf(-0.25f, m, f) * 6.283185307f;
    const float r2 = r * r;
    float ps = 2.7557319e-6f, pc = 2.4801587e-5f;
    ps = fmaf(ps, r2, -1.9841270e-4f), pc = fmaf(pc, r2, -1.3888889e-3f);
    ps = fmaf(ps, r2, 8.3333333e-3f), pc = fmaf(pc, r2, 4.1666667e-2f);
    ps = fmaf(ps, r2, -1.6666667e-1f), pc = fmaf(pc, r2, -0.5f);
    ps = fmaf(ps * r2, r, r), pc = fmaf(pc, r2, 1.0f);
    const int q = (int)m;  // quarter turns, -2 .. 2
    const bool swap = q & 1;
    s = swap ? pc : ps, c = swap ? ps : pc;
    if (q & 2) s = -s;
    if ((q + 1) & 2) c = -c;
}

}  // namespace emlab
