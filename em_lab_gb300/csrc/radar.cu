// radar.cu - back-projection imaging of the pulsed phased-array radar (src/Radar.cpp:606-646).
//
// For every image point P = tx + r * direction(az, el) inside the simulated volume, the complex
// baseband echoes z_i of all receive elements are sampled at the point's round-trip delay
// (transmit group delay of the near-field array factor, Radar.cpp:87-103, plus the distance back to
// element i), interpolated linearly between decimated samples, weighted by the receive taper and
// re-phased to the carrier: power = |sum_i w_i z_i(t_i) e^{j w t_i}|^2. One thread per image point;
// geometry in FP32 as the reference computes it (compiled without contraction). The reference spreads
// elevation rows over CPU threads; here the whole range x elevation x azimuth volume is one launch.
//
// The reference's sums are FP64, and the FP64 pipe (two multiply-adds per SM and cycle against 128 in
// FP32) bounded the image: two sincos, three divisions and about forty other FP64 operations per
// element and point. Here every FP64 quantity inside the element loops is an unevaluated pair of FP32
// (about 47 significant bits): distances are FP32 already, phases are reduced in turns exactly, sin and
// cos come from a 512-entry table of pairs and a short series, delays are summed as differences from
// the array centre's, and the common factor e^{j w t_out} of the receive sum is left out (it does not
// change the power). The weighted mean delay is formed in FP64 once per point.
//
// What the pairs cannot decide is the rounding of the interpolation weight to FP32 and whether a delay
// reaches the last sample. So each point carries a bound of its delay's error, and a point for which a
// rounding within that bound could move the power by more than 2e-8 of itself, or whose sums are out
// of the pairs' range or not finite, is formed again in FP64, in the reference's order, by its whole
// warp. Images of 9 to 64 elements agree with the FP64 kernel's to 1e-14 of their power (2% of the points
// with 36 elements, 7% with 64, take the second way). One call, 64 x 61 x 41 points and 36 elements:
// 1558 us before, 428 us here; 90 x 61 x 61 points and 64 elements: 4734 and 934 us.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <new>

#include "../../include/emlab.h"
#include "emlab_internal.h"

namespace emlab {
namespace {

struct F3 {
    float x, y, z;
};
__device__ __forceinline__ F3 sub(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ F3 add(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ F3 mul(F3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float len(F3 a) { return sqrtf(dot(a, a)); }
__device__ __forceinline__ F3 ld3(const float* p) { return {p[0], p[1], p[2]}; }

// Unevaluated sums hi + lo of two floats (Dekker, Numer. Math. 18, 1971; Knuth, TAOCP 2, 4.2.2).
struct FF {
    float h, l;
};
__host__ __device__ __forceinline__ FF to_ff(double v) {
    const float h = (float)v;
    return {h, (float)(v - (double)h)};
}
__device__ __forceinline__ double to_f64(FF a) { return (double)a.h + (double)a.l; }
__device__ __forceinline__ FF fast_sum(float a, float b) {  // |a| >= |b|
    const float s = a + b;
    return {s, b - (s - a)};
}
__device__ __forceinline__ FF two_sum(float a, float b) {
    const float s = a + b, t = s - a;
    return {s, (a - (s - t)) + (b - t)};
}
__device__ __forceinline__ FF operator+(FF a, FF b) {
    const FF s = two_sum(a.h, b.h);
    return fast_sum(s.h, s.l + (a.l + b.l));
}
__device__ __forceinline__ FF operator+(FF a, float b) {
    const FF s = two_sum(a.h, b);
    return fast_sum(s.h, s.l + a.l);
}
__device__ __forceinline__ FF operator-(FF a) { return {-a.h, -a.l}; }
__device__ __forceinline__ FF operator*(FF a, FF b) {
    const float p = a.h * b.h;
    return fast_sum(p, fmaf(a.l, b.h, fmaf(a.h, b.l, fmaf(a.h, b.h, -p))));
}
__device__ __forceinline__ FF operator*(FF a, float b) {
    const float p = a.h * b;
    return fast_sum(p, fmaf(a.l, b, fmaf(a.h, b, -p)));
}

// e^{j w d}, d >= 0 in FP32, from wt = w / 2 pi in turns per unit as a sum of three floats: the turns are
// reduced to the nearest table entry (exactly: the products with d are kept in full), the rest r,
// |r| <= pi / 512, enters through sin r = r - r^3/6 + r^5/120 and cos r = 1 - r^2/2 + r^4/24 (truncation
// below 1e-16).
constexpr int kTable = 512, kThreads = 128;
constexpr float kTurns = 4096.0f;  // the rest e below stays under 2^-12 of a turn
struct Turns {
    float h, m, l;
};
struct Phase {
    FF c, s;
};
__device__ __forceinline__ Phase phase(const float4* table, Turns wt, float d) {
    const float p = wt.h * d, u = wt.m * d;
    const FF e = two_sum(fmaf(wt.h, d, -p), u);
    const float el = e.l + fmaf(wt.l, d, fmaf(wt.m, d, -u));
    const float f = p - rintf(p);  // exact
    const float k = rintf(f * (float)kTable);
    FF t = two_sum(fmaf(k, -1.0f / kTable, f), e.h);  // turns beyond the entry; the first term is exact
    t = fast_sum(t.h, t.l + el);
    constexpr float two_pi_h = 6.28318548f, two_pi_l = -1.74845553e-7f;
    const FF r = t * FF{two_pi_h, two_pi_l};
    const float r2 = r.h * r.h;
    const FF sr = fast_sum(r.h, fmaf(r.h * r2, fmaf(r2, 8.33333377e-3f, -0.166666672f), r.l));
    const float r2l = fmaf(2.0f * r.h, r.l, fmaf(r.h, r.h, -r2));
    const FF cm = {-0.5f * r2, fmaf(r2 * r2, 4.16666679e-2f, -0.5f * r2l)};  // cos r - 1
    const float4 v = table[(int)k & (kTable - 1)];
    const FF ct = {v.x, v.y}, st = {v.z, v.w};
    // ct cos r - st sin r = ct + (ct (cos r - 1) - st sin r)
    return {ct + (ct * cm + -(st * sr)), st + (st * cm + ct * sr)};
}

struct Geo {
    F3 tx, ax0, ax1, ax2, lo, hi;
};

struct Inputs {
    const float2* z;
    int M, C, ntx;
    const float *elem_pos, *tx_pos;
    const FF *weights, *tx_amp;              // as pairs,
    const double *weights64, *tx_amp64;      // and as they came
};

// Sums whose squares and low parts stay normal numbers; false for a NaN.
__device__ __forceinline__ bool in_range(float v) { return v > 1e-18f && v < 1e18f; }

// The power at p in FP64 by one warp: the lanes form the terms of 32 elements, and one lane per sum adds
// them in the order of the elements. terms: 32 x 5 doubles of this warp.
__device__ __noinline__ double point64(const Geo& g, F3 p, const Inputs& in, double w, double dt, double sdt,
                                       double (*terms)[5]) {
    const int lane = threadIdx.x & 31;
    auto add_terms = [&](double acc, int sums, int n) {
        __syncwarp();
        if (lane < sums)
            for (int k = 0; k < n; ++k) acc += terms[k][lane];
        __syncwarp();
        return acc;
    };
    // RadarMonitor::txDelay (Radar.cpp:87-103)
    double acc = 0.0;
    for (int j0 = 0; j0 < in.ntx; j0 += 32) {
        const int j = j0 + lane;
        if (j < in.ntx) {
            const F3 v = sub(p, ld3(in.tx_pos + 3 * j));
            const double d = fmax((double)len(v), 0.5);
            const double gj = fmax((double)dot(v, g.ax2) / d, 0.0);
            const double a = in.tx_amp64[j] * gj / d;
            double s, c;
            sincos(-w * d, &s, &c);
            const double tr = a * c, ti = a * s;
            terms[lane][0] = tr, terms[lane][1] = ti;
            terms[lane][2] = d * tr, terms[lane][3] = d * ti;
            terms[lane][4] = a;
        }
        acc = add_terms(acc, 5, min(32, in.ntx - j0));
    }
    const unsigned all = 0xffffffffu;
    const double ar = __shfl_sync(all, acc, 0), ai = __shfl_sync(all, acc, 1), adr = __shfl_sync(all, acc, 2),
                 adi = __shfl_sync(all, acc, 3), mag = __shfl_sync(all, acc, 4);
    const double absa = sqrt(ar * ar + ai * ai);
    const double outbound = absa < 1e-3 * mag ? (double)len(sub(p, g.tx))
                                              : (adr * ar + adi * ai) / (ar * ar + ai * ai);  // real(ad / a)
    acc = 0.0;
    for (int i0 = 0; i0 < in.C; i0 += 32) {
        const int i = i0 + lane;
        if (i < in.C) {
            double tr = 0.0, ti = 0.0;
            const double t = outbound + (double)len(sub(p, ld3(in.elem_pos + 3 * i)));  // path delay
            const double s = (t + 0.5 * dt) / sdt;                                       // decimated sample
            if (s != s) tr = ti = s;
            if (s >= 0.0 && s < (double)(in.M - 1)) {
                const int m0 = (int)s;
                const float f = (float)(s - (double)m0);
                const float2 z0 = in.z[(long long)m0 * in.C + i], z1 = in.z[(long long)(m0 + 1) * in.C + i];
                const float vr = z0.x * (1.0f - f) + z1.x * f, vi = z0.y * (1.0f - f) + z1.y * f;
                double sn, cs;
                sincos(w * t, &sn, &cs);
                const double wr = in.weights64[i] * (double)vr, wi = in.weights64[i] * (double)vi;
                tr = wr * cs - wi * sn;
                ti = wr * sn + wi * cs;
            }
            terms[lane][0] = tr, terms[lane][1] = ti;
        }
        acc = add_terms(acc, 2, min(32, in.C - i0));
    }
    const double sr = __shfl_sync(all, acc, 0), si = __shfl_sync(all, acc, 1);
    return sr * sr + si * si;
}

struct Delay {
    double t;
    float err;  // bound of the difference from the FP64 sums; negative: to be formed in FP64
};

// RadarMonitor::txDelay (Radar.cpp:87-103). The bound scales with the cancellation in the array factor
// and was fitted on the CPU against FP64 and extended sums: arrays of 1 to 256 elements half a wavelength
// apart, 2 to 1000 cells away, with a factor of two and more in hand; cancellation beyond 100 goes to FP64.
__device__ __forceinline__ Delay tx_delay(const Geo& g, F3 p, const float4* table, Turns wt, const Inputs& in) {
    FF ar = {0, 0}, ai = ar, adr = ar, adi = ar, mag = ar;
    const float d0 = len(sub(p, g.tx));
    float spread = 0.0f, far = 0.0f;
    for (int j = 0; j < in.ntx; ++j) {
        const F3 v = sub(p, ld3(in.tx_pos + 3 * j));
        const float d = fmaxf(len(v), 0.5f);
        const float q = 1.0f / d;
        const FF inv = {q, q * fmaf(-q, d, 1.0f)};
        const FF a = (in.tx_amp[j] * (inv * inv)) * fmaxf(dot(v, g.ax2), 0.0f);  // amp (g / d) / d
        const Phase e = phase(table, wt, d);
        const FF tr = a * e.c, ti = a * e.s;  // the conjugate of a e^{-j w d}
        const FF dd = two_sum(d, -d0);
        ar = ar + tr, ai = ai + ti;
        adr = adr + tr * dd, adi = adi + ti * dd;
        mag = mag + a;
        spread = fmaxf(spread, fabsf(dd.h)), far = fmaxf(far, d);
    }
    if (!in_range(mag.h) || !in_range(fmaxf(fabsf(ar.h), fabsf(ai.h))) || !(fabsf(wt.h) * far < kTurns))
        return {0.0, -1.0f};
    const double r = to_f64(ar), i = to_f64(ai);
    const double t = (double)d0 + (to_f64(adr) * r + to_f64(adi) * i) / (r * r + i * i);  // real(ad / a)
    const float over = rsqrtf(ar.h * ar.h + ai.h * ai.h), k = mag.h * over;
    const float rest = sqrtf(adr.h * adr.h + adi.h * adi.h) * over;
    const float err = k * (0x1p-47f * (spread + rest) + 0x1p-52f * (fabsf((float)t) + d0));
    return {t, k < 100.0f && fabs(t) < 1e18 ? err : -1.0f};
}

struct RadarTable {
    float4 v[kTable];  // cos, sin of 2 pi k / kTable, each as a pair
};

__global__ void __launch_bounds__(kThreads) backproject_kernel(const __grid_constant__ emlab_radar_geometry geo,
                                                          const __grid_constant__ RadarTable tab, Turns wt, FF half_dt,
                                                          FF inv_sdt, const __grid_constant__ Inputs in, double* power) {
    __shared__ float4 table[kTable];
    __shared__ double terms[kThreads / 32][32][5];
    for (int k = threadIdx.x; k < kTable; k += kThreads) table[k] = tab.v[k];
    __syncthreads();
    const long long idx = blockIdx.x * (long long)kThreads + threadIdx.x;
    const long long total = (long long)geo.nr * geo.nel * geo.naz;
    const int ia = (int)(idx % geo.naz);
    const int ie = (int)((idx / geo.naz) % geo.nel);
    const int ir = (int)(idx / ((long long)geo.naz * geo.nel));
    Geo g;
    g.tx = ld3(geo.tx), g.ax0 = ld3(geo.axes), g.ax1 = ld3(geo.axes + 3), g.ax2 = ld3(geo.axes + 6);
    g.lo = ld3(geo.interior_min), g.hi = ld3(geo.interior_max);
    // RadarMonitor::direction (Radar.cpp:69-72)
    const float az = geo.az0 + (float)ia * geo.daz, el = geo.el0 + (float)ie * geo.del;
    const float a = az * 0.01745329251994329577f, e = el * 0.01745329251994329577f;
    const float sa = sinf(a), ca = cosf(a), se = sinf(e), ce = cosf(e);
    const F3 dir = add(add(mul(g.ax0, sa * ce), mul(g.ax1, se)), mul(g.ax2, ca * ce));
    const float r = geo.r0 + (float)ir * geo.dr;
    const F3 P = add(g.tx, mul(dir, r));
    // a point outside the simulated volume reads -1
    const bool inside = idx < total && !(P.x < g.lo.x || P.y < g.lo.y || P.z < g.lo.z || P.x > g.hi.x ||
                                         P.y > g.hi.y || P.z > g.hi.z);
    double result = -1.0;
    bool again = false;
    if (inside) {
        const Delay delay = tx_delay(g, P, table, wt, in);
        const FF outbound = to_ff(delay.t) + half_dt;  // with the half step
        const float err = fabsf(delay.err * inv_sdt.h);
        FF sr = {0, 0}, si = sr;
        bool any = false;
        float doubt = 0.0f;  // by how much roundings within the error could move the sum
        const int n = delay.err < 0.0f ? 0 : in.C;
        for (int i = 0; i < n; ++i) {
            const float d = len(sub(P, ld3(in.elem_pos + 3 * i)));  // path delay beyond the outbound one
            const FF s = (outbound + d) * inv_sdt;                   // decimated sample
            float m = floorf(s.h);
            if (m == s.h && s.l < 0.0f) m -= 1.0f;
            const float part = s.h - m, eps = err + 0x1p-47f * fabsf(s.h);
            const float f = part + s.l, above = part + (s.l + eps), below = part + (s.l - eps);
            if (above >= 1.0f || below < 0.0f || !(fabsf(s.h) < 1e9f) || !(fabsf(wt.h * d) < kTurns)) doubt = INFINITY;
            if (!(m >= 0.0f && m < (float)(in.M - 1))) continue;
            const int m0 = (int)m;
            const float2 z0 = in.z[(long long)m0 * in.C + i], z1 = in.z[(long long)(m0 + 1) * in.C + i];
            const float vr = z0.x * (1.0f - f) + z1.x * f, vi = z0.y * (1.0f - f) + z1.y * f;
            if (above != below) {
                // a unit in the last place of f and of 1 - f, and the roundings that follow from it
                const float a0 = sqrtf(z0.x * z0.x + z0.y * z0.y), a1 = sqrtf(z1.x * z1.x + z1.y * z1.y);
                doubt += fabsf(in.weights[i].h) * (0x1p-23f * (a0 + a1));
            }
            const Phase q = phase(table, wt, d);
            const FF wr = in.weights[i] * vr, wi = in.weights[i] * vi;
            sr = sr + (wr * q.c + -(wi * q.s));
            si = si + (wr * q.s + wi * q.c);
            any |= vr != 0.0f || vi != 0.0f;
        }
        const double pr = to_f64(sr), pi = to_f64(si);
        result = pr * pr + pi * pi;
        const float top = fmaxf(fabsf(sr.h), fabsf(si.h));
        again = delay.err < 0.0f || doubt > 1e-8f * top || (any && !in_range(top));
    }
    const unsigned all = 0xffffffffu;
    for (unsigned todo = __ballot_sync(all, again); todo; todo &= todo - 1) {
        const int lane = __ffs(todo) - 1;
        const F3 p = {__shfl_sync(all, P.x, lane), __shfl_sync(all, P.y, lane), __shfl_sync(all, P.z, lane)};
        const double v = point64(g, p, in, geo.omega, geo.dt, geo.sample_dt, terms[threadIdx.x / 32]);
        if ((threadIdx.x & 31) == lane) result = v;
    }
    if (idx < total) power[idx] = result;
}

}  // namespace
}  // namespace emlab

using namespace emlab;

extern "C" int emlab_radar_backproject(const emlab_radar_geometry* geo, const float* z, int M, int C,
                                       const float* elem_pos, const double* weights, const float* tx_pos,
                                       const double* tx_amp, int ntx, double* power) {
    if (!geo || !z || !elem_pos || !weights || !tx_pos || !tx_amp || !power || M < 2 || C < 1 || ntx < 1 ||
        geo->nr < 1 || geo->naz < 1 || geo->nel < 1)
        return report_error(EMLAB_ERR_INVALID, "bad radar back-projection arguments");
    const long long total = (long long)geo->nr * geo->nel * geo->naz;
    if (total > (1ll << 31)) return report_error(EMLAB_ERR_INVALID, "radar image too large");
    // device memory first: sizes that cannot be had end here, before anything is read. One buffer: z, the weights
    // and amplitudes in FP64 and as pairs, the positions, the image
    const size_t zb = (size_t)M * C * 8, nb = ((size_t)C + ntx) * 8, pb = ((size_t)C + ntx) * 12;
    const size_t bytes = (zb + 2 * nb + pb + 15) / 16 * 16;
    unsigned char* buf = nullptr;
    if ((size_t)M > SIZE_MAX / 16 / (size_t)C || cudaMalloc(&buf, bytes + (size_t)total * 8) != cudaSuccess) {
        cudaGetLastError();
        return report_error(EMLAB_ERR_OOM, "radar: device allocation failed");
    }
    // One copy for all inputs where z is short. A longer z goes from the caller's array by a copy of its own, which
    // costs less than bringing it together with the rest from about this size on.
    const size_t packed_z = zb <= (128u << 10) ? zb : 0;
    std::unique_ptr<unsigned char[]> host(new (std::nothrow) unsigned char[packed_z + 2 * nb + pb]);
    if (!host) {
        cudaFree(buf);
        return report_error(EMLAB_ERR_OOM, "radar: host allocation failed");
    }
    unsigned char* rest = host.get() + packed_z;
    if (packed_z) std::memcpy(host.get(), z, zb);
    std::memcpy(rest, weights, (size_t)C * 8);
    std::memcpy(rest + (size_t)C * 8, tx_amp, (size_t)ntx * 8);
    FF* pairs = reinterpret_cast<FF*>(rest + nb);
    for (int i = 0; i < C; ++i) pairs[i] = to_ff(weights[i]);
    for (int j = 0; j < ntx; ++j) pairs[C + j] = to_ff(tx_amp[j]);
    std::memcpy(rest + 2 * nb, elem_pos, (size_t)C * 12);
    std::memcpy(rest + 2 * nb + (size_t)C * 12, tx_pos, (size_t)ntx * 12);
    RadarTable table;
    for (int k = 0; k < kTable; ++k) {
        const double t = 6.28318530717958647692 * k / kTable;
        const FF c = to_ff(std::cos(t)), s = to_ff(std::sin(t));
        table.v[k] = make_float4(c.h, c.l, s.h, s.l);
    }
    const double turns = geo->omega / 6.28318530717958647692;
    const FF w2 = to_ff(turns);
    const Turns wt = {w2.h, w2.l, (float)(turns - (double)w2.h - (double)w2.l)};
    double* dp = reinterpret_cast<double*>(buf + bytes);
    cudaError_t e = cudaSuccess;
    if (!packed_z) e = cudaMemcpy(buf, z, zb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(buf + zb - packed_z, host.get(), packed_z + 2 * nb + pb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const double* d64 = reinterpret_cast<const double*>(buf + zb);
        const FF* dff = reinterpret_cast<const FF*>(buf + zb + nb);
        const float* pos = reinterpret_cast<const float*>(buf + zb + 2 * nb);
        const Inputs in = {reinterpret_cast<const float2*>(buf), M, C, ntx, pos, pos + 3 * (size_t)C, dff, dff + C, d64, d64 + C};
        backproject_kernel<<<(unsigned)((total + kThreads - 1) / kThreads), kThreads>>>(
            *geo, table, wt, to_ff(0.5 * geo->dt), to_ff(1.0 / geo->sample_dt), in, dp);
        count_launches(1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(power, dp, (size_t)total * 8, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    if (e != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(e));
    return EMLAB_OK;
}
