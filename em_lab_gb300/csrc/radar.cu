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
// (48 bits, radar_pairs.cuh): distances are FP32 already, phases are reduced in turns exactly, sin and
// cos come from a 512-entry table of pairs and a short series, delays are summed as differences from
// the array centre's, and the common factor e^{j w t_out} of the receive sum is left out (it does not
// change the power). The weighted mean delay is formed in FP64 once per point.
//
// What the pairs cannot decide is the rounding of the interpolation weight to FP32 and whether a delay
// reaches the last sample. So each position carries a bound of its distance from the FP64 sums', derived
// beside the code that forms it, and a point for which a rounding within that bound and the pairs' own errors
// could move the power by more than 2e-10 of itself, or whose sums are out of the pairs' range or not finite,
// is formed again in FP64, in the reference's order, by its whole warp. The power is thus within 2e-10 of the
// FP64 sums'.
// One call, 64 x 61 x 41 points and 36 elements: 1560 us with FP64 sums, 415 us here (the kernel 197 us, about 1 % of the
// points the second way); 90 x 61 x 61 points and 64 elements: 4930 and 780 us.
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <new>

#include "../../include/emlab.h"
#include "emlab_internal.h"
#include "radar_pairs.cuh"

namespace emlab {
namespace {

using namespace radar;

constexpr int kThreads = 128;

struct Geo {
    F3 tx, ax0, ax1, ax2, lo, hi;
};

struct Inputs {
    const float2* z;
    int M, C, ntx;
    const float *elem_pos, *tx_pos;
    const FF *weights, *tx_amp;              // as pairs,
    const double *weights64, *tx_amp64;      // and as they came
    bool pairs;                              // the weights can be held as pairs
};

// The reference's sums at a point in FP64: the terms of a transmitting and of a receiving element, and the delay from
// the former's sums.
struct Point64 {
    const Geo& g;
    F3 p;
    const Inputs& in;
    double w, dt, sdt;

    // RadarMonitor::txDelay (Radar.cpp:87-103)
    __device__ void tx_term(int j, double (&t)[5]) const {
        const F3 v = sub(p, ld3(in.tx_pos + 3 * j));
        const double d = fmax((double)len(v), 0.5);
        const double gj = fmax((double)dot(v, g.ax2) / d, 0.0);
        const double a = in.tx_amp64[j] * gj / d;
        double s, c;
        sincos(-w * d, &s, &c);
        t[0] = a * c, t[1] = a * s;
        t[2] = d * t[0], t[3] = d * t[1];
        t[4] = a;
    }
    __device__ double outbound(double ar, double ai, double adr, double adi, double mag) const {
        const double absa = sqrt(ar * ar + ai * ai);
        return absa < 1e-3 * mag ? (double)len(sub(p, g.tx)) : (adr * ar + adi * ai) / (ar * ar + ai * ai);  // real(ad / a)
    }
    __device__ void rx_term(int i, double outbound, double (&o)[2]) const {
        o[0] = o[1] = 0.0;
        const double t = outbound + (double)len(sub(p, ld3(in.elem_pos + 3 * i)));  // path delay
        const double s = (t + 0.5 * dt) / sdt;                                       // decimated sample
        if (s != s) o[0] = o[1] = s;
        if (s >= 0.0 && s < (double)(in.M - 1)) {
            const int m0 = (int)s;
            const float f = (float)(s - (double)m0);
            const float2 z0 = in.z[(long long)m0 * in.C + i], z1 = in.z[(long long)(m0 + 1) * in.C + i];
            const float vr = z0.x * (1.0f - f) + z1.x * f, vi = z0.y * (1.0f - f) + z1.y * f;
            double sn, cs;
            sincos(w * t, &sn, &cs);
            const double wr = in.weights64[i] * (double)vr, wi = in.weights64[i] * (double)vi;
            o[0] = wr * cs - wi * sn;
            o[1] = wr * sn + wi * cs;
        }
    }
};

// The power by one warp: the lanes form the terms of 32 elements, and one lane per sum adds them in the order of the
// elements. terms: 32 x 5 doubles of this warp.
__device__ __noinline__ double point_by_warp(const Point64& q, double (*terms)[5]) {
    const int lane = threadIdx.x & 31, ntx = q.in.ntx, C = q.in.C;
    auto add_terms = [&](double acc, int sums, int n) {
        __syncwarp();
        if (lane < sums)
            for (int k = 0; k < n; ++k) acc += terms[k][lane];
        __syncwarp();
        return acc;
    };
    double acc = 0.0;
    for (int j0 = 0; j0 < ntx; j0 += 32) {
        if (j0 + lane < ntx) {
            double t[5];
            q.tx_term(j0 + lane, t);
            for (int k = 0; k < 5; ++k) terms[lane][k] = t[k];
        }
        acc = add_terms(acc, 5, min(32, ntx - j0));
    }
    const unsigned all = 0xffffffffu;
    const double ar = __shfl_sync(all, acc, 0), ai = __shfl_sync(all, acc, 1), adr = __shfl_sync(all, acc, 2),
                 adi = __shfl_sync(all, acc, 3), mag = __shfl_sync(all, acc, 4);
    const double outbound = q.outbound(ar, ai, adr, adi, mag);
    acc = 0.0;
    for (int i0 = 0; i0 < C; i0 += 32) {
        if (i0 + lane < C) {
            double o[2];
            q.rx_term(i0 + lane, outbound, o);
            terms[lane][0] = o[0], terms[lane][1] = o[1];
        }
        acc = add_terms(acc, 2, min(32, C - i0));
    }
    const double sr = __shfl_sync(all, acc, 0), si = __shfl_sync(all, acc, 1);
    return sr * sr + si * si;
}

// The same by one lane.
__device__ __noinline__ double point_by_lane(const Point64& q) {
    double sum[5] = {}, t[5], sr = 0.0, si = 0.0, o[2];
    for (int j = 0; j < q.in.ntx; ++j) {
        q.tx_term(j, t);
        for (int k = 0; k < 5; ++k) sum[k] += t[k];
    }
    const double outbound = q.outbound(sum[0], sum[1], sum[2], sum[3], sum[4]);
    for (int i = 0; i < q.in.C; ++i) {
        q.rx_term(i, outbound, o);
        sr += o[0], si += o[1];
    }
    return sr * sr + si * si;
}

__global__ void __launch_bounds__(kThreads) backproject_kernel(const __grid_constant__ emlab_radar_geometry geo,
                                                          const __grid_constant__ RadarTable tab, Triple wt, Triple inv_sdt,
                                                          const __grid_constant__ Inputs in, double* power) {
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
        const Delay delay = tx_delay(g.tx, g.ax2, P, table, wt, {in.tx_pos, in.tx_amp, in.ntx});
        const Record rec = record_of(delay, geo.dt, geo.sample_dt, inv_sdt);
        FF sr = {0, 0}, si = sr;
        bool any = false;
        // by how much the roundings within the bounds could move the sum; and what the pairs' errors scale with: the
        // magnitudes of the terms and of the running sums, the largest distance
        float doubt = 0.0f, terms32 = 0.0f, sums = 0.0f, far = 0.0f;
        const int n = delay.err < 0.0f || !in.pairs ? 0 : in.C;
        for (int i = 0; i < n; ++i) {
            const float d = len(sub(P, ld3(in.elem_pos + 3 * i)));  // path delay beyond the outbound one
            const Sample at = sample_at(rec, d);
            if (!at.clear || !(fabsf(wt.h) * d < kTurns)) doubt = INFINITY;
            if (at.m < 0 || at.m >= in.M - 1) continue;
            const float f = at.f;
            const float2 z0 = in.z[(long long)at.m * in.C + i], z1 = in.z[(long long)(at.m + 1) * in.C + i];
            const float vr = z0.x * (1.0f - f) + z1.x * f, vi = z0.y * (1.0f - f) + z1.y * f;
            if (at.above != at.below)  // the interpolated value's range, part by part
                doubt += fabsf(in.weights[i].h) * (interpolation_range(z0.x, z1.x, at) + interpolation_range(z0.y, z1.y, at));
            const Phase q = phase(table, wt, d);
            const FF wr = in.weights[i] * vr, wi = in.weights[i] * vi;
            sr = sr + (wr * q.c + -(wi * q.s));
            si = si + (wr * q.s + wi * q.c);
            any |= vr != 0.0f || vi != 0.0f;
            terms32 += fabsf(wr.h) + fabsf(wi.h), sums += fabsf(sr.h) + fabsf(si.h), far = fmaxf(far, d);
        }
        const double pr = to_f64(sr), pi = to_f64(si);
        result = pr * pr + pi * pi;
        const float top = fmaxf(fabsf(sr.h), fabsf(si.h));
        // a term: weight 3 u^2, phase 7, products 5, additions 3 each, as in tx_delay's; FP64's w t: 2^-53 of its radians
        doubt += 0x1p-48f * (36.0f * terms32 + 3.0f * sums) + 0x1p-53f * 6.3f * (fabsf(wt.h) * far) * terms32;
        again = delay.err < 0.0f || !in.pairs || !(doubt <= 1e-10f * top) || (any && !in_range(top));
    }
    // Few points of a warp are formed again by all its lanes together, one after the other: rounds of 32 terms for each.
    // Where that is more rounds than the terms of one point, each lane takes its own (an array with an element at its
    // centre and bins a whole number of samples away has rows of such points: 64 x 61 x 41 points and one element
    // 314 us with FP64 sums, 459 with such points by the warp, 245 here).
    const unsigned all = 0xffffffffu;
    unsigned todo = __ballot_sync(all, again);
    if (__popc(todo) * ((in.ntx + 31) / 32 + (in.C + 31) / 32) > in.ntx + in.C) {
        if (again) result = point_by_lane({g, P, in, geo.omega, geo.dt, geo.sample_dt});
        todo = 0;
    }
    for (; todo; todo &= todo - 1) {
        const int lane = __ffs(todo) - 1;
        const F3 p = {__shfl_sync(all, P.x, lane), __shfl_sync(all, P.y, lane), __shfl_sync(all, P.z, lane)};
        const double v = point_by_warp({g, p, in, geo.omega, geo.dt, geo.sample_dt}, terms[threadIdx.x / 32]);
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
    double* dp = reinterpret_cast<double*>(buf + bytes);
    cudaError_t e = cudaSuccess;
    if (!packed_z) e = cudaMemcpy(buf, z, zb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess)
        e = cudaMemcpy(buf + zb - packed_z, host.get(), packed_z + 2 * nb + pb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        const double* d64 = reinterpret_cast<const double*>(buf + zb);
        const FF* dff = reinterpret_cast<const FF*>(buf + zb + nb);
        const float* pos = reinterpret_cast<const float*>(buf + zb + 2 * nb);
        const Inputs in = {reinterpret_cast<const float2*>(buf), M, C, ntx, pos, pos + 3 * (size_t)C, dff, dff + C, d64, d64 + C,
                           pairs_hold(weights, C)};
        backproject_kernel<<<(unsigned)((total + kThreads - 1) / kThreads), kThreads>>>(
            *geo, make_table(), turns_of(geo->omega), quotient(1.0, geo->sample_dt, 0.0), in, dp);
        count_launches(1);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(power, dp, (size_t)total * 8, cudaMemcpyDeviceToHost);
    cudaFree(buf);
    if (e != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(e));
    return EMLAB_OK;
}

extern "C" int emlab_debug_radar_delays(const emlab_radar_geometry* geo, const float* points, int n_points,
                                        const float* elem_pos, int C, const float* tx_pos, const double* tx_amp, int ntx,
                                        double* delays, double* samples) {
    if (!geo || !points || !elem_pos || !tx_pos || !tx_amp || !delays || !samples || n_points < 0 || C < 1 || ntx < 1)
        return report_error(EMLAB_ERR_INVALID, "bad radar delay arguments");
    const RadarTable table = make_table();
    const Triple wt = turns_of(geo->omega), inv = quotient(1.0, geo->sample_dt, 0.0);
    const std::unique_ptr<FF[]> amp(new (std::nothrow) FF[ntx]);
    if (!amp) return report_error(EMLAB_ERR_OOM, "radar: host allocation failed");
    for (int j = 0; j < ntx; ++j) amp[j] = to_ff(tx_amp[j]);
    for (int k = 0; k < n_points; ++k) {
        const F3 p = ld3(points + 3 * (size_t)k);
        const Delay delay = tx_delay(ld3(geo->tx), ld3(geo->axes + 6), p, table.v, wt, {tx_pos, amp.get(), ntx});
        const Record rec = record_of(delay, geo->dt, geo->sample_dt, inv);
        delays[2 * (size_t)k] = delay.t, delays[2 * (size_t)k + 1] = (double)delay.err;
        for (int i = 0; i < C; ++i) {
            const Sample at = sample_at(rec, len(sub(p, ld3(elem_pos + 3 * (size_t)i))));
            double* o = samples + 5 * ((size_t)k * C + i);
            o[0] = at.clear ? 1.0 : 0.0, o[1] = at.m, o[2] = at.f, o[3] = at.below, o[4] = at.above;
        }
    }
    return EMLAB_OK;
}
