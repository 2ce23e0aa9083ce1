// radar_pairs.cuh - the radar image's FP64 quantities as pairs of FP32, each with a bound of its error.
//
// Host and device functions: the self-check emlab_debug_radar_delays evaluates on the CPU what the kernel
// (radar.cu) does, operation by operation, so the bounds below are tested against extended precision there.
//
// Notation: u = 2^-24, so u^2 = 2^-48. Errors of the pair operations, relative to the result unless said
// (Joldes, Muller, Popescu, ACM TOMS 44, 2017): pair + float 2 u^2, pair * float 2 u^2, pair * pair 5 u^2, and
// for pair + pair, whose operands may cancel, 3 u^2 of the sum of their magnitudes. A double as a pair: u^2.
#pragma once

#include <cuda_runtime.h>

#include <cmath>

namespace emlab {
namespace radar {

struct F3 {
    float x, y, z;
};
#define EMLAB_HD __host__ __device__ __forceinline__
EMLAB_HD F3 sub(F3 a, F3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
EMLAB_HD F3 add(F3 a, F3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
EMLAB_HD F3 mul(F3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
EMLAB_HD float dot(F3 a, F3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
EMLAB_HD float len(F3 a) { return sqrtf(dot(a, a)); }
EMLAB_HD F3 ld3(const float* p) { return {p[0], p[1], p[2]}; }

// Unevaluated sums hi + lo of two floats (Dekker, Numer. Math. 18, 1971; Knuth, TAOCP 2, 4.2.2).
struct FF {
    float h, l;
};
EMLAB_HD FF to_ff(double v) {
    const float h = (float)v;
    return {h, (float)(v - (double)h)};
}
EMLAB_HD double to_f64(FF a) { return (double)a.h + (double)a.l; }
EMLAB_HD FF fast_sum(float a, float b) {  // |a| >= |b|
    const float s = a + b;
    return {s, b - (s - a)};
}
EMLAB_HD FF two_sum(float a, float b) {
    const float s = a + b, t = s - a;
    return {s, (a - (s - t)) + (b - t)};
}
EMLAB_HD FF operator+(FF a, FF b) {
    const FF s = two_sum(a.h, b.h);
    return fast_sum(s.h, s.l + (a.l + b.l));
}
EMLAB_HD FF operator-(FF a) { return {-a.h, -a.l}; }
EMLAB_HD FF operator*(FF a, FF b) {
    const float p = a.h * b.h;
    return fast_sum(p, fmaf(a.l, b.h, fmaf(a.h, b.l, fmaf(a.h, b.h, -p))));
}
EMLAB_HD FF operator*(FF a, float b) {
    const float p = a.h * b;
    return fast_sum(p, fmaf(a.l, b, fmaf(a.h, b, -p)));
}

// A quotient to 70 bits and more as the sum of three floats: a / b for b = bh + bl, from the double quotient and
// what it leaves.
struct Triple {
    float h, m, l;
};
inline Triple quotient(double a, double bh, double bl) {
    const double q = a / bh, rest = (std::fma(-q, bh, a) - q * bl) / bh;
    const FF f = to_ff(q);
    return {f.h, f.l, (float)(q - (double)f.h - (double)f.l + rest)};
}

// e^{j w d}, d >= 0 in FP32, from wt = w / 2 pi in turns per unit: the turns are reduced to the nearest
// table entry (exactly: the products with d are kept in full), the rest r, |r| <= pi / 512, enters through
// sin r = r - r^3/6 + r^5/120 and cos r = 1 - r^2/2 + r^4/24 (truncation below 1e-16). Both parts are within
// 7 u^2: r^3/6 rounded 2.6 u^2, the last addition 3 u^2, the table 1 u^2, the rest below u^2 / 2.
constexpr int kTable = 512;
constexpr float kTurns = 4096.0f;  // the rest e below stays under 2^-12 of a turn
struct Phase {
    FF c, s;
};
EMLAB_HD Phase phase(const float4* table, Triple wt, float d) {
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

struct RadarTable {
    float4 v[kTable];  // cos, sin of 2 pi k / kTable, each as a pair
};
inline RadarTable make_table() {
    RadarTable t;
    for (int k = 0; k < kTable; ++k) {
        const double a = 6.28318530717958647692 * k / kTable;
        const FF c = to_ff(std::cos(a)), s = to_ff(std::sin(a));
        t.v[k] = make_float4(c.h, c.l, s.h, s.l);
    }
    return t;
}
inline Triple turns_of(double omega) { return quotient(omega, 6.28318530717958647692, 2.4492935982947064e-16); }  // w / 2 pi

// Sums whose squares and low parts stay normal numbers; false for a NaN.
EMLAB_HD bool in_range(float v) { return v > 1e-18f && v < 1e18f; }

struct Delay {
    double t;
    float err;  // bound of the difference from the FP64 sums; negative: to be formed in FP64
};

// RadarMonitor::txDelay (Radar.cpp:87-103): t = d0 + Re(D / A), A = sum a_j e_j and D = sum a_j e_j (d_j - d0) over
// the elements, a_j = amp_j g_j / d_j^2 and e_j the phase of d_j, d0 the array centre's distance.
//
// The bound. An error of A and of D moves t by at most (|dD| + |D / A| |dA|) / |A|.
//  - Here: a_j is within 17 u^2 (1 / d 2, its square 9, amp 15, g 17), e_j within 7 u^2, the product 5 u^2: both parts
//    together 32 u^2 |a_j|, times d_j - d0 (exact) 37 u^2. An addition costs 3 u^2 of the running sum and the term.
//    With ma, md the sums of |a_j|, |a_j (d_j - d0)|, and ra, rd those of the running sums' parts,
//    dA <= u^2 (37 ma + 3 ra) and dD <= u^2 (42 md + 3 rd).
//  - In FP64 (v = 2^-53): a term's own roundings (9 v), and that of w d (v times its radians), move it in A and D
//    alike, by (9 + 2 pi turns) v sum |a_j (d_j - t)| <= .. (md + |D / A| ma); the products with d_j 1.5 v far ma, the
//    additions v ra and v (d0 ra + rd), the quotient 7 v of it; 7 v more for the last line here.
// The constants below are those, rounded up; float evaluation of the bound itself is in the last factor.
struct Transmit {
    const float* pos;  // n x 3
    const FF* amp;
    int n;
};
EMLAB_HD Delay tx_delay(F3 tx, F3 boresight, F3 p, const float4* table, Triple wt, const Transmit& in) {
    FF ar = {0, 0}, ai = ar, adr = ar, adi = ar, mag = ar;
    const float d0 = len(sub(p, tx));
    float far = 0.0f, ma = 0.0f, md = 0.0f, ra = 0.0f, rd = 0.0f;
    for (int j = 0; j < in.n; ++j) {
        const F3 v = sub(p, ld3(in.pos + 3 * j));
        const float d = fmaxf(len(v), 0.5f);
        const float q = 1.0f / d;
        const FF inv = {q, q * fmaf(-q, d, 1.0f)};
        const FF a = (in.amp[j] * (inv * inv)) * fmaxf(dot(v, boresight), 0.0f);  // amp (g / d) / d
        const Phase e = phase(table, wt, d);
        const FF tr = a * e.c, ti = a * e.s;  // the conjugate of a e^{-j w d}
        const FF dd = two_sum(d, -d0);
        ar = ar + tr, ai = ai + ti;
        adr = adr + tr * dd, adi = adi + ti * dd;
        mag = mag + a;
        far = fmaxf(far, d);
        ma += fabsf(a.h), md += fabsf(a.h * dd.h);
        ra += fabsf(ar.h) + fabsf(ai.h), rd += fabsf(adr.h) + fabsf(adi.h);
    }
    // beyond 2^30 the low parts of 1 / d^2 may leave the normal numbers
    if (!in_range(mag.h) || !in_range(fmaxf(fabsf(ar.h), fabsf(ai.h))) || !(fabsf(wt.h) * far < kTurns) || !(far < 0x1p30f))
        return {0.0, -1.0f};
    const double r = to_f64(ar), i = to_f64(ai);
    // real(ad / a); a single element's is 0, which an FP64 division takes several times as long for
    const double num = to_f64(adr) * r + to_f64(adi) * i, t = (double)d0 + (num == 0.0 ? 0.0 : num / (r * r + i * i));
    const float over = 1.0f / sqrtf(ar.h * ar.h + ai.h * ai.h), turns = fabsf(wt.h) * far;
    const float rest = sqrtf(adr.h * adr.h + adi.h * adi.h) * over;
    const float pairs = over * (42.0f * md + 3.0f * rd + rest * (37.0f * ma + 3.0f * ra));
    const float own = over * ((9.0f + 6.3f * turns) * (md + rest * ma) + 1.5f * far * ma + 2.0f * (d0 + rest) * ra + rd) +
                      16.0f * (d0 + rest);
    // cancellation beyond 100 goes to FP64 (at 1000 the reference takes the centre's distance)
    return {t, mag.h * over < 100.0f && fabs(t) < 1e18 ? 1.01f * (0x1p-48f * pairs + 0x1p-53f * own) : -1.0f};
}

// Positions in the record: s = (t + d + dt / 2) / sdt decimated samples for an element at distance d, as an integer
// m and the interpolation weight f of sample m + 1, rounded to FP32 as the reference rounds it.
struct Record {
    int n0;        // the point's own part, n0 + f0 with f0 in [1/2, 3/2): the whole position stays positive
    FF f0;
    Triple inv;    // 1 / sdt
    float reach0;  // |t + dt / 2| / |sdt|, rounded up
    float err;     // of the delay, in samples; infinite where positions cannot be held
};
EMLAB_HD Record record_of(Delay delay, double dt, double sdt, Triple inv) {
    const double s = (delay.t + 0.5 * dt) / sdt, n = floor(s - 0.5);
    const float ainv = fabsf(inv.h);
    if (!(fabs(s) < 1e9) || delay.err < 0.0f) return {0, {1.0f, 0.0f}, inv, 0.0f, INFINITY};
    return {(int)n, to_ff(s - n), inv, 1.0001f * (fabsf((float)delay.t) + fabsf((float)dt)) * ainv, 1.0001f * delay.err * ainv};
}
struct Sample {
    int m;
    float f;
    float below, above;  // f rounded from the ends of the interval that holds the FP64 position
    bool clear;          // m is certain
};
// d / sdt = p + e + q + .. with p, q products rounded and e what p dropped, exactly; the whole turns of p leave it
// exactly too, and three exact sums gather the rest. What is not exact: f0 as a pair (1.5 u^2), the four
// additions of low parts (2^-48, 2^-47, 2^-47.4, 2^-46.2: their magnitudes are below 2^-24 .. 2^-22), the last sum
// where c.h is smaller than they (2^-46), the ends of the interval, together below 2^-44; and FP64's roundings,
// 3 in the reference's position and 2 in s, each 2^-53 of the reach: 2^-50 is more than that.
EMLAB_HD Sample sample_at(const Record& r, float d) {
    const float p = r.inv.h * d, q = r.inv.m * d;
    const float n1 = rintf(p);
    const float low = fmaf(r.inv.l, d, fmaf(r.inv.m, d, -q));
    const FF a = two_sum(p - n1, fmaf(r.inv.h, d, -p)), b = two_sum(a.h, q), c = two_sum(b.h, r.f0.h);
    const FF s = fast_sum(c.h, ((a.l + b.l) + c.l) + (r.f0.l + low));
    float m = floorf(s.h);
    if (m == s.h && s.l < 0.0f) m -= 1.0f;
    const float part = s.h - m;  // exact for m >= 0
    const float eps = r.err + fmaf(0x1p-50f, fabsf(p) + r.reach0, 0x1p-44f);
    Sample o;
    o.f = part + s.l, o.below = part + (s.l - eps), o.above = part + (s.l + eps);
    o.clear = m >= 0.0f && o.above < 1.0f && o.below >= 0.0f && fabsf(p) < 0x1p22f;
    o.m = o.clear ? r.n0 + (int)n1 + (int)m : -1;
    return o;
}

// By how much z0 (1 - f) + z1 f in FP32 varies for f from below to above: every operation is monotonic, so each
// product lies between its values at the ends, and the sum between those of the smaller and of the larger ones.
// Most weights that are not certain are small ones, whose units in the last place are too: there it is 0.
EMLAB_HD float interpolation_range(float z0, float z1, const Sample& s) {
    const float a0 = z0 * (1.0f - s.below), a1 = z0 * (1.0f - s.above), b0 = z1 * s.below, b1 = z1 * s.above;
    return (fmaxf(a0, a1) + fmaxf(b0, b1)) - (fminf(a0, a1) + fminf(b0, b1));
}

// Whether every weight can be held as a pair without losing its low part.
inline bool pairs_hold(const double* w, int n) {
    for (int i = 0; i < n; ++i)
        if (w[i] != 0.0 && !(std::fabs(w[i]) >= 0x1p-100 && std::fabs(w[i]) <= 0x1p100)) return false;
    return true;
}
#undef EMLAB_HD

}  // namespace radar
}  // namespace emlab
