// pattern.cu - the far-field pattern sums of a Huygens box (ntff_pattern.comp:45-110,
// ntff_reduce.comp:19-39) on the FP32 pipes.
//
//   N(r) = sum_p J_p e^{+jk r.(p - c)},   L(r) = sum_p M_p e^{+jk r.(p - c)},
// J = n x H w, M = -n x E w over the nodes p of the six faces (w: the trapezoid edge weights).
//
// What bounds it is the arithmetic per (direction, node) pair. A face is a lattice (iu, iv) at a fixed
// height, so the phase is a product of three factors and the sum is
//   e^{jk r_a p_a} sum_iu U(iu) [ sum_iv V(iv) F_q(iu, iv) ],  q = the two tangential components of J, of M.
// Positions are taken from the box centre, so V at the mirror row is the conjugate of V, and a row and its
// mirror need two real factors for their sum S and difference D instead of two complex ones:
//   V F(p) + conj(V) F(-p) = cos S + j sin D.
// That is 8 multiply-adds per pair where the direct sum has 24 and a sine and a cosine; V serves all columns iu
// of a strip and U a whole column. One thread holds two directions and a strip of four columns (64 sums);
// S and D pass through shared memory as pairs of columns, so the products are packed .f32x2 multiply-adds.
// (One direction and eight columns need the same registers but twice the shared loads a multiply-add, and
// those then bound the SM.) V advances from row to row by one complex product and is evaluated anew every
// 32 rows. Strips are grouped into slices; every slice leaves its share of N and L for the reduction.
// The 10550 directions of a console report on 57624 nodes: 2650 us as direct sums, 424 us with both rows of a
// pair multiplied, 236 us folded; 650 directions at 32 frequencies on 224664 nodes: 3671 and 1990 us.
#include <algorithm>

#include "emlab_internal.h"
#include "twiddle.cuh"

namespace emlab {
namespace {

constexpr int kThreads = 128;
constexpr int kDirs = 2;    // directions of a thread
constexpr int kStrip = 4;   // columns iu of a strip
constexpr int kRows = 32;   // rows (with their mirrors) staged at a time: kRows * kStrip = one pair of nodes per thread
constexpr int kRowFloats = 4 * 4 * kStrip + 4;  // [q][S re, S im, D re, D im][column], and padding against bank conflicts

using pair_t = unsigned long long;
__device__ __forceinline__ pair_t pk(float a, float b) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 un(pair_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ void fma2(pair_t& acc, pair_t a, pair_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Surface phasors of node i at frequency f. PhasorSource: the stage-2 running averages of the
// single-frequency monitor (8 float4 per node). DftSource: the far-field DFT sums straight from X
// ([f][c][i] complex FP64), scaled and rounded to FP32, of a box whose first node in X is `first`.
struct PhasorSource {
    const float4* ph;
    __device__ void load(int, int i, float (&e)[3][2], float (&h)[3][2]) const {
        const float4* s2 = ph + 8 * (long long)i + 4;
        const float4 eR = s2[0], eI = s2[1], hR = s2[2], hI = s2[3];
        e[0][0] = eR.x, e[1][0] = eR.y, e[2][0] = eR.z, e[0][1] = eI.x, e[1][1] = eI.y, e[2][1] = eI.z;
        h[0][0] = hR.x, h[1][0] = hR.y, h[2][0] = hR.z, h[0][1] = hI.x, h[1][1] = hI.y, h[2][1] = hI.z;
    }
};
struct DftSource {
    const double* X;
    long long total;
    int first, f0;
    double scale;
    __device__ void load(int f, int i, float (&e)[3][2], float (&h)[3][2]) const {
        const double2* x = reinterpret_cast<const double2*>(X) + (size_t)(f0 + f) * 6 * total + first + i;
        double2 v[6];
#pragma unroll
        for (int c = 0; c < 6; ++c) v[c] = x[(size_t)c * total];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            e[c][0] = (float)(v[c].x * scale), e[c][1] = (float)(v[c].y * scale);
            h[c][0] = (float)(v[3 + c].x * scale), h[c][1] = (float)(v[3 + c].y * scale);
        }
    }
};

// The weighted tangential currents of every node, once for all blocks of directions (converting the
// FP64 sums in each of them would take longer than the products): cur[f][i] = (J_u re, im, J_v re, im),
// (M_u re, im, M_v re, im), and the radiated power of each block of nodes (halved at the end).
constexpr int kNodes = 256;
template <class Src>
__global__ void __launch_bounds__(kNodes) surface_currents_kernel(const int* box, Src src, int points, float4* cur,
                                                                  float* power) {
    __shared__ int sbox[13];
    __shared__ float sP[kNodes];
    const int tid = threadIdx.x, i = blockIdx.x * kNodes + tid, fq = blockIdx.y;
    if (tid < 13) sbox[tid] = box[tid];
    __syncthreads();
    float P = 0.0f;
    if (i < points) {
        int f = 0;
        for (int k = 1; k < 6; ++k)
            if (i >= sbox[6 + k]) f = k;
        const int a = f >> 1, u = a == 0 ? 1 : 0, v = a == 2 ? 1 : 2;
        const int nu1 = sbox[3 + u] - sbox[u] + 1, nv1 = sbox[3 + v] - sbox[v] + 1;
        const int local = i - sbox[6 + f], iu = local % nu1, iv = local / nu1;
        const float sign = (f & 1) ? 1.0f : -1.0f;
        const float w = ((iu == 0 || iu == nu1 - 1) ? 0.5f : 1.0f) * ((iv == 0 || iv == nv1 - 1) ? 0.5f : 1.0f);
        float e[3][2], h[3][2];
        src.load(fq, i, e, h);
        // n x F for n = sign e_a: +-F of the other tangential component (e_a x e_v = e_u for a = 1)
        const float wu = w * sign * (a == 1 ? 1.0f : -1.0f);
        float ju[2], jv[2], mu[2], mv[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float eu = u ? e[1][r] : e[0][r], ev = v == 2 ? e[2][r] : e[1][r];
            const float hu = u ? h[1][r] : h[0][r], hv = v == 2 ? h[2][r] : h[1][r];
            ju[r] = wu * hv, jv[r] = -wu * hu, mu[r] = -wu * ev, mv[r] = wu * eu;
            // (E x H*).n: e_u h_v - e_v h_u, its sign that of (u, v, a)'s order
            P += wu * -(eu * hv - ev * hu);
        }
        float4* o = cur + 2 * ((size_t)fq * points + i);
        o[0] = make_float4(ju[0], ju[1], jv[0], jv[1]);
        o[1] = make_float4(mu[0], mu[1], mv[0], mv[1]);
    }
    sP[tid] = P;
    __syncthreads();
    for (int stride = kNodes / 2; stride > 0; stride >>= 1) {
        if (tid < stride) sP[tid] = sP[tid] + sP[tid + stride];
        __syncthreads();
    }
    if (tid == 0) power[(size_t)fq * gridDim.x + blockIdx.x] = sP[0];
}

// The strips of a box, face by face: ceil(nodes along u / 4) each (u = y on the x faces, x on the others).
__host__ __device__ inline int face_strips(const int* box, int f) {
    const int u = (f >> 1) == 0 ? 1 : 0;
    return (box[3 + u] - box[u] + 1 + kStrip - 1) / kStrip;
}

// The sums of one face with normal axis A over the columns iu0 .. iu0 + 3, added to N and L of both
// directions ([direction][component]{re, im}).
template <int A>
__device__ __forceinline__ void strip_sums(const int* box, const float4* cur, int face, int iu0,
                                           const Turns (&turns)[kDirs][3], float (*sF)[kRows * kRowFloats], int& buf,
                                           float (&N)[kDirs][3][2], float (&L)[kDirs][3][2]) {
    constexpr int U = A == 0 ? 1 : 0, V = A == 2 ? 1 : 2;
    const int nu1 = box[3 + U] - box[U] + 1, nv1 = box[3 + V] - box[V] + 1, base = box[6 + face];
    const int tid = threadIdx.x, cu = tid % kStrip, rv = tid / kStrip;
    const int iu = iu0 + cu;
    // positions from the box centre (half-integers, exact)
    const float pv0 = -0.5f * (float)(nv1 - 1), pu0 = -0.5f * (float)(nu1 - 1);
    const float pa = ((face & 1) ? 0.5f : -0.5f) * (float)(box[3 + A] - box[A]);
    pair_t acc[kDirs][4][2][kStrip / 2];
    float ws[kDirs], wc[kDirs];  // V's step from row to row
#pragma unroll
    for (int t = 0; t < kDirs; ++t) {
        twiddle(turns[t][V], 1.0f, ws[t], wc[t]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < kStrip / 2; ++c) acc[t][q][0][c] = 0, acc[t][q][1][c] = 0;
    }
    const int folded = (nv1 + 1) / 2;
    for (int iv0 = 0; iv0 < folded; iv0 += kRows) {
        const int iv = iv0 + rv, mirror = nv1 - 1 - iv;
        const bool middle = mirror == iv;  // its own mirror: S its fields, D 0
        float4 j4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), m4 = j4, jm = j4, mm = j4;
        if (iu < nu1 && iv < folded) {
            const float4* p = cur + 2 * (size_t)(base + iv * nu1 + iu);
            j4 = __ldg(p), m4 = __ldg(p + 1);
            if (!middle) {
                p = cur + 2 * (size_t)(base + mirror * nu1 + iu);
                jm = __ldg(p), mm = __ldg(p + 1);
            }
        }
        float* row = sF[buf] + rv * kRowFloats + cu;
        auto put = [&](int q, float re, float im, float mre, float mim) {
            row[(4 * q + 0) * kStrip] = re + mre, row[(4 * q + 1) * kStrip] = im + mim;
            row[(4 * q + 2) * kStrip] = middle ? 0.0f : re - mre, row[(4 * q + 3) * kStrip] = middle ? 0.0f : im - mim;
        };
        put(0, j4.x, j4.y, jm.x, jm.y), put(1, j4.z, j4.w, jm.z, jm.w);
        put(2, m4.x, m4.y, mm.x, mm.y), put(3, m4.z, m4.w, mm.z, mm.w);
        float vs[kDirs], vc[kDirs];
#pragma unroll
        for (int t = 0; t < kDirs; ++t) twiddle(turns[t][V], pv0 + (float)iv0, vs[t], vc[t]);
        __syncthreads();  // the other buffer's readers are past it since the last barrier
        const int rows = min(kRows, folded - iv0);
        for (int j = 0; j < rows; ++j) {
            pair_t c2[kDirs], s2[kDirs], m2[kDirs];
#pragma unroll
            for (int t = 0; t < kDirs; ++t) {
                c2[t] = pk(vc[t], vc[t]), s2[t] = pk(vs[t], vs[t]), m2[t] = pk(-vs[t], -vs[t]);
                const float c = fmaf(vc[t], wc[t], -vs[t] * ws[t]);
                vs[t] = fmaf(vs[t], wc[t], vc[t] * ws[t]), vc[t] = c;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const ulonglong2* f = reinterpret_cast<const ulonglong2*>(sF[buf] + j * kRowFloats + 4 * q * kStrip);
                const ulonglong2 sr = f[0], si = f[1], dr = f[2], di = f[3];
#pragma unroll
                for (int t = 0; t < kDirs; ++t) {
                    fma2(acc[t][q][0][0], c2[t], sr.x), fma2(acc[t][q][0][0], m2[t], di.x);
                    fma2(acc[t][q][1][0], c2[t], si.x), fma2(acc[t][q][1][0], s2[t], dr.x);
                    fma2(acc[t][q][0][1], c2[t], sr.y), fma2(acc[t][q][0][1], m2[t], di.y);
                    fma2(acc[t][q][1][1], c2[t], si.y), fma2(acc[t][q][1][1], s2[t], dr.y);
                }
            }
        }
        buf ^= 1;
    }
#pragma unroll
    for (int t = 0; t < kDirs; ++t) {
        // columns, then the plane: columns beyond the face hold zeros
        float g[4][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) g[q][0] = g[q][1] = 0.0f;
#pragma unroll
        for (int u = 0; u < kStrip; ++u) {
            float s, c;
            twiddle(turns[t][U], pu0 + (float)(iu0 + u), s, c);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 re2 = un(acc[t][q][0][u / 2]), im2 = un(acc[t][q][1][u / 2]);
                const float re = u & 1 ? re2.y : re2.x, im = u & 1 ? im2.y : im2.x;
                g[q][0] = fmaf(c, re, fmaf(-s, im, g[q][0]));
                g[q][1] = fmaf(s, re, fmaf(c, im, g[q][1]));
            }
        }
        float s, c;
        twiddle(turns[t][A], pa, s, c);
        auto add = [&](float (&o)[2], const float (&v)[2]) {
            o[0] = fmaf(c, v[0], fmaf(-s, v[1], o[0]));
            o[1] = fmaf(s, v[0], fmaf(c, v[1], o[1]));
        };
        add(N[t][U], g[0]), add(N[t][V], g[1]), add(L[t][U], g[2]), add(L[t][V], g[3]);
    }
}

// 256 directions x one slice of the strips x one frequency per block; partials [f][slice][12][count]
// (N re, N im, L re, L im). Wavenumbers: k[f], or k0 without an array.
constexpr int kBlockDirs = kThreads * kDirs;
__global__ void __launch_bounds__(kThreads, 3) ntff_pattern_kernel(const int* box, const float4* cur, int points,
                                                                   const double* k, double k0, const float4* dirs,
                                                                   int count, int slices, float* partials) {
    __shared__ __align__(16) float sF[2][kRows * kRowFloats];
    __shared__ int sbox[13];
    const int tid = threadIdx.x, slice = blockIdx.y, fq = blockIdx.z;
    if (tid < 13) sbox[tid] = box[tid];
    __syncthreads();
    const double kf = k ? k[fq] : k0;
    Turns turns[kDirs][3];
#pragma unroll
    for (int t = 0; t < kDirs; ++t) {
        const int d = blockIdx.x * kBlockDirs + t * kThreads + tid;
        const float4 r = d < count ? dirs[d] : make_float4(0.0f, 0.0f, 1.0f, 0.0f);
        turns[t][0] = turns_per_cell(kf, r.x), turns[t][1] = turns_per_cell(kf, r.y), turns[t][2] = turns_per_cell(kf, r.z);
    }
    cur += 2 * (size_t)fq * points;
    int strips = 0;
    for (int f = 0; f < 6; ++f) strips += face_strips(sbox, f);
    const int from = (int)((long long)strips * slice / slices), to = (int)((long long)strips * (slice + 1) / slices);
    float N[kDirs][3][2] = {}, L[kDirs][3][2] = {};
    int buf = 0;
    for (int f = 0, first = 0; f < 6; ++f) {
        const int n = face_strips(sbox, f);
        for (int s = max(from, first); s < min(to, first + n); ++s) {
            const int iu0 = (s - first) * kStrip;
            if (f < 2) strip_sums<0>(sbox, cur, f, iu0, turns, sF, buf, N, L);
            else if (f < 4) strip_sums<1>(sbox, cur, f, iu0, turns, sF, buf, N, L);
            else strip_sums<2>(sbox, cur, f, iu0, turns, sF, buf, N, L);
        }
        first += n;
    }
#pragma unroll
    for (int t = 0; t < kDirs; ++t) {
        const int d = blockIdx.x * kBlockDirs + t * kThreads + tid;
        if (d >= count) continue;
        float* o = partials + ((size_t)fq * slices + slice) * 12 * count + d;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            o[(size_t)c * count] = N[t][c][0], o[(size_t)(3 + c) * count] = N[t][c][1];
            o[(size_t)(6 + c) * count] = L[t][c][0], o[(size_t)(9 + c) * count] = L[t][c][1];
        }
    }
}

// ntff_reduce.comp:19-39: out[(f * total + first + d) * 2] = |N_perp - r x L|^2 over both parts; the
// radiated power at the frequency's first direction, 0 at the others. 32 directions per block, four
// warps of slices.
__global__ void __launch_bounds__(128) ntff_reduce_kernel(const float4* dirs, const float* partials, const float* power,
                                                          int n_power, int first, int count, int total, int slices,
                                                          float* out) {
    __shared__ float part[3][12][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, fq = blockIdx.y;
    const int d = blockIdx.x * 32 + lane;
    float v[12];
#pragma unroll
    for (int c = 0; c < 12; ++c) v[c] = 0.0f;
    if (d < count) {
        const float* p = partials + (size_t)fq * slices * 12 * count + d;
#pragma unroll 2
        for (int s = warp; s < slices; s += 4)
#pragma unroll
            for (int c = 0; c < 12; ++c) v[c] += __ldg(p + ((size_t)s * 12 + c) * count);
    }
    float P = 0.0f;
    if (warp == 3 && first + blockIdx.x == 0) {  // the power of the frequency, by one warp
        for (int i = lane; i < n_power; i += 32) P += power[(size_t)fq * n_power + i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) P += __shfl_xor_sync(0xffffffffu, P, o);
        if (lane == 0) out[(size_t)fq * total * 2 + 1] = 0.5f * P;
    }
    if (warp)
#pragma unroll
        for (int c = 0; c < 12; ++c) part[warp - 1][c][lane] = v[c];
    __syncthreads();
    if (warp || d >= count) return;
#pragma unroll
    for (int c = 0; c < 12; ++c) v[c] = (v[c] + part[0][c][lane]) + (part[1][c][lane] + part[2][c][lane]);
    const float4 r = dirs[d];
    const float rv[3] = {r.x, r.y, r.z};
    float F2 = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float *N = v + 3 * h, *L = v + 6 + 3 * h;
        const float dn = N[0] * rv[0] + N[1] * rv[1] + N[2] * rv[2];
        const float F0 = (N[0] - dn * rv[0]) - (rv[1] * L[2] - L[1] * rv[2]);
        const float F1 = (N[1] - dn * rv[1]) - (rv[2] * L[0] - L[2] * rv[0]);
        const float Fz = (N[2] - dn * rv[2]) - (rv[0] * L[1] - L[0] * rv[1]);
        F2 = F2 + (F0 * F0 + F1 * F1 + Fz * Fz);
    }
    float* o = out + ((size_t)fq * total + first + d) * 2;
    o[0] = F2;
    if (first + d) o[1] = 0.0f;
}

int power_blocks(int points) { return (points + kNodes - 1) / kNodes; }

// Frequencies f of nf in groups of plan.freqs (the surface currents of a group fit the scratch),
// directions in groups of plan.chunk.
template <class MakeSrc>
void launch(const int* dbox, int points, int nf, const double* k, double k0, const float4* dirs, int n_dirs,
            const PatternPlan& plan, float* scratch, float* out, cudaStream_t s, MakeSrc&& make) {
    float4* cur = reinterpret_cast<float4*>(scratch);
    float* power = scratch + (size_t)plan.freqs * points * 8;
    float* partials = power + (size_t)plan.freqs * power_blocks(points);
    for (int f0 = 0; f0 < nf; f0 += plan.freqs) {
        const int n = std::min(plan.freqs, nf - f0);
        const auto src = make(f0);
        surface_currents_kernel<<<dim3(power_blocks(points), n), kNodes, 0, s>>>(dbox, src, points, cur, power);
        for (int first = 0; first < n_dirs; first += plan.chunk) {
            const int count = std::min(plan.chunk, n_dirs - first);
            ntff_pattern_kernel<<<dim3((count + kBlockDirs - 1) / kBlockDirs, plan.slices, n), kThreads, 0, s>>>(
                dbox, cur, points, k ? k + f0 : nullptr, k0, dirs + first, count, plan.slices, partials);
            ntff_reduce_kernel<<<dim3((count + 31) / 32, n), 128, 0, s>>>(dirs + first, partials, power,
                                                                         power_blocks(points), first, count, n_dirs,
                                                                         plan.slices, out + (size_t)f0 * n_dirs * 2);
        }
    }
}

}  // namespace

PatternPlan pattern_plan(const int* box, int nf, int n_dirs) {
    PatternPlan p;
    const long long points = box[12];
    int strips = 0;
    for (int f = 0; f < 6; ++f) strips += face_strips(box, f);
    // frequencies whose currents (32 bytes a node) take 256 MB together
    p.freqs = (int)std::clamp<long long>((256ll << 20) / (32 * points), 1, nf);
    // slices: just under four blocks for each that the device holds (three to an SM), so that the last wave is
    // nearly full, but no more than there are strips, and 64 at most (the reduction reads all of them)
    const long long blocks = (long long)((n_dirs + kBlockDirs - 1) / kBlockDirs) * p.freqs;
    p.slices = (int)std::max<long long>(1, std::min<long long>(std::min(strips, 64), 4 * 3 * sm_count() / blocks));
    // directions per launch: all of them unless their partial sums would pass 256 MB
    const long long per_dir = 48ll * p.slices * p.freqs;
    p.chunk = (int)std::max<long long>(kBlockDirs, std::min<long long>(n_dirs, (256ll << 20) / per_dir / kBlockDirs * kBlockDirs));
    const int groups = (nf + p.freqs - 1) / p.freqs;
    p.launches = groups * (1 + 2 * ((n_dirs + p.chunk - 1) / p.chunk));
    p.scratch = (size_t)p.freqs * ((size_t)points * 8 + power_blocks((int)points) +
                                   (size_t)p.slices * 12 * (size_t)std::min(p.chunk, n_dirs));
    return p;
}

void launch_pattern_phasors(const int* dbox, int points, const float* phasors, double k, const float4* dirs, int n_dirs,
                            const PatternPlan& plan, float* scratch, float* out, cudaStream_t s) {
    launch(dbox, points, 1, nullptr, k, dirs, n_dirs, plan, scratch, out, s,
           [&](int) { return PhasorSource{reinterpret_cast<const float4*>(phasors)}; });
}

void launch_pattern_dft(const int* dbox, int points, const double* X, int first, int total_points, int f0, int nf,
                        const double* omega, double scale, const float4* dirs, int n_dirs, const PatternPlan& plan,
                        float* scratch, float* out, cudaStream_t s) {
    launch(dbox, points, nf, omega + f0, 0.0, dirs, n_dirs, plan, scratch, out, s,
           [&](int f) { return DftSource{X, total_points, first, f0 + f, scale}; });
}

}  // namespace emlab
