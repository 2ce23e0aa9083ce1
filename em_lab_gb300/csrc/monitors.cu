// monitors.cu - per-step and on-demand monitor kernels on sm_103a.
//
// Each kernel restates one reference shader (file:line on each) and, like the solver, is compiled
// with -fmad=false so its per-step FP32 arithmetic matches the CPU restatement bit for bit.
// Monitors read the field generation that the step just produced.
#include "emlab_internal.h"

namespace emlab {

namespace {

__host__ __device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }

__device__ __forceinline__ long long cidx(const MonitorArgs& m, int x, int y, int z) {
    x = clampi(x, 0, m.nx - 1), y = clampi(y, 0, m.ny - 1), z = clampi(z, 0, m.nz - 1);
    return (long long)z * m.plane + (long long)y * m.pitch + x;
}

__device__ __forceinline__ const float* ecomp(const MonitorArgs& m, int c) { return c == 0 ? m.ex : (c == 1 ? m.ey : m.ez); }
__device__ __forceinline__ const float* bcomp(const MonitorArgs& m, int c) { return c == 0 ? m.bx : (c == 1 ? m.by : m.bz); }

// field_sampling.glsl:17-23 (clamp-to-edge fetches)
__device__ __forceinline__ void e_at_node(const MonitorArgs& m, int x, int y, int z, float& ex, float& ey, float& ez) {
    ex = 0.5f * (m.ex[cidx(m, x, y, z)] + m.ex[cidx(m, x - 1, y, z)]);
    ey = 0.5f * (m.ey[cidx(m, x, y, z)] + m.ey[cidx(m, x, y - 1, z)]);
    ez = 0.5f * (m.ez[cidx(m, x, y, z)] + m.ez[cidx(m, x, y, z - 1)]);
}

// field_sampling.glsl:25-32
__device__ __forceinline__ void b_at_node(const MonitorArgs& m, int x, int y, int z, float& bx, float& by, float& bz) {
    const float sx = m.bx[cidx(m, x, y, z)] + m.bx[cidx(m, x, y - 1, z)] + m.bx[cidx(m, x, y, z - 1)] +
                     m.bx[cidx(m, x, y - 1, z - 1)];
    const float sy = m.by[cidx(m, x, y, z)] + m.by[cidx(m, x - 1, y, z)] + m.by[cidx(m, x, y, z - 1)] +
                     m.by[cidx(m, x - 1, y, z - 1)];
    const float sz = m.bz[cidx(m, x, y, z)] + m.bz[cidx(m, x - 1, y, z)] + m.bz[cidx(m, x, y - 1, z)] +
                     m.bz[cidx(m, x - 1, y - 1, z)];
    bx = 0.25f * sx, by = 0.25f * sy, bz = 0.25f * sz;
}

// port_accumulate.comp:46-50
__device__ __forceinline__ float edge_current(const MonitorArgs& m, int x, int y, int z, int a) {
    const int u = (a + 1) % 3, v = (a + 2) % 3;
    int pu[3] = {x, y, z}, pv[3] = {x, y, z};
    pu[u] -= 1, pv[v] -= 1;
    const float b0v = bcomp(m, v)[cidx(m, x, y, z)], b0u = bcomp(m, u)[cidx(m, x, y, z)];
    const float buv = bcomp(m, v)[cidx(m, pu[0], pu[1], pu[2])];
    const float bvu = bcomp(m, u)[cidx(m, pv[0], pv[1], pv[2])];
    return (b0v - buv) - (b0u - bvu);
}

// port_accumulate.comp:52-83
__global__ void ports_kernel(MonitorArgs m, const int4* ports, int n, float* ph, float* series, long long rec,
                             const float4* rot, const float* blend, int k) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int4 p = ports[2 * i], info = ports[2 * i + 1];
    const float4 r = __ldcg(rot + k);
    const float b = __ldcg(blend + k);
    float* q = ph + 8 * i;
    float4 s1 = __ldcg(reinterpret_cast<const float4*>(q)), s2 = __ldcg(reinterpret_cast<const float4*>(q) + 1);
    chain_wait();
    chain_next();
    const int a = p.w;
    const float s = (float)info.y;
    float V = 0.0f, I = 0.0f;
    if (info.x == 4) {
        int eu[3] = {0, 0, 0}, ev[3] = {0, 0, 0};
        eu[(a + 1) % 3] = 1, ev[(a + 2) % 3] = 1;
        for (int q = 0; q < 4; ++q) {
            const int ox = (q & 1 ? eu[0] : 0) + (q & 2 ? ev[0] : 0);
            const int oy = (q & 1 ? eu[1] : 0) + (q & 2 ? ev[1] : 0);
            const int oz = (q & 1 ? eu[2] : 0) + (q & 2 ? ev[2] : 0);
            V = V + 0.25f * ecomp(m, a)[cidx(m, p.x + ox, p.y + oy, p.z + oz)];
            I = I + edge_current(m, p.x + ox, p.y + oy, p.z + oz, a);
        }
    } else {
        V = ecomp(m, a)[cidx(m, p.x, p.y, p.z)];
        I = edge_current(m, p.x, p.y, p.z, a);
    }
    V = V * s;
    I = I * s;
    if (rec >= 0) {
        series[(rec * n + i) * 2 + 0] = V;
        series[(rec * n + i) * 2 + 1] = I;
    }
    const float o0 = (2.0f * r.x) * V, o1 = (-2.0f * r.y) * V, o2 = (2.0f * r.z) * I, o3 = (-2.0f * r.w) * I;
    s1.x = s1.x + b * (o0 - s1.x);
    s1.y = s1.y + b * (o1 - s1.y);
    s1.z = s1.z + b * (o2 - s1.z);
    s1.w = s1.w + b * (o3 - s1.w);
    s2.x = s2.x + b * (s1.x - s2.x);
    s2.y = s2.y + b * (s1.y - s2.y);
    s2.z = s2.z + b * (s1.z - s2.z);
    s2.w = s2.w + b * (s1.w - s2.w);
    reinterpret_cast<float4*>(q)[0] = s1, reinterpret_cast<float4*>(q)[1] = s2;
}

// ntff_common.glsl:30-53; box = (min xyz, max xyz, face offsets[7])
__device__ __forceinline__ void ntff_point(const int* box, int index, int node[3], float n[3], float& w) {
    int f = 0;
    for (int i = 1; i < 6; ++i)
        if (index >= box[6 + i]) f = i;
    const int a = f >> 1, side = f & 1;
    const int u = a == 0 ? 1 : 0, v = a == 2 ? 1 : 2;
    const int nu = box[3 + u] - box[u], nv = box[3 + v] - box[v];
    const int local = index - box[6 + f];
    const int iu = local % (nu + 1), iv = local / (nu + 1);
    node[0] = box[0], node[1] = box[1], node[2] = box[2];
    node[a] = side == 1 ? box[3 + a] : box[a];
    node[u] = box[u] + iu;
    node[v] = box[v] + iv;
    w = ((iu == 0 || iu == nu) ? 0.5f : 1.0f) * ((iv == 0 || iv == nv) ? 0.5f : 1.0f);
    n[0] = n[1] = n[2] = 0.0f;
    n[a] = side == 1 ? 1.0f : -1.0f;
}

// E and H of consecutive surface nodes, one a lane of a full warp (live: the lane has one; xface: it lies on a
// face of constant x; first: the first node of a row of its face, whose neighbour in y is not the lane
// before). On the x faces consecutive nodes lie rows apart, so every load is a sector a lane and the
// kernels wait for their number: nine of them here instead of eighteen (the values one row back come from
// the lane before, x and x - 1 are one load where they share eight bytes). The same sums as above. A step of
// 128 x 128 x 128 cells with the per-step accumulation 37.5 us before, 36.8 here; of 80 x 80 x 647 cells with
// the surface DFT 91.6 and 90.0; on large grids DRAM bounds the x faces either way.
__device__ __forceinline__ float2 at_x_pair(const float* f, const MonitorArgs& m, int x, int y, int z) {  // (x - 1, x)
    const long long i = cidx(m, x, y, z), j = cidx(m, x - 1, y, z);
    if ((i & 1) && j == i - 1) return *reinterpret_cast<const float2*>(f + j);
    return make_float2(f[j], f[i]);
}
__device__ __forceinline__ void surface_fields(const MonitorArgs& m, bool live, bool xface, bool first, const int p[3],
                                               float E[3], float H[3]) {
    const unsigned all = 0xffffffffu;
    const int x = p[0], y = p[1], z = p[2];
    if (__any_sync(all, live && xface)) {
        float2 ex{}, by{}, bym{}, bz{}, bzy{};
        float ey = 0.0f, bx = 0.0f, bxm = 0.0f, ez = 0.0f, ezm = 0.0f;
        if (live && xface) {
            ex = at_x_pair(m.ex, m, x, y, z), by = at_x_pair(m.by, m, x, y, z), bym = at_x_pair(m.by, m, x, y, z - 1);
            bz = at_x_pair(m.bz, m, x, y, z);
            ey = m.ey[cidx(m, x, y, z)], ez = m.ez[cidx(m, x, y, z)], ezm = m.ez[cidx(m, x, y, z - 1)];
            bx = m.bx[cidx(m, x, y, z)], bxm = m.bx[cidx(m, x, y, z - 1)];
        }
        float eyy = __shfl_up_sync(all, ey, 1), bxy = __shfl_up_sync(all, bx, 1), bxmy = __shfl_up_sync(all, bxm, 1);
        bzy.x = __shfl_up_sync(all, bz.x, 1), bzy.y = __shfl_up_sync(all, bz.y, 1);
        if (live && xface) {
            if (first || threadIdx.x % 32 == 0) {
                eyy = m.ey[cidx(m, x, y - 1, z)], bxy = m.bx[cidx(m, x, y - 1, z)], bxmy = m.bx[cidx(m, x, y - 1, z - 1)];
                bzy = at_x_pair(m.bz, m, x, y - 1, z);
            }
            E[0] = 0.5f * (ex.y + ex.x), E[1] = 0.5f * (ey + eyy), E[2] = 0.5f * (ez + ezm);
            H[0] = 0.25f * (bx + bxy + bxm + bxmy);
            H[1] = 0.25f * (by.y + by.x + bym.y + bym.x);
            H[2] = 0.25f * (bz.y + bz.x + bzy.y + bzy.x);
        }
    }
    if (live && !xface) {
        e_at_node(m, x, y, z, E[0], E[1], E[2]);
        b_at_node(m, x, y, z, H[0], H[1], H[2]);
    }
}

// ntff_accumulate.comp:30-52: 32 floats per point (stage1 eRe, eIm, hRe, hIm, stage2 ...). The
// block's 128 x 128 B of state move between HBM and shared memory as one contiguous chunk
// (consecutive threads, consecutive float4s), rows padded to 9 float4s against bank conflicts;
// each thread then updates its own point there. The state is read ahead of the wait (this kernel's
// own stores of the step before), the 18 field values of a node in one round trip after it. Same
// arithmetic per point.
constexpr int kNtffThreads = 128;
__global__ void __launch_bounds__(kNtffThreads) ntff_kernel(MonitorArgs m, const int* box, int points, float4* ph,
                                                            const float4* rot, const float* blend, int k) {
    __shared__ int sbox[13];
    __shared__ float4 st[kNtffThreads * 9];
    if (threadIdx.x < 13) sbox[threadIdx.x] = box[threadIdx.x];
    const int first = blockIdx.x * kNtffThreads;
    const int count = min(kNtffThreads, points - first);
    float4* base = ph + 8 * (long long)first;
    float4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = threadIdx.x + q * kNtffThreads;
        if (j < 8 * count) v[q] = __ldcg(base + j);
    }
    __syncthreads();  // sbox
    const int i = first + threadIdx.x;
    const bool live = i < points;
    float E[3], Hh[3];
    int node[3] = {0, 0, 0};
    float n[3] = {0.0f, 0.0f, 0.0f}, w;
    if (live) ntff_point(sbox, i, node, n, w);
    const float4 r = __ldcg(rot + k);
    const float b = __ldcg(blend + k);
    chain_wait();
    surface_fields(m, live, n[0] != 0.0f, node[1] == sbox[1], node, E, Hh);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = threadIdx.x + q * kNtffThreads;
        if (j < 8 * count) st[9 * (j >> 3) + (j & 7)] = v[q];
    }
    __syncthreads();
    if (live) {
        float4* p = st + 9 * threadIdx.x;
        float4 s1[4] = {p[0], p[1], p[2], p[3]}, s2[4] = {p[4], p[5], p[6], p[7]};
        const float f[4] = {2.0f * r.x, -2.0f * r.y, 2.0f * r.z, -2.0f * r.w};
        for (int q = 0; q < 4; ++q) {
            const float* src = q < 2 ? E : Hh;
            s1[q].x = s1[q].x + b * (f[q] * src[0] - s1[q].x);
            s1[q].y = s1[q].y + b * (f[q] * src[1] - s1[q].y);
            s1[q].z = s1[q].z + b * (f[q] * src[2] - s1[q].z);
        }
        for (int q = 0; q < 4; ++q) {
            s2[q].x = s2[q].x + b * (s1[q].x - s2[q].x);
            s2[q].y = s2[q].y + b * (s1[q].y - s2[q].y);
            s2[q].z = s2[q].z + b * (s1[q].z - s2[q].z);
        }
        for (int q = 0; q < 4; ++q) p[q] = s1[q], p[4 + q] = s2[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = threadIdx.x + q * kNtffThreads;
        if (j < 8 * count) base[j] = st[9 * (j >> 3) + (j & 7)];
    }
}

// line_accumulate.comp:30-48
__global__ void lines_kernel(MonitorArgs m, const int4* qs, int nq, const int4* terms, const float* weights, float4* ph,
                             float* now, const float4* rot, const float* blend, int k) {
    const int qi = blockIdx.x * blockDim.x + threadIdx.x;
    chain_wait();
    chain_next();
    if (qi >= nq) return;
    const int4 info = qs[qi];
    float sum = 0.0f;
    for (int t = info.x; t < info.x + info.y; ++t) {
        const int4 tt = terms[t];
        const long long j = cidx(m, tt.x, tt.y, tt.z);
        const float f = tt.w < 3 ? ecomp(m, tt.w % 3)[j] : bcomp(m, tt.w % 3)[j];
        sum = sum + weights[t] * f;
    }
    now[qi] = sum;
    const float4 r = rot[k];
    const float b = blend[k];
    const float r0 = info.z == 0 ? r.x : r.z, r1 = info.z == 0 ? r.y : r.w;
    const float o0 = (2.0f * sum) * r0, o1 = (2.0f * sum) * -r1;
    float4 p = ph[qi];
    p.x = p.x + b * (o0 - p.x);
    p.y = p.y + b * (o1 - p.y);
    p.z = p.z + b * (p.x - p.z);
    p.w = p.w + b * (p.y - p.w);
    ph[qi] = p;
}

// probe_gather.comp:20-26 (alpha channels are filled on the host)
__global__ void probe_kernel(MonitorArgs m, const int4* origins, int n, float4* out) {
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= n * 54) return;
    const int probe = id / 54, k = id % 54, t = k % 27;
    const int4 o = origins[probe];
    const long long j = cidx(m, o.x + t % 3, o.y + (t / 3) % 3, o.z + t / 9);
    out[id] = k < 27 ? make_float4(m.ex[j], m.ey[j], m.ez[j], 0.0f) : make_float4(m.bx[j], m.by[j], m.bz[j], 0.0f);
}

// poynting_flux.comp:32-63: one partial per 16x16 workgroup, tree reduction in the shader's order. The
// workgroups of up to kFluxPlanes planes in one launch (a box's six planes of 16 x 16 nodes are six
// workgroups: launches, not work, bounded them one plane at a time).
constexpr int kFluxPlanes = 16;
struct FluxList {
    FluxRect r[kFluxPlanes];
    int n;
};
__global__ void __launch_bounds__(256) flux_kernel(MonitorArgs m, const __grid_constant__ FluxList list,
                                                   float* partials) {
    __shared__ float sp[256];
    int q = 0, group = blockIdx.x;
    while (group >= list.r[q].groups) group -= list.r[q++].groups;
    const int axis = list.r[q].axis, index = list.r[q].index, rmin0 = list.r[q].m0, rmin1 = list.r[q].m1;
    const int rs0 = list.r[q].r0, rs1 = list.r[q].r1, across = (rs0 + 15) / 16;
    const int lu = group % across * 16 + threadIdx.x, lv = group / across * 16 + threadIdx.y;
    const int lid = threadIdx.y * 16 + threadIdx.x;
    float flux = 0.0f;
    if (lu < rs0 && lv < rs1) {
        const int u = rmin0 + lu, v = rmin1 + lv;
        int p[3];
        if (axis == 0) p[0] = index, p[1] = u, p[2] = v;
        else if (axis == 1) p[0] = u, p[1] = index, p[2] = v;
        else p[0] = u, p[1] = v, p[2] = index;
        if (p[0] >= 0 && p[1] >= 0 && p[2] >= 0 && p[0] < m.nx && p[1] < m.ny && p[2] < m.nz) {
            float E[3], Bn[3];
            e_at_node(m, p[0], p[1], p[2], E[0], E[1], E[2]);
            b_at_node(m, p[0], p[1], p[2], Bn[0], Bn[1], Bn[2]);
            const float S0 = E[1] * Bn[2] - Bn[1] * E[2];
            const float S1 = E[2] * Bn[0] - Bn[2] * E[0];
            const float S2 = E[0] * Bn[1] - Bn[0] * E[1];
            flux = axis == 0 ? S0 : (axis == 1 ? S1 : S2);
        }
    }
    sp[lid] = flux;
    __syncthreads();
    for (int stride = 128; stride > 0; stride >>= 1) {
        if (lid < stride) sp[lid] = sp[lid] + sp[lid + stride];
        __syncthreads();
    }
    if (lid == 0) partials[list.r[q].first + group] = sp[0];
}

// PortMonitor::evaluateSweep sums (Ports.cpp:215-242) in FP64: one block per (port, frequency)
__global__ void __launch_bounds__(256) sweep_kernel(const float* series, long long steps, int nports, double nu_lo,
                                                    double nu_hi, int points, double dt, double* out) {
    const int pf = blockIdx.x;
    const int p = pf / points, f = pf % points;
    const double nu = nu_lo + (nu_hi - nu_lo) * f / (points - 1);
    const double w = 6.283185307179586476925 * nu;
    double acc[4] = {0, 0, 0, 0};
    for (long long k = threadIdx.x; k < steps; k += blockDim.x) {
        double s, c;
        sincos(-w * dt * (double)k, &s, &c);
        const double V = (double)series[(k * nports + p) * 2], I = (double)series[(k * nports + p) * 2 + 1];
        acc[0] += V * c, acc[1] += V * s, acc[2] += I * c, acc[3] += I * s;
    }
    __shared__ double red[4][256];
    for (int q = 0; q < 4; ++q) red[q][threadIdx.x] = acc[q];
    __syncthreads();
    for (int stride = blockDim.x / 2; stride > 0; stride >>= 1) {
        if (threadIdx.x < stride)
            for (int q = 0; q < 4; ++q) red[q][threadIdx.x] += red[q][threadIdx.x + stride];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        double sh, ch;
        sincos(w * 0.5 * dt, &sh, &ch);
        double* o = out + (long long)pf * 4;
        o[0] = red[0][0], o[1] = red[1][0];
        o[2] = red[2][0] * ch - red[3][0] * sh, o[3] = red[2][0] * sh + red[3][0] * ch;
    }
}

__global__ void finite_kernel(MonitorArgs m, unsigned* flag) {
    const long long total = (long long)m.nz * m.plane;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(i % m.pitch);
        if (x >= m.nx) continue;
        if (!isfinite(m.ex[i]) || !isfinite(m.ey[i]) || !isfinite(m.ez[i]) || !isfinite(m.bx[i]) ||
            !isfinite(m.by[i]) || !isfinite(m.bz[i])) {
            atomicOr(flag, 1u);
            return;
        }
    }
}

// Multi-frequency far-field DFT, per step: the co-located E and H (field_sampling.glsl:17-32) of
// every Huygens-box node into slot t of the time block, component-major: blk[(t * 6 + c) * P + i],
// P the points of all boxes, i = the box's first point + the node's index in its box. blockIdx.y is
// the box.
__global__ void __launch_bounds__(256) dft_sample_kernel(MonitorArgs m, const int* boxes, int points, float* blk,
                                                         int t) {
    __shared__ int sbox[kDftBoxInts];
    chain_next();  // the last kernel of a step: the next solver pass may come in
    if (threadIdx.x < kDftBoxInts) sbox[threadIdx.x] = boxes[(size_t)blockIdx.y * kDftBoxInts + threadIdx.x];
    __syncthreads();
    const int local = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = local < sbox[14];
    const int i = sbox[13] + local;
    int node[3] = {0, 0, 0};
    float n[3] = {0.0f, 0.0f, 0.0f}, w;
    if (live) ntff_point(sbox, local, node, n, w);
    chain_wait();
    float E[3], Hh[3];
    surface_fields(m, live, n[0] != 0.0f, node[1] == sbox[1], node, E, Hh);
    if (!live) return;
    float* o = blk + (size_t)t * 6 * points + i;
    o[0] = E[0], o[(size_t)points] = E[1], o[2 * (size_t)points] = E[2];
    o[3 * (size_t)points] = Hh[0], o[4 * (size_t)points] = Hh[1], o[5 * (size_t)points] = Hh[2];
}

// Folds T samples of every column (component c of node i) into the FP64 sums:
//   X_f += e^{-i w_f t0} sum_k F(t0 + k dt) e^{-i w_f k dt},
// t0 = n0 dt for E and (n0 - 1/2) dt for H (B lags half a step). The block-relative twiddles
// W[f][k] = (cos w_f k dt, -sin w_f k dt) are FP32 (from FP64 on the host); the in-block sums are
// FP32 (<= 64 terms); the block phase e^{-i w_f t0} is evaluated in FP64 once per CTA and applied in
// FP32; the accumulation is FP64. X layout: [f][c][i][re, im]. The CUDA-core twin of the
// tensor-core fold (dft_tc.cu), which differs only in how the in-block sums are formed.
constexpr int kDftMaxT = 64;
__global__ void __launch_bounds__(128) dft_fold_kernel(const float* blk, int T, int points, int nf, const float2* W,
                                                       const double* omega, long long n0, double dt, double* X) {
    extern __shared__ float2 sW[];  // [nf][kDftMaxT], then the block phases [nf][E, H]
    float2* rot = sW + nf * kDftMaxT;
    for (int j = threadIdx.x; j < nf * kDftMaxT; j += blockDim.x) sW[j] = W[j];
    for (int j = threadIdx.x; j < 2 * nf; j += blockDim.x) {
        const double t0 = ((double)n0 - ((j & 1) ? 0.5 : 0.0)) * dt;
        double sn, cs;
        sincos(omega[j >> 1] * t0, &sn, &cs);
        rot[j] = make_float2((float)cs, (float)sn);
    }
    __syncthreads();
    const long long col = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (col >= 6ll * points) return;
    const int c = (int)(col / points), i = (int)(col % points), h = c >= 3 ? 1 : 0;
    float v[kDftMaxT];
#pragma unroll
    for (int k = 0; k < kDftMaxT; ++k) v[k] = k < T ? blk[(size_t)k * 6 * points + col] : 0.0f;
    double2* xo = reinterpret_cast<double2*>(X) + (size_t)c * points + i;  // + f * 6 * points
    const size_t fstride = (size_t)6 * points;
    constexpr int G = 4;  // frequencies per group: their X loads are issued before any store
    for (int f0 = 0; f0 < nf; f0 += G) {
        double2 acc[G];
#pragma unroll
        for (int g = 0; g < G; ++g)
            if (f0 + g < nf) acc[g] = xo[(size_t)(f0 + g) * fstride];
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const int f = f0 + g;
            if (f >= nf) break;
            float re = 0.0f, im = 0.0f;
#pragma unroll
            for (int k = 0; k < kDftMaxT; ++k) {
                const float2 w = sW[f * kDftMaxT + k];
                re = re + w.x * v[k];
                im = im + w.y * v[k];
            }
            const float2 r = rot[2 * f + h];
            const float xr = re * r.x + im * r.y, xi = im * r.x - re * r.y;  // (re + i im)(cos - i sin)
            acc[g].x += (double)xr, acc[g].y += (double)xi;
            xo[(size_t)f * fstride] = acc[g];
        }
    }
}

// The sums of the boxes a stack compaction keeps, moved to their places in the shorter point list.
__global__ void dft_gather_kernel(const double2* x_old, int old_points, const int* map, int new_points,
                                  double2* x_new) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= new_points) return;
    const size_t fc = blockIdx.y;
    x_new[fc * new_points + j] = x_old[fc * old_points + map[j]];
}

__global__ void expf_kernel(const float* in, float* out, size_t n) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = emlab_expf(in[i]);
}

}  // namespace

void launch_ports(const MonitorArgs& m, const int4* ports, int n, float* phasors, float* series, long long rec,
                  const float4* rot, const float* blend, int k, const Chain& s) {
    launch_chained(s, ports_kernel, (n + 63) / 64, 64, 0, m, ports, n, phasors, series, rec, rot, blend, k);
}

void launch_ntff(const MonitorArgs& m, const int* box, int points, float* phasors, const float4* rot,
                 const float* blend, int k, const Chain& s) {
    launch_chained(s, ntff_kernel, (points + kNtffThreads - 1) / kNtffThreads, kNtffThreads, 0, m, box, points,
                   reinterpret_cast<float4*>(phasors), rot, blend, k);
}

void launch_lines(const MonitorArgs& m, const int4* q, int nq, const int4* terms, const float* weights,
                  float* phasors, float* now, const float4* rot, const float* blend, int k, const Chain& s) {
    launch_chained(s, lines_kernel, (nq + 63) / 64, 64, 0, m, q, nq, terms, weights, reinterpret_cast<float4*>(phasors),
                   now, rot, blend, k);
}

void launch_probe_gather(const MonitorArgs& m, const int4* origins, int n, float4* out, const float*, const float*,
                         cudaStream_t s) {
    probe_kernel<<<(n * 54 + 63) / 64, 64, 0, s>>>(m, origins, n, out);
}

FluxRect flux_rect(const emlab_flux_plane& p, const int size[3], long long first) {
    FluxRect r{clampi(p.axis, 0, 2), p.index, max(p.rect_min[0], 0), max(p.rect_min[1], 0), 0, 0, 0, first};
    const int u = r.axis == 0 ? 1 : 0, v = r.axis == 2 ? 1 : 2;
    r.r0 = min(p.rect_max[0], size[u]) - r.m0, r.r1 = min(p.rect_max[1], size[v]) - r.m1;
    if (p.index >= 0 && p.index < size[r.axis] && r.r0 > 0 && r.r1 > 0) r.groups = (r.r0 + 15) / 16 * ((r.r1 + 15) / 16);
    return r;
}

int launch_flux_planes(const MonitorArgs& m, const FluxRect* rects, int n, float* partials, cudaStream_t s) {
    int launches = 0;
    for (int i = 0; i < n;) {
        FluxList list;
        int groups = 0;
        list.n = 0;
        for (; i < n && list.n < kFluxPlanes; ++i)
            if (rects[i].groups) list.r[list.n++] = rects[i], groups += rects[i].groups;
        if (!groups) continue;
        flux_kernel<<<groups, dim3(16, 16), 0, s>>>(m, list, partials);
        ++launches;
    }
    return launches;
}

void launch_sweep_sums(const float* series, long long steps, int nports, double nu_lo, double nu_hi, int points,
                       double dt, double* out, cudaStream_t s) {
    sweep_kernel<<<nports * points, 256, 0, s>>>(series, steps, nports, nu_lo, nu_hi, points, dt, out);
}

// Ring-down residual of every port (PortMonitor::evaluateSweep, Ports.cpp:206-213): the largest |V|
// of the last max(n / 20, 1) recorded steps over the largest |V| of all n (1 when there is no
// signal). One block per port; |V| maxima are exact in any order, so the result equals the host's.
__global__ void __launch_bounds__(256) residual_kernel(const float* series, long long steps, int nports, double* out) {
    __shared__ float s_peak[256], s_late[256];
    const int p = blockIdx.x;
    const long long tail = steps / 20 > 1 ? steps / 20 : 1, late_from = steps - tail;
    float peak = 0.0f, late = 0.0f;
    for (long long k = threadIdx.x; k < steps; k += blockDim.x) {
        const float v = fabsf(series[(k * nports + p) * 2]);
        peak = fmaxf(peak, v);
        if (k >= late_from) late = fmaxf(late, v);
    }
    s_peak[threadIdx.x] = peak, s_late[threadIdx.x] = late;
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if ((int)threadIdx.x < w) {
            s_peak[threadIdx.x] = fmaxf(s_peak[threadIdx.x], s_peak[threadIdx.x + w]);
            s_late[threadIdx.x] = fmaxf(s_late[threadIdx.x], s_late[threadIdx.x + w]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) out[p] = s_peak[0] > 0.0f ? (double)s_late[0] / (double)s_peak[0] : 1.0;
}

void launch_port_residuals(const float* series, long long steps, int nports, double* out, cudaStream_t s) {
    residual_kernel<<<nports, 256, 0, s>>>(series, steps, nports, out);
}

void launch_check_finite(const MonitorArgs& m, unsigned* flag, cudaStream_t s) {
    finite_kernel<<<sm_count() * 8, 256, 0, s>>>(m, flag);
}

void launch_dft_sample(const MonitorArgs& m, const int* boxes, int nbox, int box_max, int points, float* blk, int t,
                       const Chain& s) {
    launch_chained(s, dft_sample_kernel, dim3((box_max + 255) / 256, nbox), 256, 0, m, boxes, points, blk, t);
}

void launch_dft_gather(const double* x_old, int old_points, const int* map, int new_points, int nf, double* x_new,
                       cudaStream_t s) {
    dft_gather_kernel<<<dim3((new_points + 255) / 256, nf * 6), 256, 0, s>>>(
        reinterpret_cast<const double2*>(x_old), old_points, map, new_points, reinterpret_cast<double2*>(x_new));
}

void launch_dft_fold(const float* blk, int T, int points, int nf, const float2* W, const double* omega, long long n0,
                     double dt, double* X, cudaStream_t s) {
    const long long cols = 6ll * points;
    const size_t smem = (size_t)(nf * kDftMaxT + 2 * nf) * sizeof(float2);
    static size_t smem_set = 48 * 1024;
    if (smem > smem_set &&
        cudaFuncSetAttribute(dft_fold_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess)
        smem_set = smem;
    dft_fold_kernel<<<(unsigned)((cols + 127) / 128), 128, smem, s>>>(blk, T, points, nf, W, omega, n0, dt, X);
}

void launch_debug_expf(const float* in, float* out, size_t n, cudaStream_t s) {
    expf_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(in, out, n);
}

}  // namespace emlab
