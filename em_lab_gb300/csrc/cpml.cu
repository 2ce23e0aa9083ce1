// cpml.cu - the opt-in convolutional PML (no counterpart in the reference).
//
// The reference absorbs outgoing waves with a graded conductivity and a matched magnetic loss
// (shaders/common.glsl:15-43, update_E.comp:51-61, update_B.comp:58-66); that stays the default and
// the parity path. emlab_grid_set_cpml replaces it with a convolutional PML with a
// complex-frequency-shifted stretch (Roden & Gedney 2000): inside the absorber slabs every spatial
// derivative dF of the curl along an axis a becomes dF / kappa_a + psi, with the auxiliary field
// psi <- b_a psi + c_a dF kept per cell and per (component, axis) pair. Coefficients b, c, 1/kappa
// depend on the position along one axis only (emlab_cpml_coef) and live in per-axis tables for
// the integer positions (the E update's backward differences) and the half-integer positions (the B
// update's forward differences). The reference absorber's conductivity is switched off (its tables
// are built with sigma_max 0, which leaves the plain update bit for bit), so the materials' own
// (ca, cb) and thin-wire factors apply everywhere.
//
// psi storage: only the slabs, L + 1 cells at each end of the axis the derivative runs along
// (S = 2 (L + 1) positions per axis), four FP32 arrays per axis: the two E components and the two
// B components whose curl differentiates along it. Array slot j of axis a: 0 = E component
// (a+2)%3 (its term0 = d_a F), 1 = E component (a+1)%3 (its term1 = d_a F), 2 and 3 the same for
// B. Layout per axis (s = slab position): x: ((z ny + y) S + s), y: ((z S + s) pitch + x),
// z: ((s ny + y) pitch + x), so consecutive threads (consecutive x) touch consecutive entries except
// along x.
//
// The step runs as two in-place passes over the current field generation, B then E (the
// reference's pass order, SimulationGrid.cpp:394-410), followed by the ordinary source pass.
// What a pass moves (the three components it reads, the three it updates, the class index, the psi of
// slab cells: about 45 bytes a cell) bounds it, so long as enough loads are in flight: a thread takes two
// cells of a row through a chunk of planes, copies the next plane's operands into shared memory of its own
// while it works on one, keeps the plane neighbour in registers and takes the row neighbour from the next
// lane. The E pass takes the chunks from the top down, so that it starts on what the B pass left in L2 and
// the next B pass on what it leaves. A step of 192 x 168 x 144 cells with sources, of 20 waited for
// together: 124 us with a cell a thread, whose stores of psi and of one component stood before the loads
// of the next; 106 us with two cells in registers, 88 us with the copies ahead, 80 us with the E pass
// turned round.
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "emlab_internal.h"
#include "emlab_math.h"
#include "grid_state.h"

namespace emlab {

namespace {

struct CpmlArgs {
    const float4* coef;  // [lattice: 0 integer, 1 half][axis][stride]: (b, c, 1/kappa, 0)
    int stride;
    int L1;              // slab positions per side: L + 1
    float* psi[3];       // per derivative axis: 4 arrays of slab[axis] entries
    long long slab[3];
};

__device__ __forceinline__ int slab_pos(int i, int n, int L1) {
    return i < L1 ? i : (i >= n - L1 ? i - n + 2 * L1 : -1);
}

// A stretched derivative, psi updated: psi <- b psi + c d, d / kappa + psi. k: (b, c, 1/kappa)
__device__ __forceinline__ void stretch(const float4& k, float& d, float& psi) {
    psi = k.x * psi + k.y * d;
    d = d * k.z + psi;
}

__device__ __forceinline__ void get2(const float* p, float v[2]) {
    const float2 t = *reinterpret_cast<const float2*>(p);
    v[0] = t.x, v[1] = t.y;
}
__device__ __forceinline__ void put2(float* p, bool first, bool second, const float v[2]) {
    if (second) *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
    else if (first) *p = v[0];
}
// cp.async of N bytes into shared memory, zeros instead where !valid
template <int N>
__device__ __forceinline__ void copy_async(unsigned dst, const void* src, bool valid = true) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(N), "r"(valid ? N : 0) : "memory");
}

constexpr int kCpmlThreads = 128;
// A plane's operands of a thread on their way: float2 slots (differentiated field, its row neighbour,
// updated field, psi along y and z, class pair) and floats (row-end neighbour, psi along x).
constexpr int kStages = 2, kStageBytes = kCpmlThreads * 128;
enum { kF = 0, kRow = 3, kG = 5, kPsiY = 8, kPsiZ = 10, kCls = 12, kFloats = 13, kOver = 0, kPsiX = 2 };

// One pass: thread (two cells from x, row y) through planes zs .. ze. kB: B^{n+1/2} = B^{n-1/2} - dt curl E^n
// (forward differences at the half-integer positions; E beyond the upper faces is 0 as in
// update_B.comp:27-29). Otherwise E^{n+1} = ca E^n + cb curl B^{n+1/2} (backward differences at the
// integer positions; B below the lower faces is 0 as in update_E.comp:27-29), (ca, cb) of the edge material
// (no absorber conductivity). F: the field differentiated, G: the one updated. LX lanes share a row.
template <typename Idx, int LX, bool kB>
__global__ void __launch_bounds__(kCpmlThreads, 5) cpml_kernel(YeeArgs a, CpmlArgs p, int zchunk) {
    extern __shared__ __align__(16) unsigned char smem[];
    chain_wait();
    chain_next();
    const int lane = threadIdx.x % LX;
    const int xt = (blockIdx.x * LX + lane) * 2, yt = blockIdx.y * (kCpmlThreads / LX) + threadIdx.x / LX;
    const bool c0 = xt < a.nx && yt < a.ny, c1 = xt + 1 < a.nx && yt < a.ny;
    // a thread beyond the grid reads along inside the row's padding or in the last row and stores nothing
    const int x = min(xt, a.pitch - 2), y = min(yt, a.ny - 1);
    const int zs = (kB ? blockIdx.z : gridDim.z - 1 - blockIdx.z) * zchunk, ze = min(a.nz, zs + zchunk);
    constexpr int lattice = kB ? 1 : 0, slot = kB ? 2 : 0;
    const float* const F[3] = {kB ? a.wex : a.wbx, kB ? a.wey : a.wby, kB ? a.wez : a.wbz};
    float* const G[3] = {kB ? a.wbx : a.wex, kB ? a.wby : a.wey, kB ? a.wbz : a.wez};
    // neighbours along y and beyond the row's end: the side the differences take
    const bool yn = kB ? y + 1 < a.ny : y > 0;
    const long long row = kB ? a.pitch : -(long long)a.pitch;
    const bool right = x + 2 < a.nx;  // the next lane's first cell is in the grid
    const bool edge = kB ? lane == LX - 1 && right : lane == 0 && x > 0;
    const int S = 2 * p.L1, sy = c0 ? slab_pos(y, a.ny, p.L1) : -1;
    const int sx0 = c0 ? slab_pos(x, a.nx, p.L1) : -1, sx1 = c1 ? slab_pos(x + 1, a.nx, p.L1) : -1;
    const float4* coef = p.coef + lattice * 3 * p.stride;
    float4 kx0{}, kx1{}, ky{};
    if (sx0 >= 0) kx0 = __ldg(coef + x);
    if (sx1 >= 0) kx1 = __ldg(coef + x + 1);
    if (sy >= 0) ky = __ldg(coef + p.stride + y);
    struct alignas(2 * sizeof(Idx)) Pair {
        Idx v[2];
    };
    const unsigned sm = (unsigned)__cvta_generic_to_shared(smem);
    const unsigned my8 = threadIdx.x * 8, my4 = kFloats * kCpmlThreads * 8 + threadIdx.x * 4;
    // offsets of the plane being copied: fields, psi along x and y; psi along z by its slab position
    const long long step_x = (long long)a.ny * S, step_y = (long long)S * a.pitch, step_z = (long long)a.ny * a.pitch;
    float* psi_x = p.psi[0] + slot * p.slab[0] + zs * step_x + (long long)y * S;
    float* psi_y = p.psi[1] + slot * p.slab[1] + zs * step_y + (long long)sy * a.pitch + x;
    float* const psi_z = p.psi[2] + slot * p.slab[2] + (long long)y * a.pitch + x;
    long long q = (long long)zs * a.plane + (long long)y * a.pitch + x;
    // f: the cell's own F; for B the plane above is read ahead and becomes f, for E the plane below is kept
    float f[3][2], fz[3][2] = {};
    if (kB) {
        for (int c = 0; c < 3; ++c) get2(F[c] + q, f[c]);
    } else if (zs > 0) {
        for (int c = 0; c < 2; ++c) get2(F[c] + q - a.plane, fz[c]);
    }
    // plane z into stage st; each thread copies for itself: no barrier, only its own groups to wait for
    auto issue = [&](int z, unsigned st, long long q, const float* rx, const float* ry) {
        if (z < ze) {
            const unsigned d8 = sm + st + my8, d4 = sm + st + my4;
            constexpr int w8 = kCpmlThreads * 8, w4 = kCpmlThreads * 4;
            const bool fv = !kB || z + 1 < a.nz;
            const long long qf = kB && fv ? q + a.plane : q, qr = yn ? q + row : q;
            for (int c = 0; c < 3; ++c) copy_async<8>(d8 + (kF + c) * w8, F[c] + qf, fv);
            copy_async<8>(d8 + kRow * w8, F[0] + qr, yn);
            copy_async<8>(d8 + (kRow + 1) * w8, F[2] + qr, yn);
            for (int c = 0; c < 3; ++c) copy_async<8>(d8 + (kG + c) * w8, G[c] + q);
            copy_async<2 * sizeof(Idx)>(d8 + kCls * w8, static_cast<const Idx*>(a.cls) + q);
            if (edge) {
                copy_async<4>(d4 + kOver * w4, F[1] + (kB ? q + 2 : q - 1));
                copy_async<4>(d4 + (kOver + 1) * w4, F[2] + (kB ? q + 2 : q - 1));
            }
            if (sx0 >= 0) {
                copy_async<4>(d4 + kPsiX * w4, rx + sx0);
                copy_async<4>(d4 + (kPsiX + 2) * w4, rx + p.slab[0] + sx0);
            }
            if (sx1 >= 0) {
                copy_async<4>(d4 + (kPsiX + 1) * w4, rx + sx1);
                copy_async<4>(d4 + (kPsiX + 3) * w4, rx + p.slab[0] + sx1);
            }
            if (sy >= 0) {
                copy_async<8>(d8 + kPsiY * w8, ry);
                copy_async<8>(d8 + (kPsiY + 1) * w8, ry + p.slab[1]);
            }
            const int sz = slab_pos(z, a.nz, p.L1);
            if (sz >= 0) {
                copy_async<8>(d8 + kPsiZ * w8, psi_z + sz * step_z);
                copy_async<8>(d8 + (kPsiZ + 1) * w8, psi_z + p.slab[2] + sz * step_z);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned st = 0;
    issue(zs, st, q, psi_x, psi_y);
    for (int z = zs; z < ze; ++z, st ^= kStageBytes, q += a.plane, psi_x += step_x, psi_y += step_y) {
        issue(z + 1, st ^ kStageBytes, q + a.plane, psi_x + step_x, psi_y + step_y);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        auto get = [&](int slot8, float v[2]) {
            get2(reinterpret_cast<const float*>(smem + st + my8 + slot8 * kCpmlThreads * 8), v);
        };
        auto get4 = [&](int k) { return *reinterpret_cast<const float*>(smem + st + my4 + k * kCpmlThreads * 4); };
        float fy0[2], fy2[2], over1 = 0.0f, over2 = 0.0f, g[3][2];
        for (int c = 0; c < 3; ++c) get(kF + c, kB ? fz[c] : f[c]);
        get(kRow, fy0), get(kRow + 1, fy2);
        for (int c = 0; c < 3; ++c) get(kG + c, g[c]);
        if (edge) over1 = get4(kOver), over2 = get4(kOver + 1);
        const Pair cp = *reinterpret_cast<const Pair*>(smem + st + my8 + kCls * kCpmlThreads * 8);
        const unsigned cls[2] = {cp.v[0], c1 ? cp.v[1] : cp.v[0]};
        const int sz = slab_pos(z, a.nz, p.L1);
        // curl_c F = t0 - t1, t0 = d_{c+1} F_{c+2}, t1 = d_{c+2} F_{c+1}
        float t0[3][2], t1[3][2];
        if (kB) {
            float fx1 = __shfl_down_sync(0xffffffffu, f[1][0], 1, LX), fx2 = __shfl_down_sync(0xffffffffu, f[2][0], 1, LX);
            if (lane == LX - 1 || !right) fx1 = over1, fx2 = over2;
            for (int j = 0; j < 2; ++j) {
                const float n1 = j ? fx1 : (c1 ? f[1][1] : 0.0f), n2 = j ? fx2 : (c1 ? f[2][1] : 0.0f);  // one cell up in x
                t0[0][j] = fy2[j] - f[2][j], t0[1][j] = fz[0][j] - f[0][j], t0[2][j] = n1 - f[1][j];
                t1[0][j] = fz[1][j] - f[1][j], t1[1][j] = n2 - f[2][j], t1[2][j] = fy0[j] - f[0][j];
                if (cls[j] >= a.wire_start) {
                    const float4 w0 = __ldg(a.tabW + 2 * cls[j]), w1 = __ldg(a.tabW + 2 * cls[j] + 1);
                    t0[0][j] = t0[0][j] * w0.x, t0[1][j] = t0[1][j] * w0.y, t0[2][j] = t0[2][j] * w0.z;
                    t1[0][j] = t1[0][j] * w0.w, t1[1][j] = t1[1][j] * w1.x, t1[2][j] = t1[2][j] * w1.y;
                }
            }
        } else {
            float fx1 = __shfl_up_sync(0xffffffffu, f[1][1], 1, LX), fx2 = __shfl_up_sync(0xffffffffu, f[2][1], 1, LX);
            if (lane == 0) fx1 = over1, fx2 = over2;
            for (int j = 0; j < 2; ++j) {
                const float n1 = j ? f[1][0] : fx1, n2 = j ? f[2][0] : fx2;  // one cell down in x
                t0[0][j] = f[2][j] - fy2[j], t0[1][j] = f[0][j] - fz[0][j], t0[2][j] = f[1][j] - n1;
                t1[0][j] = f[1][j] - fz[1][j], t1[1][j] = f[2][j] - n2, t1[2][j] = f[0][j] - fy0[j];
            }
        }
        // psi of the slabs the cells lie in: along x each cell for itself, along y and z both
        for (int j = 0; j < 2; ++j) {
            if (j ? sx1 < 0 : sx0 < 0) continue;
            float* rx = psi_x + (j ? sx1 : sx0);
            for (int t = 0; t < 2; ++t) {
                float v = get4(kPsiX + 2 * t + j);
                stretch(j ? kx1 : kx0, t ? t1[1][j] : t0[2][j], v);
                rx[t * p.slab[0]] = v;
            }
        }
        if (sy >= 0) {
            for (int t = 0; t < 2; ++t) {
                float v[2];
                get(kPsiY + t, v);
                for (int j = 0; j < 2; ++j) stretch(ky, t ? t1[2][j] : t0[0][j], v[j]);
                put2(psi_y + t * p.slab[1], c0, c1, v);
            }
        }
        if (sz >= 0) {
            const float4 kz = __ldg(coef + 2 * p.stride + z);
            for (int t = 0; t < 2; ++t) {
                float v[2];
                get(kPsiZ + t, v);
                for (int j = 0; j < 2; ++j) stretch(kz, t ? t1[0][j] : t0[1][j], v[j]);
                put2(psi_z + t * p.slab[2] + sz * step_z, c0, c1, v);
            }
        }
        if (kB) {
            for (int c = 0; c < 3; ++c)
                for (int j = 0; j < 2; ++j) g[c][j] = g[c][j] - a.dt * (t0[c][j] - t1[c][j]);
        } else {
            float4 m0 = __ldg(a.tabE + 2 * cls[0]), m1 = __ldg(a.tabE + 2 * cls[0] + 1);
            for (int j = 0; j < 2; ++j) {
                if (j && cls[1] != cls[0]) m0 = __ldg(a.tabE + 2 * cls[1]), m1 = __ldg(a.tabE + 2 * cls[1] + 1);
                const float ca[3] = {m0.x, m0.y, m0.z}, cb[3] = {m0.w, m1.x, m1.y};
                for (int c = 0; c < 3; ++c) g[c][j] = ca[c] * g[c][j] + cb[c] * (t0[c][j] - t1[c][j]);
            }
        }
        for (int c = 0; c < 3; ++c) put2(G[c] + q, c0, c1, g[c]);
        for (int c = 0; c < 3; ++c)
            for (int j = 0; j < 2; ++j) {
                if (kB) f[c][j] = fz[c][j];
                else fz[c][j] = f[c][j];
            }
    }
}

template <typename Idx, int LX, bool kB>
void launch_pass(const YeeArgs& a, const CpmlArgs& p, const Chain& s) {
    constexpr int rows = kCpmlThreads / LX;
    const dim3 tiles((a.nx + 2 * LX - 1) / (2 * LX), (a.ny + rows - 1) / rows);
    // Chunks re-read the plane neighbour of their first plane, and a launch wants its blocks (five to an SM) to
    // come out in several waves: the deepest chunk of at most eight planes with four waves, or single planes.
    const int want = 4 * 5 * sm_count(), least = (int)std::min<long long>(a.nz, (want + tiles.x * tiles.y - 1) / (tiles.x * tiles.y));
    const int zc = std::max(1, std::min(8, a.nz / least));
    launch_chained(s, cpml_kernel<Idx, LX, kB>, dim3(tiles.x, tiles.y, (a.nz + zc - 1) / zc), kCpmlThreads, kStages * kStageBytes, a, p, zc);
}

template <typename Idx>
void launch_step(const YeeArgs& a, const CpmlArgs& p, const Chain& s) {
    // rows of 64 cells a warp, or of 32 where that leaves fewer lanes idle
    if ((a.nx + 63) / 64 * 64 == (a.nx + 31) / 32 * 32) {
        launch_pass<Idx, 32, true>(a, p, s);
        launch_pass<Idx, 32, false>(a, p, {s.stream, true});
    } else {
        launch_pass<Idx, 16, true>(a, p, s);
        launch_pass<Idx, 16, false>(a, p, {s.stream, true});
    }
}

CpmlArgs cpml_args(emlab_grid* g) {
    CpmlArgs p{};
    p.coef = g->cpml_coef.p;
    p.stride = g->cpml_stride;
    p.L1 = g->cfg.pml_thickness + 1;
    for (int ax = 0; ax < 3; ++ax) {
        p.slab[ax] = g->cpml_slab[ax];
        p.psi[ax] = g->cpml_psi.p + g->cpml_psi_off[ax];
    }
    return p;
}

}  // namespace

int cpml_prepare(emlab_grid* g) {
    const emlab_grid_config& c = g->cfg;
    const int n[3] = {c.nx, c.ny, c.nz};
    const int L = c.pml_thickness, L1 = L + 1, S = 2 * L1;
    const int stride = std::max(c.nx, std::max(c.ny, c.nz));
    std::vector<float4> coef((size_t)2 * 3 * stride, make_float4(1.0f, 0.0f, 1.0f, 0.0f));
    for (int lat = 0; lat < 2; ++lat)
        for (int ax = 0; ax < 3; ++ax)
            for (int i = 0; i < n[ax]; ++i) {
                float k[3];
                emlab_cpml_coef((double)i + (lat ? 0.5 : 0.0), n[ax], L, g->cpml.sigma_max, g->cpml.kappa_max,
                                g->cpml.alpha_max, g->cpml.order, (double)c.courant, k);
                coef[((size_t)lat * 3 + ax) * stride + i] = make_float4(k[0], k[1], k[2], 0.0f);
            }
    g->cpml_stride = stride;
    const long long area[3] = {(long long)c.ny * c.nz, (long long)g->pitch * c.nz, (long long)g->pitch * c.ny};
    long long total = 0;
    for (int ax = 0; ax < 3; ++ax) {
        g->cpml_slab[ax] = area[ax] * S;
        g->cpml_psi_off[ax] = total;
        total += 4 * g->cpml_slab[ax];
    }
    EMLAB_CUDA(g->cpml_coef.alloc(coef.size()));
    EMLAB_CUDA(cudaMemcpyAsync(g->cpml_coef.p, coef.data(), coef.size() * sizeof(float4), cudaMemcpyHostToDevice, g->stream));
    EMLAB_CUDA(g->cpml_psi.alloc((size_t)total));
    EMLAB_CUDA(cudaMemsetAsync(g->cpml_psi.p, 0, (size_t)total * sizeof(float), g->stream));
    return EMLAB_OK;
}

int cpml_clear(emlab_grid* g) {
    if (g->cpml_on && g->cpml_psi.p)
        EMLAB_CUDA(cudaMemsetAsync(g->cpml_psi.p, 0, g->cpml_psi.n * sizeof(float), g->stream));
    return EMLAB_OK;
}

void launch_cpml(emlab_grid* g, const YeeArgs& a, bool wide, const Chain& s) {
    const CpmlArgs p = cpml_args(g);
    if (wide) launch_step<uint32_t>(a, p, s);
    else launch_step<uint16_t>(a, p, s);
}

}  // namespace emlab

using namespace emlab;

extern "C" int emlab_grid_set_cpml(emlab_grid* g, const emlab_cpml* params) {
    if (int rc = require_grid(g)) return rc;
    EMLAB_REQUIRE(g->stack.scenes() == 0, "the convolutional PML is not available for stacks of scenes");
    if (params) {
        EMLAB_REQUIRE(params->sigma_max >= 0.0f && params->kappa_max >= 1.0f && params->alpha_max >= 0.0f &&
                          params->order >= 1.0f && params->order <= 8.0f,
                      "CPML parameters out of range (sigma_max >= 0, kappa_max >= 1, alpha_max >= 0, 1 <= order <= 8)");
    }
    EMLAB_CUDA(cudaSetDevice(g->device));
    EMLAB_CUDA(cudaStreamSynchronize(g->stream));
    g->cpml_on = params != nullptr;
    if (params) g->cpml = *params;
    if (int rc = upload_pml(g)) return rc;  // the reference absorber's tables: off under the CPML
    if (g->cpml_on) {
        if (int rc = cpml_prepare(g)) return rc;
    } else {
        g->cpml_psi.release(), g->cpml_coef.release();
    }
    if (int rc = clear_fields(g)) return rc;
    g->step = 0;
    return EMLAB_OK;
}
