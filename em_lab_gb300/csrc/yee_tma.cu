// yee_tma.cu - the fused Yee step with TMA-staged z planes (sm_103a).
//
// Same arithmetic and traversal as yee_fused (yee.cu): a CTA owns a 32 x TY column of cells and
// marches it along z, computing B^{n+1/2} for its cells plus the -x/-y halo cells, then E^{n+1}.
// Difference: the inputs of each z plane (E^n with a one-cell halo, B^n and the class index with
// the low halo) arrive by cp.async.bulk.tensor into a 4- or 6-deep shared-memory ring, issued by
// a control warp and completed on per-stage mbarriers, so several planes are in flight while the
// CTA computes; threads never form global addresses for loads. The control warp also computes the
// halo B components, so the cell warps run a branch-free update with hoisted invariants.
// B^{n+1/2} of the plane is kept in a double-buffered shared tile so one __syncthreads per plane
// suffices. Results go to the other field generation with coalesced 128-byte warp stores.
//
// TMA boxes start at x0-4 (x0-8 for a 16-bit class index) so the innermost coordinate stays
// 16-byte aligned; coordinates outside the grid read zeros, which is exactly the reference's
// rule that E beyond the upper faces is 0 (update_B.comp:27-29). Every mbarrier wait is bounded:
// on expiry the CTA records an error word and leaves (the host reports EMLAB_ERR_TIMEOUT).
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "yee_common.cuh"

namespace emlab {

struct TmaMaps {
    CUtensorMap e[2][3];   // single-cell tiles: one map per component
    CUtensorMap b[2][3];
    CUtensorMap e3[2], b3[2];  // pair tiles: the three components of E, of B, as the fourth dimension
    CUtensorMap cls;
    bool ok[2] = {false, false};
    bool cls_ok = false;
    int tiling = -1;  // YeeArgs::tile_rows that the boxes were made for
};

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: `polls` tries, about a second of polling at the default kWaitPolls (try_wait itself
// suspends for a while); 0 tries gives up at once (the test hook of emlab_debug_set_wait_limit).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int polls = kWaitPolls) {
    for (int i = 0; i < polls; ++i)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// One copy of a tile's plane of all three components (component index 0 of the map's last dimension).
__device__ __forceinline__ void tma_load_3comp(void* dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(0), "r"(smem_u32(bar))
        : "memory");
}

template <int TY, typename Idx>
struct Layout {
    static constexpr int STAGES = TY <= 8 ? 6 : 4;           // planes in the shared-memory ring
    static constexpr int EW = 40;                         // E box: x0-4 .. x0+35, TY+2 rows
    static constexpr int BW = 36;                         // B box: x0-4 .. x0+31, TY+1 rows
    static constexpr int CW = sizeof(Idx) == 2 ? 40 : 36;  // class box width
    static constexpr int CX = sizeof(Idx) == 2 ? 8 : 4;    // class box starts at x0 - CX
    static constexpr int E_BYTES = EW * (TY + 2) * 4;
    static constexpr int B_BYTES = BW * (TY + 1) * 4;
    static constexpr int C_BYTES = CW * (TY + 1) * (int)sizeof(Idx);
    static constexpr int EP = (E_BYTES + 127) / 128 * 128;  // 128-byte aligned TMA destinations
    static constexpr int BP = (B_BYTES + 127) / 128 * 128;
    static constexpr int CP = (C_BYTES + 127) / 128 * 128;
    static constexpr int E_OFF = 0;
    static constexpr int B_OFF = 3 * EP;
    static constexpr int C_OFF = B_OFF + 3 * BP;
    static constexpr int STAGE = C_OFF + CP;
    static constexpr uint32_t TX_BYTES = 3 * E_BYTES + 3 * B_BYTES + C_BYTES;
    static constexpr int SB_OFF = STAGES * STAGE;                    // B^{n+1/2}: [2][3][TY+1][33]
    static constexpr int SB_BYTES = 2 * 3 * (TY + 1) * 33 * 4;
    static constexpr int BAR_OFF = (SB_OFF + SB_BYTES + 127) / 128 * 128;
    static constexpr int SMEM = BAR_OFF + 8 * STAGES;
};

// Warps 0..TY-1 own the tile's cells (warp w = row y0+w, lane = x0+lane). Warp TY is the halo and
// control warp: it issues the TMA copies, waits on the mbarriers (so no other warp ever polls), and
// computes the B^{n+1/2} components of the -y row and -x column that the E update of the tile
// needs (Bx, Bz at (x0+lane, y0-1); By, Bz at (x0-1, y0+lane)).
template <int TY, typename Idx>
__global__ void __launch_bounds__(32 * (TY + 1), TY <= 8 ? 3 : 1)
    yee_tma(const __grid_constant__ CUtensorMap tex, const __grid_constant__ CUtensorMap tey,
            const __grid_constant__ CUtensorMap tez, const __grid_constant__ CUtensorMap tbx,
            const __grid_constant__ CUtensorMap tby, const __grid_constant__ CUtensorMap tbz,
            const __grid_constant__ CUtensorMap tcls, YeeArgs a, unsigned* err) {
    using Lay = Layout<TY, Idx>;
    constexpr int S_ = Lay::STAGES;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Lay::BAR_OFF);
    float* sB = reinterpret_cast<float*>(smem + Lay::SB_OFF);

    const int lane = threadIdx.x, warp = threadIdx.y;
    const bool ctl = warp == TY;
    const int x0 = blockIdx.x * 32, y0 = blockIdx.y * TY;
    const int zs = blockIdx.z * a.zchunk;
    const int ze = min(a.nz, zs + a.zchunk);
    if (zs >= ze) return;
    const int zstart = zs > 0 ? zs - 1 : zs;  // a chunk above z = 0 first rebuilds B^{n+1/2}(zs-1)
    const int zlast = ze;                      // planes zstart .. ze are read (ze as the "z+1" plane)

    auto issue = [&](int p) {
        unsigned char* st = smem + ((p - zstart) % S_) * Lay::STAGE;
        uint64_t* bar = bars + (p - zstart) % S_;
        mbar_expect_tx(bar, Lay::TX_BYTES);
        tma_load_3d(st + Lay::E_OFF + 0 * Lay::EP, &tex, x0 - 4, y0 - 1, p, bar);
        tma_load_3d(st + Lay::E_OFF + 1 * Lay::EP, &tey, x0 - 4, y0 - 1, p, bar);
        tma_load_3d(st + Lay::E_OFF + 2 * Lay::EP, &tez, x0 - 4, y0 - 1, p, bar);
        tma_load_3d(st + Lay::B_OFF + 0 * Lay::BP, &tbx, x0 - 4, y0 - 1, p, bar);
        tma_load_3d(st + Lay::B_OFF + 1 * Lay::BP, &tby, x0 - 4, y0 - 1, p, bar);
        tma_load_3d(st + Lay::B_OFF + 2 * Lay::BP, &tbz, x0 - 4, y0 - 1, p, bar);
        tma_load_3d(st + Lay::C_OFF, &tcls, x0 - Lay::CX, y0 - 1, p, bar);
    };
    const bool leader = ctl && lane == 0;
    if (leader) {
        for (int s = 0; s < S_; ++s) mbar_init(bars + s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    chain_wait();
    chain_next();
    bool failed = false;
    int issued_hi = zstart - 1;  // leader: last plane whose loads were issued
    int waited_ok = zstart - 1;  // leader: last plane whose loads were seen complete
    // on an expired wait: record the error, then give every copy still in flight (the plane that
    // timed out included) a bounded time to land before the CTA leaves and its shared memory goes
    auto bail = [&]() {
        if (leader) {
            atomicOr(err, 1u);
            for (int p = waited_ok + 1; p <= issued_hi; ++p)
                mbar_wait(bars + (p - zstart) % S_, ((p - zstart) / S_) & 1);
        }
    };
    if (leader) {
        for (int p = zstart; p <= zlast && p < zstart + S_; ++p) issue(p), issued_hi = p;
        // planes zstart and zstart+1 before the first B phase; later planes one iteration ahead,
        // just before the per-plane barrier, which passes the TMA writes on to the other warps
        failed = !mbar_wait(bars + 0, 0, a.wait_polls);
        if (!failed) waited_ok = zstart, failed = !mbar_wait(bars + 1, 0, a.wait_polls);
        if (!failed) waited_ok = zstart + 1;
    }
    if (__syncthreads_or(failed)) {
        bail();
        return;
    }

    auto SB = [&](int buf, int c, int r, int col) -> float& { return sB[((buf * 3 + c) * (TY + 1) + r) * 33 + col]; };
    constexpr int EPF = Lay::EP / 4, BPF = Lay::BP / 4;
    const int L = a.L, K = a.pml_K, PS = a.pml_stride;
    const unsigned char* pcls = a.pml_cls;
    const float2* T = a.pml_coef;
    const float dt = a.dt;

    // ---- per-thread invariants of the z march ----
    // own warps: cell (x, y); halo warp: row cell (x0+lane, y0-1) and column cell (x0-1, y0+lane)
    const int x = ctl ? x0 + lane : x0 + lane;
    const int y = ctl ? y0 - 1 : y0 + warp;
    const bool own = !ctl && x < a.nx && y < a.ny;
    const bool row_live = ctl && y0 > 0 && x < a.nx;                        // (x0+lane, y0-1)
    const int cy = y0 + lane;                                               // column cell y
    const bool col_live = ctl && lane < TY && x0 > 0 && cy < a.ny;          // (x0-1, y0+lane)
    auto pml_rows = [&](int px, int py, int& R1, int& R2, int& R3, int& R4) {
        const int ix = __ldg(pcls + px), iy = __ldg(pcls + PS + py), hx = __ldg(pcls + 3 * PS + px),
                  hy = __ldg(pcls + 4 * PS + py);
        R1 = hy * K + ix, R2 = iy * K + hx, R3 = hy * K + hx, R4 = iy * K + ix;
    };
    auto pml_xy_of = [&](int px, int py) { return px < L || py < L || px >= a.nx - (L + 1) || py >= a.ny - (L + 1); };
    int R1 = 0, R2 = 0, R3 = 0, R4 = 0, C1 = 0, C2 = 0, C3 = 0, C4 = 0;
    if (own || row_live) pml_rows(x, y, R1, R2, R3, R4);
    if (col_live) pml_rows(x0 - 1, cy, C1, C2, C3, C4);
    const bool pml_xy = (own || row_live) && pml_xy_of(x, y);
    const bool pml_xy_c = col_live && pml_xy_of(x0 - 1, cy);
    // shared-memory offsets: own/row cell and column cell (E/B box column 3 = x0-1)
    const int me = (ctl ? 0 : warp + 1) * Lay::EW + lane + 4;
    const int mb = (ctl ? 0 : warp + 1) * Lay::BW + lane + 4;
    const int mc = (ctl ? 0 : warp + 1) * Lay::CW + lane + Lay::CX;
    const int ce = (lane + 1) * Lay::EW + 3, cb = (lane + 1) * Lay::BW + 3, cc = (lane + 1) * Lay::CW + Lay::CX - 1;
    const long long row_off = (long long)y * a.pitch + x;

    float bpx = 0.0f, bpy = 0.0f;  // B^{n+1/2}(x, y, z-1).xy (B below the lower face is 0)
    for (int z = zstart; z < ze; ++z) {
        const int rel = z - zstart;
        const unsigned char* st = smem + (rel % S_) * Lay::STAGE;
        const unsigned char* st1 = smem + ((rel + 1) % S_) * Lay::STAGE;
        const bool emit = z >= zs;
        const int buf = rel & 1;
        const bool pz = __ldg(a.pml_z + z) != 0;
        const int iz = __ldg(pcls + 2 * PS + z) * K * K, hz = __ldg(pcls + 5 * PS + z) * K * K;  // table planes
        const float* Es = reinterpret_cast<const float*>(st + Lay::E_OFF);
        const float* E1 = reinterpret_cast<const float*>(st1 + Lay::E_OFF);
        const float* Bs = reinterpret_cast<const float*>(st + Lay::B_OFF);
        const Idx* Cs = reinterpret_cast<const Idx*>(st + Lay::C_OFF);
        const long long off = (long long)z * a.plane + row_off;
        float bx = 0.0f, by = 0.0f, bz = 0.0f, e0x = 0.0f, e0y = 0.0f, e0z = 0.0f;
        unsigned c = 0;
        if (own) {
            // update_B.comp:35-67 for the own cell
            e0x = Es[me], e0y = Es[EPF + me], e0z = Es[2 * EPF + me];
            bx = Bs[mb], by = Bs[BPF + mb], bz = Bs[2 * BPF + mb];
            c = (unsigned)Cs[mc];
            const float exy = Es[EPF + me + 1], exz = Es[2 * EPF + me + 1];
            const float eyx = Es[me + Lay::EW], eyz = Es[2 * EPF + me + Lay::EW];
            const float ezx = E1[me], ezy = E1[EPF + me];
            float t0x = eyz - e0z, t0y = ezx - e0x, t0z = exy - e0y;
            float t1x = ezy - e0y, t1y = exz - e0z, t1z = eyx - e0x;
            if (c >= a.wire_start) {
                const float4 w0 = __ldg(a.tabW + 2 * c), w1 = __ldg(a.tabW + 2 * c + 1);
                t0x = t0x * w0.x, t0y = t0y * w0.y, t0z = t0z * w0.z;
                t1x = t1x * w0.w, t1y = t1y * w1.x, t1z = t1z * w1.y;
            }
            const float cx = t0x - t1x, cy_ = t0y - t1y, cz = t0z - t1z;
            if (pml_xy || pz) {
                const float2 kx = __ldg(T + R1 + hz), ky = __ldg(T + R2 + hz), kz = __ldg(T + R3 + iz);
                bx = kx.x * bx - kx.y * cx;
                by = ky.x * by - ky.y * cy_;
                bz = kz.x * bz - kz.y * cz;
            } else {
                bx = bx - dt * cx;
                by = by - dt * cy_;
                bz = bz - dt * cz;
            }
            SB(buf, 0, warp + 1, lane + 1) = bx, SB(buf, 1, warp + 1, lane + 1) = by, SB(buf, 2, warp + 1, lane + 1) = bz;
            if (emit) a.nbx[off] = bx, a.nby[off] = by, a.nbz[off] = bz;
        } else if (ctl && emit) {
            // -y row: Bx, Bz at (x0+lane, y0-1) (update_B.comp:41-66, components x and z)
            float hbx = 0.0f, hbz = 0.0f;  // B below the lower faces is 0
            if (row_live) {
                const float f0x = Es[me], f0y = Es[EPF + me], f0z = Es[2 * EPF + me];
                const unsigned hc = (unsigned)Cs[mc];
                float t0x = Es[2 * EPF + me + Lay::EW] - f0z, t1x = E1[EPF + me] - f0y;  // d_y Ez, d_z Ey
                float t0z = Es[EPF + me + 1] - f0y, t1z = Es[me + Lay::EW] - f0x;      // d_x Ey, d_y Ex
                if (hc >= a.wire_start) {
                    const float4 w0 = __ldg(a.tabW + 2 * hc), w1 = __ldg(a.tabW + 2 * hc + 1);
                    t0x = t0x * w0.x, t0z = t0z * w0.z, t1x = t1x * w0.w, t1z = t1z * w1.y;
                }
                const float cx = t0x - t1x, cz = t0z - t1z;
                hbx = Bs[mb], hbz = Bs[2 * BPF + mb];
                if (pml_xy || pz) {
                    const float2 kx = __ldg(T + R1 + hz), kz = __ldg(T + R3 + iz);
                    hbx = kx.x * hbx - kx.y * cx;
                    hbz = kz.x * hbz - kz.y * cz;
                } else {
                    hbx = hbx - dt * cx;
                    hbz = hbz - dt * cz;
                }
            }
            SB(buf, 0, 0, lane + 1) = hbx, SB(buf, 2, 0, lane + 1) = hbz;
            // -x column: By, Bz at (x0-1, y0+lane)
            if (lane < TY) {
                float hby = 0.0f, hbz2 = 0.0f;
                if (col_live) {
                    const float f0x = Es[ce], f0y = Es[EPF + ce], f0z = Es[2 * EPF + ce];
                    const unsigned hc = (unsigned)Cs[cc];
                    float t0y = E1[ce] - f0x, t1y = Es[2 * EPF + ce + 1] - f0z;   // d_z Ex, d_x Ez
                    float t0z = Es[EPF + ce + 1] - f0y, t1z = Es[ce + Lay::EW] - f0x;  // d_x Ey, d_y Ex
                    if (hc >= a.wire_start) {
                        const float4 w0 = __ldg(a.tabW + 2 * hc), w1 = __ldg(a.tabW + 2 * hc + 1);
                        t0y = t0y * w0.y, t0z = t0z * w0.z, t1y = t1y * w1.x, t1z = t1z * w1.y;
                    }
                    const float cyy = t0y - t1y, cz = t0z - t1z;
                    hby = Bs[BPF + cb], hbz2 = Bs[2 * BPF + cb];
                    if (pml_xy_c || pz) {
                        const float2 ky = __ldg(T + C2 + hz), kz = __ldg(T + C3 + iz);
                        hby = ky.x * hby - ky.y * cyy;
                        hbz2 = kz.x * hbz2 - kz.y * cz;
                    } else {
                        hby = hby - dt * cyy;
                        hbz2 = hbz2 - dt * cz;
                    }
                }
                SB(buf, 1, lane + 1, 0) = hby, SB(buf, 2, lane + 1, 0) = hbz2;
            }
        }
        // the next iteration's B phase reads plane z+2: the leader waits for it before the barrier
        if (leader && z + 1 < ze) {
            failed = !mbar_wait(bars + (rel + 2) % S_, ((rel + 2) / S_) & 1, a.wait_polls);
            if (!failed) waited_ok = z + 2;
        }
        if (__syncthreads_or(failed)) {
            bail();
            return;
        }
        // every warp is past its reads of plane z-1's stage: refill it with plane z-1+STAGES
        if (leader && z > zstart && z - 1 + S_ <= zlast) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(z - 1 + S_);
            issued_hi = z - 1 + S_;
        }
        if (emit && own) {
            // update_E.comp:41-64 for the own cell
            const float bxm_y = SB(buf, 1, warp + 1, lane), bxm_z = SB(buf, 2, warp + 1, lane);  // B(x-1)
            const float bym_x = SB(buf, 0, warp, lane + 1), bym_z = SB(buf, 2, warp, lane + 1);  // B(y-1)
            const float cx = (bz - bym_z) - (by - bpy);
            const float cy_ = (bx - bpx) - (bz - bxm_z);
            const float cz = (by - bxm_y) - (bx - bym_x);
            float ex = e0x, ey = e0y, ez = e0z;
            if (!(pml_xy || pz)) {
                if (c == 0) {  // vacuum: ca = 1 and cb = dt exactly, so 1 * e + dt * curl == e + dt * curl
                    ex = ex + dt * cx;
                    ey = ey + dt * cy_;
                    ez = ez + dt * cz;
                } else {
                    const float4 t0 = __ldg(a.tabE + 2 * c), t1 = __ldg(a.tabE + 2 * c + 1);
                    ex = t0.x * ex + t0.w * cx;
                    ey = t0.y * ey + t1.x * cy_;
                    ez = t0.z * ez + t1.y * cz;
                }
            } else if (c == 0) {
                const float2 kx = __ldg(T + R2 + iz), ky = __ldg(T + R1 + iz), kz = __ldg(T + R4 + hz);
                ex = kx.x * ex + kx.y * cx;
                ey = ky.x * ey + ky.y * cy_;
                ez = kz.x * ez + kz.y * cz;
            } else {
                e_cell(a, ex, ey, ez, cx, cy_, cz, c, x, y, z);
            }
            a.nex[off] = ex, a.ney[off] = ey, a.nez[off] = ez;
        }
        bpx = bx, bpy = by;
    }
}

// ------------------------------------------------------------------------------------------------
// Two cells per thread along x: a CTA owns a 64 x TY tile (warp w = row y0+w, lane l = cells
// x0+2l and x0+2l+1) or a 32 x 2 TY tile (two rows a warp, XL = 16 lanes each) and marches it along z.
// Same arithmetic per cell as above, bit for bit.
//
// What bounds it: HBM traffic (48.2 bytes a cell-step; 0.87 of the copy rate at 512 x 512 x 512 cells, 0.6 at 256 x 256 x
// 256) together with the plane barrier, and before these the instructions issued per cell, so the own warps' inner loop is written for few of them:
//  * every field is a pair of FP32 in one 64-bit register and the curls and updates are packed
//    .f32x2 operations (each half rounds as the scalar operation does, no contraction);
//  * the branches are uniform over the warp: a row of 64 cells outside the absorber takes one of two
//    straight paths (all vacuum, or the class table for every lane: the vacuum entry (1, dt) gives
//    the same bits), a row that touches the absorber reads the (e^-x, dt phi) table in every lane
//    (class 0 outside the layer is (1, dt) again); only rows with non-vacuum cells inside the
//    absorber, and rows with a thin-wire cell, branch per lane;
//  * outside the z layers the coefficients of a cell of the x / y layers do not change along z: they
//    are read once per item and kept in shared memory as the packed operands (one 16-byte load each);
//  * E(z+1).x and .y, read for B at plane z, stay in registers as plane z+1's own E;
//  * the halo (row y0-1 and column x0-1) and the copies have warps of their own (TY, TY+1). Issuing a
//    copy takes its thread about a hundred cycles, so a plane's E and B are one copy each (the three
//    components are the fourth dimension of the tensor map): three copies a plane instead of seven,
//    and nothing else in that warp's way; it was the longest chain of the plane.
template <int TY, typename Idx, int XL = 32>
struct Layout2 {
    static constexpr int STAGES = 4;
    static constexpr int ROWS = TY * 32 / XL;           // a warp holds 32 / XL rows of 2 XL cells
    static constexpr int W = 2 * XL + 8;                // box row width of E, B and the class index
    static constexpr int CX = sizeof(Idx) == 2 ? 8 : 4;  // boxes start at x0 - 4 (16-bit class: x0 - 8)
    static constexpr int DC = CX - 4;                   // class element offset from the E/B element
    static constexpr int EP = W * (ROWS + 2) * 4;       // one component: rows y0-1 .. y0+ROWS
    static constexpr int BP = W * (ROWS + 1) * 4;       // rows y0-1 .. y0+ROWS-1
    static constexpr int C_BYTES = W * (ROWS + 1) * (int)sizeof(Idx);
    static constexpr int E_OFF = 0;                     // the three components of a copy lie back to back
    static constexpr int B_OFF = (3 * EP + 127) / 128 * 128;
    static constexpr int C_OFF = B_OFF + (3 * BP + 127) / 128 * 128;
    static constexpr int STAGE = C_OFF + (C_BYTES + 127) / 128 * 128;
    static constexpr uint32_t TX_BYTES = 3 * EP + 3 * BP + C_BYTES;
    // B tile row: element e of a box row maps to slot e - 2 (col 1 = x0-1, col 2+i = x0+i)
    static constexpr int SB_OFF = STAGES * STAGE;
    static constexpr int SB_BYTES = 2 * 3 * (ROWS + 1) * W * 4;
    // absorber coefficients of every own pair outside the z layers: [entry r1..r4][thread]{decay, gain}
    static constexpr int COEF_OFF = (SB_OFF + SB_BYTES + 127) / 128 * 128;
    static constexpr int COEF_BYTES = 4 * 32 * TY * 16;
    static constexpr int BAR_OFF = COEF_OFF + COEF_BYTES;
    static constexpr int QUEUE_OFF = BAR_OFF + 8 * STAGES;  // item numbers [8], -1 = done
    static constexpr int STOP_OFF = QUEUE_OFF + 8 * 4;       // barrier after which every warp leaves, -1 = none
    static constexpr int SMEM = STOP_OFF + 16;
    static constexpr int CTAS = TY == 4 ? 3 : (TY == 8 ? 2 : 1);  // per SM
    static_assert(BAR_OFF % 8 == 0 && SB_OFF % 16 == 0, "shared-memory alignment");
    static_assert(SMEM <= 227 * 1024, "shared memory per CTA");
};

// A pair of FP32 (cells xa and xa+1) in one 64-bit register; packed IEEE operations (sm_100+).
using pair_t = unsigned long long;
__device__ __forceinline__ pair_t pk(float lo, float hi) {
    pair_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float lo_of(pair_t v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a;
}
__device__ __forceinline__ float hi_of(pair_t v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return b;
}
__device__ __forceinline__ pair_t add2(pair_t a, pair_t b) {
    pair_t r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ pair_t sub2(pair_t a, pair_t b) {
    pair_t r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// a * b, rounded once: a * b + (-0). The compiler merges a packed multiply with the packed addition
// that uses it into one multiply-add with one rounding, whatever -fmad says, and folds a constant -0
// away; mz (YeeArgs::minus_zero) is a -0 it cannot see.
__device__ __forceinline__ pair_t mul2(pair_t a, pair_t b, pair_t mz) {
    pair_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(mz));
    return r;
}
__device__ __forceinline__ pair_t lds2(const float* p) { return *reinterpret_cast<const pair_t*>(p); }
__device__ __forceinline__ void sts2(float* p, pair_t v) { *reinterpret_cast<pair_t*>(p) = v; }

// The next field generation is not read again in the launch: its stores leave L2 first, so the
// current generation's planes stay for the neighbouring tiles' halo reads. The policy is made at
// each use (one instruction) rather than held in a register across the z march.
__device__ __forceinline__ uint64_t evict_first_policy() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void st_pair(float* p, pair_t v, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.b64 [%0], %1, %2;" ::"l"(p), "l"(v), "l"(policy) : "memory");
}
__device__ __forceinline__ void st_one(float* p, float v, uint64_t policy) {
    asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(policy) : "memory");
}
// The pair's cells inside the scene: both (o1), the first (o0), or none.
__device__ __forceinline__ void st_cells(float* p, pair_t v, bool o0, bool o1, uint64_t policy) {
    if (o1) st_pair(p, v, policy);
    else if (o0) st_one(p, lo_of(v), policy);
}

template <typename Idx>
__device__ __forceinline__ void load_class_pair(const Idx* p, unsigned& a, unsigned& b);
template <>
__device__ __forceinline__ void load_class_pair<uint16_t>(const uint16_t* p, unsigned& a, unsigned& b) {
    const unsigned v = *reinterpret_cast<const unsigned*>(p);
    a = v & 0xffffu, b = v >> 16;
}
template <>
__device__ __forceinline__ void load_class_pair<uint32_t>(const uint32_t* p, unsigned& a, unsigned& b) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    a = v.x, b = v.y;
}

// Absorber coefficients (e^-x, dt phi) of a pair from the table entries ia, ib (ia alone where both
// cells of every lane of the warp share their x depth class).
__device__ __forceinline__ void coef_pair(const YeeArgs& a, int ia, int ib, bool same, pair_t& decay, pair_t& gain) {
    const float2 ka = __ldg(a.pml_coef + ia);
    float2 kb = ka;
    if (!same) kb = __ldg(a.pml_coef + ib);
    decay = pk(ka.x, kb.x), gain = pk(ka.y, kb.y);
}

// E^{n+1} of one cell from its curl (update_E.comp:41-64).
__device__ __forceinline__ void e_update(const YeeArgs& a, float& ex, float& ey, float& ez, float cx, float cy,
                                         float cz, unsigned c, bool inp, int R1, int R2, int R4, int iz, int hz, int x,
                                         int y, int z, int scene) {
    if (!inp) {
        const float4 t0 = __ldg(a.tabE + 2 * c), t1 = __ldg(a.tabE + 2 * c + 1);
        ex = t0.x * ex + t0.w * cx;
        ey = t0.y * ey + t1.x * cy;
        ez = t0.z * ez + t1.y * cz;
    } else if (c == 0) {
        const float2 kx = __ldg(a.pml_coef + R2 + iz), ky = __ldg(a.pml_coef + R1 + iz),
                     kz = __ldg(a.pml_coef + R4 + hz);
        ex = kx.x * ex + kx.y * cx;
        ey = ky.x * ey + ky.y * cy;
        ez = kz.x * ez + kz.y * cz;
    } else {
        // a non-vacuum edge material inside the absorber (update_E.comp:51-64), the x / y profiles
        // those of the cell's scene: e_cell's arithmetic
        const float4 m0 = __ldg(a.tabM + 2 * c), m1 = __ldg(a.tabM + 2 * c + 1);
        const float* pxy = a.pml_xy + (long long)scene * a.pml_xy_scene;
        const int SX = a.pml_xy_stride, S = a.pml_stride;
        const float ix = __ldg(pxy + x), iy = __ldg(pxy + SX + y), izv = __ldg(a.pml + 2 * S + z);
        const float hx = __ldg(pxy + 3 * SX + x), hy = __ldg(pxy + 4 * SX + y), hzv = __ldg(a.pml + 5 * S + z);
        ex = e_pml(ex, cx, m0.x + ((hx + iy) + izv), m0.w, a.dt);
        ey = e_pml(ey, cy, m0.y + ((ix + hy) + izv), m1.x, a.dt);
        ez = e_pml(ez, cz, m0.z + ((ix + iy) + hzv), m1.y, a.dt);
    }
}

// Schedule of the persistent pair kernel: work items are (z chunk, tile) pairs, chunk-major. CTA b
// starts with item b; the later ones are handed out in order by a ticket counter. Items in progress
// at any moment are a window of consecutive tiles at nearly the same z, so the halos that
// neighbouring tiles share are L2 hits; a static assignment lets slow CTAs (absorber columns) drift
// planes apart from their neighbours. work[0] counts tickets, work[1] the CTAs that have left: the
// last to leave, also after a wait that ran out, clears both, so every launch starts at zero.
struct PairSched {
    int tiles_x;  // tiles along x
    int tiles;    // tiles per z chunk
    int items;    // tiles * z chunks
    int zc;       // planes per z chunk
    unsigned long long* work;
    const int4* tab;  // a stack of scenes with their own cross-sections: the items themselves
};

struct PairItem {
    int x0, y0, zs, ze, zstart, scene;
};

template <int XT, int ROWS>
__device__ __forceinline__ PairItem pair_item(const PairSched& ps, int nz, int item) {
    PairItem it;
    if (ps.tab) {
        const int4 t = __ldg(ps.tab + item);
        it.x0 = t.x & 0xffff, it.y0 = (int)((unsigned)t.x >> 16), it.zs = t.y, it.ze = t.z, it.scene = t.w;
    } else {
        const int c = item / ps.tiles, t = item - c * ps.tiles;
        it.x0 = (t % ps.tiles_x) * XT;
        it.y0 = (t / ps.tiles_x) * ROWS;
        it.zs = c * ps.zc;
        it.ze = min(nz, it.zs + ps.zc);
        it.scene = 0;
    }
    it.zstart = it.zs > 0 ? it.zs - 1 : 0;  // a chunk above z = 0 first rebuilds B^{n+1/2}(zs-1)
    return it;
}

// Places of the depth classes of column (px, py) in a z plane of the table: r1 is (ix, hy), r2 (hx, iy),
// r3 (hx, hy), r4 (ix, iy).
struct PmlRows {
    int r1, r2, r3, r4;
};
__device__ __forceinline__ PmlRows pml_rows(const unsigned char* pcx, int SX, int K, int px, int py) {
    const int ix = __ldg(pcx + px), iy = __ldg(pcx + SX + py), hx = __ldg(pcx + 3 * SX + px),
              hy = __ldg(pcx + 4 * SX + py);
    return {hy * K + ix, iy * K + hx, hy * K + hx, iy * K + ix};
}

// A plane's absorber data, packed on the host: bit 0 in the absorber, bits 8-15 the integer depth
// class, bits 16-23 the half-integer one; here as the table planes of those classes.
__device__ __forceinline__ int z_iz(unsigned v, int K) { return (int)((v >> 8) & 0xff) * K * K; }
__device__ __forceinline__ int z_hz(unsigned v, int K) { return (int)((v >> 16) & 0xff) * K * K; }

template <int TY>
__device__ __forceinline__ void plane_sync() {  // every warp of the CTA, once per plane
    asm volatile("bar.sync 1, %0;" ::"n"(32 * (TY + 2)) : "memory");
}

// The CTA's loads form one sequence over its items: for each item, planes zstart .. ze (plane ze
// is read as the "z+1" neighbour of the last plane; ze = nz reads TMA zeros). Load j goes to ring
// stage j % STAGES and completes phase (j / STAGES) & 1 of that stage's mbarrier. The ring runs
// on across item boundaries, so the pipeline never drains inside a launch. The leader (lane 0 of
// warp TY+1) takes the next item when its loads near it and posts the item number in a small
// shared ring that the other warps read at their item boundary (always at least one barrier later).
// 64 x 4 tiles: three 192-thread CTAs per SM; 64 x 8 and 32 x 16: two 320-thread CTAs; 64 x 16: one 576-thread
// CTA. Registers are allocated per SM quadrant and 18-20 warps put 5 warps on one quadrant: 96
// registers at most.
template <int TY, typename Idx, int XL>
__global__ void __launch_bounds__(32 * (TY + 2), Layout2<TY, Idx, XL>::CTAS)
    yee_tma2(const __grid_constant__ CUtensorMap te, const __grid_constant__ CUtensorMap tb,
             const __grid_constant__ CUtensorMap tcls, YeeArgs a, PairSched ps, unsigned* err) {
    static_assert(TY == 4 || TY == 8 || TY == 16, "register budget assumes 6, 10 or 18 warps per CTA");
    using Lay = Layout2<TY, Idx, XL>;
    static_assert(XL == 32 || XL == 16, "a warp holds one row or two");
    constexpr int S_ = Lay::STAGES, ROWS = Lay::ROWS;
    constexpr int EPF = Lay::EP / 4, BPF = Lay::BP / 4, W = Lay::W, SBC = (ROWS + 1) * W;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + Lay::BAR_OFF);
    float* sB = reinterpret_cast<float*>(smem + Lay::SB_OFF);
    volatile int* queue = reinterpret_cast<volatile int*>(smem + Lay::QUEUE_OFF);  // item of ordinal n at [n & 7]
    volatile int* stop = reinterpret_cast<volatile int*>(smem + Lay::STOP_OFF);

    const int lane = threadIdx.x, warp = threadIdx.y;
    const int L = a.L, K = a.pml_K, SX = a.pml_xy_stride;
    if (warp == TY + 1 && lane == 0) {
        for (int s = 0; s < S_; ++s) mbar_init(bars + s, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        queue[0] = blockIdx.x;
        *stop = -1;
    }
    __syncthreads();
    chain_wait();
    chain_next();

    // the absorber of an item's scene (common.glsl:40-43 with the scene's own nx, ny)
    auto scene_size = [&](int scene, int& snx, int& sny) {
        snx = a.nx, sny = a.ny;
        if (a.scene_xy) {
            const int2 d = __ldg(a.scene_xy + scene);
            snx = d.x, sny = d.y;
        }
    };

    if (warp == TY + 1) {
        // ---- the copies (lane 0) ----
        const bool leader = lane == 0;
        int p_x = 0, p_y = 0, p_z = 0, p_end = -1;  // the next load: its tile and plane, the item's last plane
        int issued = 0, waited = -1, p_ord = 0;
        bool more = true;
        unsigned long long ticket = 0;
        auto seek = [&](int item) {
            const PairItem it = pair_item<2 * XL, Lay::ROWS>(ps, a.nz, item);
            p_x = it.x0 - 4, p_y = it.y0 - 1, p_z = it.zstart, p_end = it.ze;
        };
        auto issue_upto = [&](int last) {  // issue loads up to index `last` while the sequence lasts
            while (issued <= last && more) {
                unsigned char* st = smem + (issued % S_) * Lay::STAGE;
                uint64_t* bar = bars + issued % S_;
                mbar_expect_tx(bar, Lay::TX_BYTES);
                tma_load_3comp(st + Lay::E_OFF, &te, p_x, p_y, p_z, bar);
                tma_load_3comp(st + Lay::B_OFF, &tb, p_x, p_y, p_z, bar);
                tma_load_3d(st + Lay::C_OFF, &tcls, p_x - Lay::DC, p_y, p_z, bar);
                ++issued;
                // the ticket of the next item is drawn one load ahead (every item has at least two
                // loads), so its round trip to L2 hides behind that load's plane
                if (p_z == p_end - 1) ticket = atomicAdd(ps.work, 1ull);
                if (++p_z > p_end) {
                    const int left = ps.items - (int)gridDim.x;  // items handed out by ticket
                    const int next = ticket < (unsigned long long)left ? (int)gridDim.x + (int)ticket : -1;
                    queue[++p_ord & 7] = next;
                    more = next >= 0;
                    if (more) seek(next);
                }
            }
        };
        auto wait_upto = [&](int last) {  // false if a load did not complete within the bound
            bool ok = true;
            while (ok && waited < last) {
                ++waited;
                ok = mbar_wait(bars + waited % S_, (waited / S_) & 1, a.wait_polls);
            }
            return ok;
        };
        // the CTA leaves: on an expired wait record the error and give every copy still in flight
        // (from the load whose wait ran out on) a bounded time to land before the CTA's shared
        // memory goes; then count the CTA out
        auto leave = [&](bool failed) {
            if (!leader) return;
            if (failed) {
                atomicOr(err, 1u);
                for (int w = waited < 0 ? 0 : waited; w < issued; ++w) mbar_wait(bars + w % S_, (w / S_) & 1);
            }
            __threadfence();  // this CTA's tickets before its count
            if (atomicAdd(ps.work + 1, 1ull) == (unsigned long long)gridDim.x - 1) ps.work[0] = 0, ps.work[1] = 0;
        };
        if (leader) {
            seek(blockIdx.x);
            issue_upto(S_ - 1);
            if (!wait_upto(1)) *stop = 0;  // the first iteration reads loads 0 and 1
        }
        plane_sync<TY>();
        if (*stop == 0) return leave(true);
        int k = 0, iter = 0;
        for (int ord = 0, item = queue[0]; item >= 0; item = queue[++ord & 7]) {
            const PairItem it = pair_item<2 * XL, Lay::ROWS>(ps, a.nz, item);
            for (int z = it.zstart; z < it.ze; ++z, ++k, ++iter) {
                // the next iteration reads loads k+1, k+2 (or k+2, k+3 at the start of the next item,
                // which was taken when the last load of this one was issued)
                if (leader) {
                    const int need = z + 1 < it.ze ? k + 2 : (queue[(ord + 1) & 7] < 0 ? -1 : k + 3);
                    if (!wait_upto(need)) *stop = iter + 1;
                }
                plane_sync<TY>();
                if (*stop == iter + 1) return leave(true);
                // every warp is past its reads of loads <= k: refill up to k + STAGES
                if (leader) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    issue_upto(k + S_);
                }
            }
            ++k;  // the item's last load (plane ze) was only read as the z+1 neighbour
        }
        return leave(false);
    }

    // The word names the barrier (0: this one, iter + 1: iteration iter's) after which all leave: a
    // warp that is late to read it after one barrier may already see what the leader found before the
    // next, and has to arrive there with the others.
    plane_sync<TY>();
    if (*stop == 0) return;
    // box element of the own / halo-row pair (E, B and 32-bit class boxes share it; the 16-bit class
    // box is DC elements further); B tile slot = element - 2
    const bool row = warp == TY;  // the halo warp; its row: Bx, Bz of (xa, y0-1), (xa+1, y0-1)
    // two rows a warp: the halo warp's upper half repeats its lower half
    const int lx = lane % XL, mine = warp * (32 / XL) + lane / XL;  // the pair's place in its row, the own row
    const int me = (row ? 0 : mine + 1) * W + 2 * lx + 4;
    const pair_t dt2 = pk(a.dt, a.dt), mz = pk(a.minus_zero, a.minus_zero);
    int k = 0;     // load index of the current iteration's plane z
    int iter = 0;  // iteration counter: parity selects the B tile buffer
    for (int ord = 0, item = queue[0]; item >= 0; item = queue[++ord & 7]) {
        const PairItem it = pair_item<2 * XL, Lay::ROWS>(ps, a.nz, item);
        int snx, sny;
        scene_size(it.scene, snx, sny);
        // cells outside the item's scene (a ragged stack's frozen cells) are neither updated nor
        // written: they keep their initial 0 in both field generations
        const int xa = it.x0 + 2 * lx;
        const int y = row ? it.y0 - 1 : it.y0 + mine;
        const bool rowok = row ? it.y0 > 0 : y < sny;
        const bool o0 = rowok && xa < snx, o1 = rowok && xa + 1 < snx;
        const unsigned char* pcx = a.pml_cls_xy + (long long)it.scene * a.pml_xy_scene;
        PmlRows A{}, B{};
        if (o0) A = pml_rows(pcx, SX, K, xa, y);
        if (o1) B = pml_rows(pcx, SX, K, xa + 1, y);
        auto inxy = [&](int px) { return px < L || y < L || px >= snx - (L + 1) || y >= sny - (L + 1); };
        const bool pxy0 = o0 && inxy(xa), pxy1 = o1 && inxy(xa + 1);
        const bool pmlrow = __any_sync(0xffffffffu, pxy0 || pxy1);  // uniform: the warp's row touches the layer
        const bool same = __all_sync(0xffffffffu, A.r1 == B.r1 && A.r2 == B.r2 && A.r3 == B.r3 && A.r4 == B.r4);
        unsigned zi = __ldg(a.pml_zi + it.zstart);

        if (row) {
            // the -x halo column too: By, Bz of (x0-1, y0 + lane), lanes 0 .. ROWS-1 (the others repeat the
            // last one). Its cells always read the table: (1, dt) outside the layer
            const int cl = min(lane, ROWS - 1), ce = (cl + 1) * W + 3;
            const bool clive = it.x0 > 0 && it.y0 + cl < sny;
            PmlRows C{};
            if (clive) C = pml_rows(pcx, SX, K, it.x0 - 1, it.y0 + cl);
            for (int z = it.zstart; z < it.ze; ++z, ++k, ++iter) {
                const unsigned char* st = smem + (k % S_) * Lay::STAGE;
                const unsigned zn = __ldg(a.pml_zi + min(z + 1, a.nz - 1));
                if (z >= it.zs) {
                    float* sb = sB + (iter & 1) * 3 * SBC - 2;
                    const float* Es = reinterpret_cast<const float*>(st + Lay::E_OFF);
                    const float* E1 = reinterpret_cast<const float*>(smem + ((k + 1) % S_) * Lay::STAGE + Lay::E_OFF);
                    const float* Bs = reinterpret_cast<const float*>(st + Lay::B_OFF);
                    const Idx* Cs = reinterpret_cast<const Idx*>(st + Lay::C_OFF) + Lay::DC;
                    {
                        const unsigned hc = (unsigned)Cs[ce];
                        const float2 ky = __ldg(a.pml_coef + C.r2 + z_hz(zi, K)), kz = __ldg(a.pml_coef + C.r3 + z_iz(zi, K));
                        const float f0x = Es[ce], f0y = Es[EPF + ce], f0z = Es[2 * EPF + ce];
                        float t0y = E1[ce] - f0x, t0z = Es[EPF + ce + 1] - f0y, t1y = Es[2 * EPF + ce + 1] - f0z,
                              t1z = Es[ce + W] - f0x;
                        if (__any_sync(0xffffffffu, hc >= a.wire_start)) {
                            const float4 w0 = __ldg(a.tabW + 2 * hc), w1 = __ldg(a.tabW + 2 * hc + 1);
                            t0y = t0y * w0.y, t0z = t0z * w0.z, t1y = t1y * w1.x, t1z = t1z * w1.y;
                        }
                        const float hby = ky.x * Bs[BPF + ce] - ky.y * (t0y - t1y);
                        const float hbz = kz.x * Bs[2 * BPF + ce] - kz.y * (t0z - t1z);
                        if (lane < ROWS) sb[SBC + ce] = clive ? hby : 0.0f, sb[2 * SBC + ce] = clive ? hbz : 0.0f;
                    }
                    pair_t hx2 = 0, hz2 = 0;  // B below the lower face is 0
                    if (rowok) {
                        unsigned ha, hb;
                        load_class_pair<Idx>(Cs + me, ha, hb);
                        const pair_t f0x = lds2(Es + me), f0y = lds2(Es + EPF + me), f0z = lds2(Es + 2 * EPF + me);
                        pair_t t0x = sub2(lds2(Es + 2 * EPF + me + W), f0z), t1x = sub2(lds2(E1 + EPF + me), f0y);
                        pair_t t0z = sub2(pk(hi_of(f0y), Es[EPF + me + 2]), f0y), t1z = sub2(lds2(Es + me + W), f0x);
                        if (__any_sync(0xffffffffu, max(ha, hb) >= a.wire_start)) {
                            const float4 w0 = __ldg(a.tabW + 2 * ha), w1 = __ldg(a.tabW + 2 * ha + 1);
                            const float4 v0 = __ldg(a.tabW + 2 * hb), v1 = __ldg(a.tabW + 2 * hb + 1);
                            t0x = mul2(t0x, pk(w0.x, v0.x), mz), t0z = mul2(t0z, pk(w0.z, v0.z), mz);
                            t1x = mul2(t1x, pk(w0.w, v0.w), mz), t1z = mul2(t1z, pk(w1.y, v1.y), mz);
                        }
                        const pair_t cx = sub2(t0x, t1x), cz = sub2(t0z, t1z);
                        hx2 = lds2(Bs + me), hz2 = lds2(Bs + 2 * BPF + me);
                        if (pmlrow || (zi & 1)) {
                            pair_t d, g;
                            coef_pair(a, A.r1 + z_hz(zi, K), B.r1 + z_hz(zi, K), same, d, g);
                            hx2 = sub2(mul2(d, hx2, mz), mul2(g, cx, mz));
                            coef_pair(a, A.r3 + z_iz(zi, K), B.r3 + z_iz(zi, K), same, d, g);
                            hz2 = sub2(mul2(d, hz2, mz), mul2(g, cz, mz));
                        } else {
                            hx2 = sub2(hx2, mul2(dt2, cx, mz));
                            hz2 = sub2(hz2, mul2(dt2, cz, mz));
                        }
                    }
                    sts2(sb + me, hx2);
                    sts2(sb + 2 * SBC + me, hz2);
                }
                plane_sync<TY>();
                if (*stop == iter + 1) return;
                zi = zn;
            }
            ++k;
            continue;
        }

        const bool full = __all_sync(0xffffffffu, o1);
        ulonglong2* coef = reinterpret_cast<ulonglong2*>(smem + Lay::COEF_OFF) + warp * 32 + lane;  // + entry * 32 TY
        if (pmlrow) {  // the thread's own slots: no other thread reads them
            pair_t d, g;
            coef_pair(a, A.r1, B.r1, same, d, g), coef[0] = make_ulonglong2(d, g);
            coef_pair(a, A.r2, B.r2, same, d, g), coef[32 * TY] = make_ulonglong2(d, g);
            coef_pair(a, A.r3, B.r3, same, d, g), coef[64 * TY] = make_ulonglong2(d, g);
            coef_pair(a, A.r4, B.r4, same, d, g), coef[96 * TY] = make_ulonglong2(d, g);
        }
        long long off = (long long)it.zstart * a.plane + (long long)y * a.pitch + xa;
        pair_t bpx = 0, bpy = 0;  // B^{n+1/2}(z-1).x, .y of the pair
        const float* E0 = reinterpret_cast<const float*>(smem + (k % S_) * Lay::STAGE + Lay::E_OFF) + me;
        pair_t e0x = lds2(E0), e0y = lds2(E0 + EPF);
        for (int z = it.zstart; z < it.ze; ++z, ++k, ++iter, off += a.plane) {
            const unsigned char* st = smem + (k % S_) * Lay::STAGE;
            const bool emit = z >= it.zs;
            float* sb = sB + (iter & 1) * 3 * SBC - 2 + me;  // the pair's slot; indexed by box element
            const unsigned zn = __ldg(a.pml_zi + min(z + 1, a.nz - 1));
            const float* Es = reinterpret_cast<const float*>(st + Lay::E_OFF) + me;
            const float* E1 = reinterpret_cast<const float*>(smem + ((k + 1) % S_) * Lay::STAGE + Lay::E_OFF) + me;
            const float* Bs = reinterpret_cast<const float*>(st + Lay::B_OFF) + me;
            // update_B.comp:35-67 for both cells (halo values beyond the grid are TMA zeros)
            unsigned ca, cb;
            load_class_pair<Idx>(reinterpret_cast<const Idx*>(st + Lay::C_OFF) + Lay::DC + me, ca, cb);
            const pair_t e0z = lds2(Es + 2 * EPF);
            const pair_t ezx = lds2(E1), ezy = lds2(E1 + EPF);  // E(z+1)
            pair_t bx = lds2(Bs), by = lds2(Bs + BPF), bz = lds2(Bs + 2 * BPF);
            pair_t t0x = sub2(lds2(Es + 2 * EPF + W), e0z), t1x = sub2(ezy, e0y);
            pair_t t0y = sub2(ezx, e0x), t1y = sub2(pk(hi_of(e0z), Es[2 * EPF + 2]), e0z);
            pair_t t0z = sub2(pk(hi_of(e0y), Es[EPF + 2]), e0y), t1z = sub2(lds2(Es + W), e0x);
            const bool mat = __any_sync(0xffffffffu, (ca | cb) != 0);  // uniform: a non-vacuum cell in the row
            if (mat && __any_sync(0xffffffffu, max(ca, cb) >= a.wire_start)) {
                // thin-wire factors; the entries of other classes are 1
                const float4 w0 = __ldg(a.tabW + 2 * ca), w1 = __ldg(a.tabW + 2 * ca + 1);
                const float4 v0 = __ldg(a.tabW + 2 * cb), v1 = __ldg(a.tabW + 2 * cb + 1);
                t0x = mul2(t0x, pk(w0.x, v0.x), mz), t0y = mul2(t0y, pk(w0.y, v0.y), mz), t0z = mul2(t0z, pk(w0.z, v0.z), mz);
                t1x = mul2(t1x, pk(w0.w, v0.w), mz), t1y = mul2(t1y, pk(w1.x, v1.x), mz), t1z = mul2(t1z, pk(w1.y, v1.y), mz);
            }
            const bool pml = pmlrow || (zi & 1);
            {
                const pair_t cx = sub2(t0x, t1x), cy = sub2(t0y, t1y), cz = sub2(t0z, t1z);
                if (!(zi & 1)) {
                    if (pmlrow) {
                        const ulonglong2 k1 = coef[0], k2 = coef[32 * TY], k3 = coef[64 * TY];
                        bx = sub2(mul2(k1.x, bx, mz), mul2(k1.y, cx, mz));
                        by = sub2(mul2(k2.x, by, mz), mul2(k2.y, cy, mz));
                        bz = sub2(mul2(k3.x, bz, mz), mul2(k3.y, cz, mz));
                    } else {
                        bx = sub2(bx, mul2(dt2, cx, mz));
                        by = sub2(by, mul2(dt2, cy, mz));
                        bz = sub2(bz, mul2(dt2, cz, mz));
                    }
                } else {
                    pair_t d, g;
                    coef_pair(a, A.r1 + z_hz(zi, K), B.r1 + z_hz(zi, K), same, d, g);
                    bx = sub2(mul2(d, bx, mz), mul2(g, cx, mz));
                    coef_pair(a, A.r2 + z_hz(zi, K), B.r2 + z_hz(zi, K), same, d, g);
                    by = sub2(mul2(d, by, mz), mul2(g, cy, mz));
                    coef_pair(a, A.r3 + z_iz(zi, K), B.r3 + z_iz(zi, K), same, d, g);
                    bz = sub2(mul2(d, bz, mz), mul2(g, cz, mz));
                }
            }
            sts2(sb, bx);
            sts2(sb + SBC, by);
            sts2(sb + 2 * SBC, bz);
            if (emit) {
                const uint64_t evict_first = evict_first_policy();
                if (full) {
                    st_pair(a.nbx + off, bx, evict_first);
                    st_pair(a.nby + off, by, evict_first);
                    st_pair(a.nbz + off, bz, evict_first);
                } else {
                    st_cells(a.nbx + off, bx, o0, o1, evict_first);
                    st_cells(a.nby + off, by, o0, o1, evict_first);
                    st_cells(a.nbz + off, bz, o0, o1, evict_first);
                }
            }
            plane_sync<TY>();
            const bool quit = *stop == iter + 1;
            if (emit) {
                // update_E.comp:41-64 for both cells
                const float bxm_y = sb[SBC - 1], bxm_z = sb[2 * SBC - 1];                 // B(xa-1).y, .z
                const pair_t bym_x = lds2(sb - W), bym_z = lds2(sb + 2 * SBC - W);          // B(y-1).x, .z
                const pair_t cx = sub2(sub2(bz, bym_z), sub2(by, bpy));
                const pair_t cy = sub2(sub2(bx, bpx), sub2(bz, pk(bxm_z, lo_of(bz))));
                const pair_t cz = sub2(sub2(by, pk(bxm_y, lo_of(by))), sub2(bx, bym_x));
                pair_t ex, ey, ez;
                if (!pml) {
                    if (!mat) {  // vacuum: ca = 1 and cb = dt exactly, so 1 * e + dt * curl == e + dt * curl
                        ex = add2(e0x, mul2(dt2, cx, mz));
                        ey = add2(e0y, mul2(dt2, cy, mz));
                        ez = add2(e0z, mul2(dt2, cz, mz));
                    } else {
                        const float4 p0 = __ldg(a.tabE + 2 * ca), p1 = __ldg(a.tabE + 2 * ca + 1);
                        const float4 q0 = __ldg(a.tabE + 2 * cb), q1 = __ldg(a.tabE + 2 * cb + 1);
                        ex = add2(mul2(pk(p0.x, q0.x), e0x, mz), mul2(pk(p0.w, q0.w), cx, mz));
                        ey = add2(mul2(pk(p0.y, q0.y), e0y, mz), mul2(pk(p1.x, q1.x), cy, mz));
                        ez = add2(mul2(pk(p0.z, q0.z), e0z, mz), mul2(pk(p1.y, q1.y), cz, mz));
                    }
                } else if (!mat && !(zi & 1)) {
                    const ulonglong2 k2 = coef[32 * TY], k1 = coef[0], k4 = coef[96 * TY];
                    ex = add2(mul2(k2.x, e0x, mz), mul2(k2.y, cx, mz));
                    ey = add2(mul2(k1.x, e0y, mz), mul2(k1.y, cy, mz));
                    ez = add2(mul2(k4.x, e0z, mz), mul2(k4.y, cz, mz));
                } else if (!mat) {
                    pair_t d, g;
                    coef_pair(a, A.r2 + z_iz(zi, K), B.r2 + z_iz(zi, K), same, d, g);
                    ex = add2(mul2(d, e0x, mz), mul2(g, cx, mz));
                    coef_pair(a, A.r1 + z_iz(zi, K), B.r1 + z_iz(zi, K), same, d, g);
                    ey = add2(mul2(d, e0y, mz), mul2(g, cy, mz));
                    coef_pair(a, A.r4 + z_hz(zi, K), B.r4 + z_hz(zi, K), same, d, g);
                    ez = add2(mul2(d, e0z, mz), mul2(g, cz, mz));
                } else {
                    float x0 = lo_of(e0x), y0 = lo_of(e0y), z0 = lo_of(e0z), x1 = hi_of(e0x), y1 = hi_of(e0y),
                          z1 = hi_of(e0z);
                    if (o0)
                        e_update(a, x0, y0, z0, lo_of(cx), lo_of(cy), lo_of(cz), ca, pxy0 || (zi & 1), A.r1, A.r2, A.r4,
                                 z_iz(zi, K), z_hz(zi, K), xa, y, z, it.scene);
                    if (o1)
                        e_update(a, x1, y1, z1, hi_of(cx), hi_of(cy), hi_of(cz), cb, pxy1 || (zi & 1), B.r1, B.r2, B.r4,
                                 z_iz(zi, K), z_hz(zi, K), xa + 1, y, z, it.scene);
                    ex = pk(x0, x1), ey = pk(y0, y1), ez = pk(z0, z1);
                }
                const uint64_t evict_first = evict_first_policy();
                if (full) {
                    st_pair(a.nex + off, ex, evict_first);
                    st_pair(a.ney + off, ey, evict_first);
                    st_pair(a.nez + off, ez, evict_first);
                } else {
                    st_cells(a.nex + off, ex, o0, o1, evict_first);
                    st_cells(a.ney + off, ey, o0, o1, evict_first);
                    st_cells(a.nez + off, ez, o0, o1, evict_first);
                }
            }
            if (quit) return;
            bpx = bx, bpy = by;
            e0x = ezx, e0y = ezy;
            zi = zn;
        }
        ++k;  // the item's last load (plane ze) was only read as the z+1 neighbour
    }
}

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
    static const EncodeFn fn = [] {  // initialised once, thread-safe
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeFn>(p);
        return (EncodeFn) nullptr;
    }();
    return fn;
}

std::mutex g_launch_setup;  // the launchers' one-time attribute set-up (grids may step from several threads)

bool encode(CUtensorMap* m, CUtensorMapDataType type, int elem, const void* base, const YeeArgs& a, int box_w,
            int box_h) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)a.nx, (cuuint64_t)a.ny, (cuuint64_t)a.nz};
    const cuuint64_t strides[2] = {(cuuint64_t)a.pitch * elem, (cuuint64_t)a.plane * elem};
    const cuuint32_t box[3] = {(cuuint32_t)box_w, (cuuint32_t)box_h, 1};
    const cuuint32_t estr[3] = {1, 1, 1};
    return fn(m, type, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// tiling modes: 8, 16 = 32 x TY tiles of single cells (yee_tma); 32, 64, 128 = 64 x 4, 64 x 8 and 64 x 16
// tiles of cell pairs, kNarrowPairTiles = 32 x 16 (yee_tma2)
// The three component arrays from base, `comp` floats apart, as one map: the copies of the pair tiles.
bool encode3(CUtensorMap* m, const float* base, long long comp, const YeeArgs& a, int box_w, int box_h) {
    EncodeFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)a.nx, (cuuint64_t)a.ny, (cuuint64_t)a.nz, 3};
    const cuuint64_t strides[3] = {(cuuint64_t)a.pitch * 4, (cuuint64_t)a.plane * 4, (cuuint64_t)comp * 4};
    const cuuint32_t box[4] = {(cuuint32_t)box_w, (cuuint32_t)box_h, 1, 3};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float*>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool narrow_tiles(const YeeArgs& a) { return a.tile_rows == kNarrowPairTiles; }
int tile_rows(const YeeArgs& a) {
    return a.tile_rows == 16 || a.tile_rows == 128 || narrow_tiles(a) ? 16 : (a.tile_rows == 32 ? 4 : 8);
}
bool pair_tiles(const YeeArgs& a) {
    return a.tile_rows == 32 || a.tile_rows == 64 || a.tile_rows == 128 || narrow_tiles(a);
}

template <int TY, typename Idx>
bool launch_t(const YeeArgs& a, const TmaMaps* m, int gen, unsigned* err, const Chain& s) {
    using Lay = Layout<TY, Idx>;
    static bool configured = false;
    {
        std::lock_guard<std::mutex> lk(g_launch_setup);
        if (!configured) {
            if (cudaFuncSetAttribute(yee_tma<TY, Idx>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::SMEM) !=
                cudaSuccess)
                return false;
            configured = true;
        }
    }
    const dim3 grid((a.nx + 31) / 32, (a.ny + TY - 1) / TY, (a.nz + a.zchunk - 1) / a.zchunk);
    launch_chained(s, yee_tma<TY, Idx>, grid, dim3(32, TY + 1), Lay::SMEM, m->e[gen][0], m->e[gen][1], m->e[gen][2],
                   m->b[gen][0], m->b[gen][1], m->b[gen][2], m->cls, a, err);
    return true;
}

// Chooses the z chunk length of the persistent schedule: the CTA with the most items bounds the
// launch, and every chunk above z = 0 re-reads one plane, so minimise ceil(items / G) * (zc + 1).
// Items differ in cost (a tile with absorber or material cells takes longer per plane), and the
// ticket schedule evens them out only when every CTA takes several: the chunk length is chosen among
// those giving at least kItemsPerCta items per CTA, as far as chunks of kMinBalancedPlanes planes
// allow (shorter chunks would re-read too many planes: every chunk above z = 0 re-reads one).
constexpr int kItemsPerCta = 4;
constexpr int kMinBalancedPlanes = 16;

PairSched pair_schedule(const YeeArgs& a, int xt, int rows, int G) {
    PairSched ps;
    ps.tiles_x = (a.nx + xt - 1) / xt;
    ps.tiles = ps.tiles_x * ((a.ny + rows - 1) / rows);
    const int max_chunks = std::max(1, a.nz / 4);
    const long long want = std::min((long long)kItemsPerCta * G,
                                    (long long)std::max(1, a.nz / kMinBalancedPlanes) * ps.tiles);
    long long best = -1;
    for (int chunks = 1; chunks <= max_chunks; ++chunks) {
        const int zc = (a.nz + chunks - 1) / chunks;
        const int n = (a.nz + zc - 1) / zc;
        const long long items = (long long)n * ps.tiles;
        if (items < want) continue;
        const long long cost = (items + G - 1) / G * (zc + (n > 1 ? 1 : 0));
        if (best < 0 || cost < best) best = cost, ps.zc = zc, ps.items = (int)items;
    }
    if (best < 0) {  // no chunk count reaches `want` exactly (zc rounding): the finest split
        ps.zc = (a.nz + max_chunks - 1) / max_chunks;
        ps.items = (int)((long long)((a.nz + ps.zc - 1) / ps.zc) * ps.tiles);
    }
    return ps;
}

// Grids too small for that balance (the rule above leaves fewer than kItemsPerCta items per CTA). An
// item costs its planes plus about two and a half (the re-read plane and its start); r = items / G
// rounds of them take a time between r (items of unequal cost even out over the tickets) and the
// whole rounds, and the last item of a CTA sticks out by most of its length:
//   cost = (zc + 2.5) (r / 2 + ceil(r) / 2 + 3/4).
// Measured over thirteen sizes from 48 x 48 x 48 to 320 x 300 x 280 and chunks of 1 to 48 planes, the
// chunk it picks is within 2.6 % of the best one (worst 13 %): 48 x 48 x 48 one plane (13.0 us a step
// against 20.7 for the rule above), 211 x 147 x 93 eight (52.0 against 59.7), 192 x 192 x 128 eight
// (61.0 against 75.2).
void small_grid_schedule(PairSched& ps, int nz, int G) {
    double best = -1.0;
    for (int zc = 1; zc <= nz; ++zc) {
        const long long items = (long long)((nz + zc - 1) / zc) * ps.tiles;
        const double r = (double)items / G;
        const double cost = (zc + 2.5) * (0.5 * r + 0.5 * (double)((items + G - 1) / G) + 0.75);
        if (best < 0.0 || cost < best) best = cost, ps.zc = zc, ps.items = (int)items;
    }
}

// What is launched on a single grid: the first rule, or the second where it leaves fewer than kItemsPerCta items per CTA.
PairSched uniform_schedule(const YeeArgs& a, int xt, int rows, int G) {
    PairSched ps = pair_schedule(a, xt, rows, G);
    if (ps.items < kItemsPerCta * G) small_grid_schedule(ps, a.nz, G);
    return ps;
}

template <int TY, int XL, typename Idx>
bool launch_p(const YeeArgs& a, const TmaMaps* m, int gen, unsigned* err, const Chain& s) {
    using Lay = Layout2<TY, Idx, XL>;
    static int resident = 0, sms = 0;  // per process: one device model
    std::unique_lock<std::mutex> lk(g_launch_setup);
    if (!resident) {
        int dev = 0, smem_sm = 0;
        // shared-memory carveout for exactly the CTAs wanted per SM (two 64 x 8 or one 64 x 16): the
        // rest of the SM's 256 KB stays L1, which caches the per-class and absorber tables
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
            smem_sm <= 0 ||
            cudaFuncSetAttribute(yee_tma2<TY, Idx, XL>, cudaFuncAttributeMaxDynamicSharedMemorySize, Lay::SMEM) !=
                cudaSuccess ||
            cudaFuncSetAttribute(yee_tma2<TY, Idx, XL>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 std::min(100, (100 * Lay::CTAS * (Lay::SMEM + 1024) +
                                                smem_sm - 1) / smem_sm)) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, yee_tma2<TY, Idx, XL>, 32 * (TY + 2), Lay::SMEM) !=
                cudaSuccess ||
            resident < 1) {
            resident = 0;
            return false;
        }
    }
    lk.unlock();
    PairSched ps{};
    if (a.items) {
        ps.items = a.n_items;
        ps.tab = a.items;
    } else {
        ps = uniform_schedule(a, 2 * XL, Lay::ROWS, resident * sms);
        ps.tab = nullptr;
    }
    if (ps.items <= 0) return false;
    const int grid = std::min(ps.items, resident * sms);
    ps.work = a.work;
    launch_chained(s, yee_tma2<TY, Idx, XL>, grid, dim3(32, TY + 2), Lay::SMEM, m->e3[gen], m->b3[gen], m->cls, a, ps, err);
    return true;
}

}  // namespace

TmaMaps* tma_maps_create() { return new TmaMaps(); }
void tma_maps_destroy(TmaMaps* m) { delete m; }

bool tma_maps_encode(TmaMaps* m, int gen, const YeeArgs& a, bool wide) {
    const int ty = tile_rows(a);
    const bool pair = pair_tiles(a);
    const int pair_w = narrow_tiles(a) ? 40 : 72;
    const int cw16 = pair ? pair_w : 40, cw32 = pair ? pair_w : 36;
    bool ok = (a.pitch % 4) == 0;
    if (pair) {
        const long long comp = a.ey - a.ex;  // the six arrays of a generation lie one after the other
        ok = ok && a.ez - a.ex == 2 * comp && a.by - a.bx == comp && a.bz - a.bx == 2 * comp &&
             encode3(&m->e3[gen], a.ex, comp, a, pair_w, ty + 2) &&
             encode3(&m->b3[gen], a.bx, comp, a, pair_w, ty + 1);
    }
    const float* e[3] = {a.ex, a.ey, a.ez};
    const float* b[3] = {a.bx, a.by, a.bz};
    for (int c = 0; c < 3 && ok && !pair; ++c) {
        ok = encode(&m->e[gen][c], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, e[c], a, 40, ty + 2) &&
             encode(&m->b[gen][c], CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, b[c], a, 36, ty + 1);
    }
    if (ok)
        ok = wide ? encode(&m->cls, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, a.cls, a, cw32, ty + 1)
                  : encode(&m->cls, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, a.cls, a, cw16, ty + 1);
    m->ok[gen] = ok;
    m->cls_ok = ok;
    m->tiling = a.tile_rows;
    return ok;
}

bool tma_maps_ready(const TmaMaps* m, int gen) { return m && m->ok[gen] && m->cls_ok; }

void pair_schedule_shape(int nx, int ny, int nz, int ty, int g, int* zc, int* items) {
    YeeArgs a{};
    a.nx = nx, a.ny = ny, a.nz = nz;
    const PairSched ps = pair_schedule(a, 64, ty, g);
    *zc = ps.zc, *items = ps.items;
}

void pair_launch_shape(int nx, int ny, int nz, int xt, int ty, int g, int* zc, int* items) {
    YeeArgs a{};
    a.nx = nx, a.ny = ny, a.nz = nz;
    const PairSched ps = uniform_schedule(a, xt, ty, g);
    *zc = ps.zc, *items = ps.items;
}

std::vector<int4> ragged_items(const std::vector<int>& z0, const std::vector<int>& nx, const std::vector<int>& ny,
                               const std::vector<int>& nz, int ty, int g, int xt) {
    const size_t n = z0.size();
    std::vector<long long> tiles(n);
    int deepest = 1;
    for (size_t i = 0; i < n; ++i) {
        tiles[i] = (long long)((nx[i] + xt - 1) / xt) * ((ny[i] + ty - 1) / ty);
        deepest = std::max(deepest, nz[i]);
    }
    // one chunk length for every scene: the CTA with the most items bounds the launch, and every
    // chunk above a scene's first plane re-reads one plane
    // as pair_schedule: at least kItemsPerCta items per CTA where the scenes allow it
    long long finest = 0;
    for (size_t i = 0; i < n; ++i) finest += tiles[i] * std::max(1, nz[i] / kMinBalancedPlanes);
    const long long want = std::min((long long)kItemsPerCta * g, finest);
    int zc_best = std::min(deepest, 4);
    long long best = -1;
    for (int zc = std::min(deepest, 4); zc <= deepest; ++zc) {
        long long items = 0, extra = 0;
        for (size_t i = 0; i < n; ++i) {
            const long long c = (nz[i] + zc - 1) / zc;
            items += tiles[i] * c;
            extra += c > 1 ? 1 : 0;
        }
        if (items < want) continue;
        const long long cost = (items + g - 1) / g * (zc + (extra ? 1 : 0));
        if (best < 0 || cost < best) best = cost, zc_best = zc;
    }
    std::vector<int4> out;
    for (size_t i = 0; i < n; ++i) {
        const int tx = (nx[i] + xt - 1) / xt, tyn = (ny[i] + ty - 1) / ty;
        for (int zs = 0; zs < nz[i]; zs += zc_best)
            for (int t = 0; t < tx * tyn; ++t)
                out.push_back(make_int4((t % tx) * xt | ((t / tx) * ty) << 16, z0[i] + zs,
                                        z0[i] + std::min(nz[i], zs + zc_best), (int)i));
    }
    return out;
}

bool launch_yee_tma(const YeeArgs& a, const TmaMaps* m, int gen, bool wide, unsigned* err, const Chain& s) {
    if (!m || !m->ok[gen] || !m->cls_ok || m->tiling != a.tile_rows) return false;
    if (narrow_tiles(a))
        return wide ? launch_p<8, 16, uint32_t>(a, m, gen, err, s)
                    : launch_p<8, 16, uint16_t>(a, m, gen, err, s);
    if (pair_tiles(a) && tile_rows(a) == 16)
        return wide ? launch_p<16, 32, uint32_t>(a, m, gen, err, s)
                    : launch_p<16, 32, uint16_t>(a, m, gen, err, s);
    if (pair_tiles(a) && tile_rows(a) == 4)
        return wide ? launch_p<4, 32, uint32_t>(a, m, gen, err, s)
                    : launch_p<4, 32, uint16_t>(a, m, gen, err, s);
    if (pair_tiles(a))
        return wide ? launch_p<8, 32, uint32_t>(a, m, gen, err, s)
                    : launch_p<8, 32, uint16_t>(a, m, gen, err, s);
    if (tile_rows(a) == 16) return wide ? launch_t<16, uint32_t>(a, m, gen, err, s) : launch_t<16, uint16_t>(a, m, gen, err, s);
    return wide ? launch_t<8, uint32_t>(a, m, gen, err, s) : launch_t<8, uint16_t>(a, m, gen, err, s);
}

}  // namespace emlab
