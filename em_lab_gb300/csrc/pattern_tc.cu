// pattern_tc.cu - the far-field pattern of a Huygens box as per-face GEMMs on the tensor cores.
//
// The pattern sums of ntff_pattern.comp:45-110 over the box surface,
//   N(r) = sum_p J_p e^{+jk r.(p - c)},   L(r) = sum_p M_p e^{+jk r.(p - c)},
// with J = n x H w and M = -n x E w (w: the trapezoid edge weights), are separable on a face: its
// nodes form an (nu + 1) x (nv + 1) lattice at fixed a (the face normal axis), so
//   N_q(r) = e^{jk r_a p_a} sum_iu e^{jk r_u p_u(iu)} [ sum_iv e^{jk r_v p_v(iv)} F_q(iv, iu) ]
// for the four tangential fields F_q = J_u, J_v, M_u, M_v. The lattice lies symmetrically about the
// centre, so the rows at +-p_v fold into one term, cos(k r_v p_v) (F(+) + F(-)) + j sin(k r_v p_v) (F(+) -
// F(-)), and the bracket is a real GEMM over the folded rows for all directions: a row (cos, sin) per
// direction times columns (Fe re, -Fo im) and (Fe im, Fo re), K = nv + 1, N = 8 (nu + 1); half the
// products of the complex form. It runs on the tcgen05 tensor cores with every operand split into a
// BF16 high and low half (A_hi B_hi + A_lo B_hi + A_hi B_lo: about 16 significant bits per operand, FP32
// accumulation in tensor memory). |N_perp - r x L|^2 and the radiated power follow ntff_reduce.comp:19-39.
//
// One persistent kernel does everything for 128 directions of a frequency at a time, so that neither
// the twiddles nor the products ever leave the SM: the direction's rows of A are generated in shared
// memory (the faces share them: V runs along z on four faces and along y on two), B streams through a
// ring of bulk copies from tiles that a first kernel lays out in the tensor core's own layout, the
// products of 32 columns iu accumulate in one half of tensor memory while eight warps contract the
// other half with e^{jk r_u p_u} in registers, and the direction's result leaves as one number. Bound
// by the tensor pipe: 9.4 ms (8.5 ms in the kernel, 1.3 PFLOP/s of BF16 products, 0.70 of the measured
// peak) for 181 x 361 directions, 32 frequencies and 102872 nodes, against 147 ms with operands and
// products through global memory, plain-load staging and one complex GEMM per face and frequency.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "../../include/emlab.h"
#include "grid_state.h"
#include "twiddle.cuh"

using namespace emlab;

namespace {

constexpr int kDirs = 128;               // directions per tile: MMA M, TMEM lanes
constexpr int kCols = 32;                // columns iu per block: 8 MMA columns each (4 fields x re, im)
constexpr int kN = 8 * kCols;            // MMA N
constexpr int kKc = 32;                  // K of a B tile: 16 folded rows
constexpr int kTile = kN * kKc * 2;      // 16 KB
constexpr int kStages = 3;
constexpr int kMaxKc = 10;               // chunks of A held at once: 160 folded rows (longer faces in segments)
constexpr int kAPart = kDirs * kKc * 2;  // one chunk of A, high or low half
constexpr int kComputeWarps = 8, kThreads = 32 * (kComputeWarps + 2);
constexpr int kAOff = kStages * kTile, kCombineOff = kAOff + 2 * kMaxKc * kAPart;
constexpr int kBarOff = kCombineOff + kDirs * 12 * 4;
constexpr int kSmem = kBarOff + 256;
static_assert(kSmem <= 227 * 1024, "shared memory per CTA");

// A face's lattice and its tiles of B: `segs` segments of 16 kc folded rows (kc chunks of K),
// blocks of kCols columns iu; tile (segment, block, chunk, high / low) at `tile0` in that order.
struct Face {
    int nu1, nv1, segs, kc, blocks, first, tile0;
    float sign;
};
struct Box {
    Face f[6];
    float half[3];  // half extents: positions run from -half to +half on every axis
    int tiles;      // of a frequency
    int parts;      // power partial sums of a frequency
};

__host__ Box make_box(const int* b) {
    Box x{};
    for (int a = 0; a < 3; ++a) x.half[a] = 0.5f * (float)(b[3 + a] - b[a]);
    for (int f = 0; f < 6; ++f) {
        const int a = f >> 1, u = a == 0 ? 1 : 0, v = a == 2 ? 1 : 2;
        Face& q = x.f[f];
        q.nu1 = b[3 + u] - b[u] + 1, q.nv1 = b[3 + v] - b[v] + 1;
        const int rows = (q.nv1 + 1) / 2;  // folded: i and nv1 - 1 - i
        q.segs = (rows + 16 * kMaxKc - 1) / (16 * kMaxKc);
        q.kc = ((rows + q.segs - 1) / q.segs + 15) / 16;
        q.blocks = (q.nu1 + kCols - 1) / kCols;
        q.first = b[13] + b[6 + f];
        q.sign = (f & 1) ? 1.0f : -1.0f;
        q.tile0 = x.tiles;
        x.tiles += q.segs * q.blocks * q.kc * 2;
    }
    return x;
}

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float bf16_part(float x) { return __bfloat162float(__float2bfloat16(x)); }

// ---- B: the weighted tangential fields in tiles ----------------------------------------------------
// Thread: a column iu and four folded rows i of a face (16 bytes along K), i the nodes iv = i (at -p_v)
// and nv1 - 1 - i (at +p_v); the middle row of an odd lattice, at 0, is its own partner and counts once. Tile layout: 16-byte piece (K group
// g of 8, MMA column n) at (g * kN + n) * 16.
constexpr int kFieldThreads = 128;
__global__ void __launch_bounds__(kFieldThreads) face_tiles_kernel(Box box, const double2* X, long long total, int f0,
                                                                   double scale, unsigned char* B, float* power) {
    __shared__ float sP[kFieldThreads];
    const int fi = blockIdx.y % 6, fq = blockIdx.y / 6;
    const Face q = box.f[fi];
    const int a = fi >> 1, u = a == 0 ? 1 : 0, v = a == 2 ? 1 : 2;
    const int cols = q.blocks * kCols, groups = q.segs * q.kc * 4;  // groups of four rows
    const long long id = blockIdx.x * (long long)kFieldThreads + threadIdx.x;
    float P = 0.0f;
    if (id < (long long)cols * groups) {
        const int iu = (int)(id % cols), grp = (int)(id / cols);
        const int seg = grp / (q.kc * 4), in_seg = grp - seg * q.kc * 4;
        uint4 hi[4][2], lo[4][2];  // [field][re, im column]: eight K values each
        uint32_t *h = &hi[0][0].x, *l = &lo[0][0].x;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int i = grp * 4 + r;
            float even[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}}, odd[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll
            for (int side = 0; side < 2; ++side) {  // the node at -p_v, then its partner at +p_v
                const int iv = side ? q.nv1 - 1 - i : i;
                const bool middle = 2 * i == q.nv1 - 1;
                if (iu >= q.nu1 || 2 * i > q.nv1 - 1 || (side && middle)) continue;
                const double2* x = X + (size_t)(f0 + fq) * 6 * total + q.first + (size_t)iv * q.nu1 + iu;
                const double2 xeu = x[(size_t)u * total], xev = x[(size_t)v * total];
                const double2 xhu = x[(size_t)(3 + u) * total], xhv = x[(size_t)(3 + v) * total];
                const float w = ((iu == 0 || iu == q.nu1 - 1) ? 0.5f : 1.0f) * ((iv == 0 || iv == q.nv1 - 1) ? 0.5f : 1.0f);
                // n x F for n = sign e_a: +-F of the other tangential component (e_a x e_v = e_u for a = 1)
                const float wu = w * q.sign * (a == 1 ? 1.0f : -1.0f);
                const float eu[2] = {(float)(xeu.x * scale), (float)(xeu.y * scale)};
                const float ev[2] = {(float)(xev.x * scale), (float)(xev.y * scale)};
                const float hu[2] = {(float)(xhu.x * scale), (float)(xhu.y * scale)};
                const float hv[2] = {(float)(xhv.x * scale), (float)(xhv.y * scale)};
                const float flip = middle ? 0.0f : (side ? 1.0f : -1.0f);
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const float val[4] = {wu * hv[p], -wu * hu[p], -wu * ev[p], wu * eu[p]};
#pragma unroll
                    for (int c = 0; c < 4; ++c) even[c][p] += val[c], odd[c][p] += flip * val[c];
                    P += wu * -(eu[p] * hv[p] - ev[p] * hu[p]);  // Re(E x H*).n w, halved at the end
                }
            }
#pragma unroll
            for (int c = 0; c < 4; ++c) {  // times (cos, sin): real column (even re, -odd im), imaginary (even im, odd re)
                const float re[2] = {even[c][0], -odd[c][1]}, im[2] = {even[c][1], odd[c][0]};
                h[(c * 2 + 0) * 4 + r] = pack_bf16(re[0], re[1]), h[(c * 2 + 1) * 4 + r] = pack_bf16(im[0], im[1]);
                l[(c * 2 + 0) * 4 + r] = pack_bf16(re[0] - bf16_part(re[0]), re[1] - bf16_part(re[1]));
                l[(c * 2 + 1) * 4 + r] = pack_bf16(im[0] - bf16_part(im[0]), im[1] - bf16_part(im[1]));
            }
        }
        const int chunk = in_seg >> 2, g = in_seg & 3;
        const size_t tile = (size_t)fq * box.tiles + q.tile0 +
                            ((size_t)(seg * q.blocks + iu / kCols) * q.kc + chunk) * 2;
        unsigned char* o = B + tile * kTile + (size_t)(g * kN + iu % kCols * 8) * 16;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            *reinterpret_cast<uint4*>(o + c * 16) = (&hi[0][0])[c];
            *reinterpret_cast<uint4*>(o + kTile + c * 16) = (&lo[0][0])[c];
        }
    }
    sP[threadIdx.x] = P;
    __syncthreads();
    for (int s = kFieldThreads / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sP[threadIdx.x] = sP[threadIdx.x] + sP[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) power[(size_t)fq * box.parts + fi * gridDim.x + blockIdx.x] = sP[0];
}

// ---- the fused pattern kernel --------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(saddr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait; also gives up once another thread of the CTA has (*abort).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int polls) {
    for (int i = 0; i < polls; ++i) {
        if (mbar_test(bar, parity)) return true;
        if (*abort) return false;
    }
    *abort = 1;
    return false;
}
__device__ __forceinline__ void drain(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < kWaitPolls; ++i)
        if (mbar_test(bar, parity)) return;
}

__device__ __forceinline__ uint64_t operand_desc(const void* p, uint32_t lbo, uint32_t sbo) {
    const uint64_t a = saddr(p);
    return ((a & 0x3FFFFull) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}
// kind::f16, D FP32, A and B BF16, both K-major, M 128, N 256
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(kDirs >> 4) << 24);

__device__ __forceinline__ void mma(uint32_t tmem, uint64_t a, uint64_t b, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(a), "l"(b), "r"(kIdesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(saddr(bar)) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

// Sequence of every role: items (frequency, tile of directions), frequency-major so that a frequency's
// B stays in L2; for each the two sets of faces that share A (normals x and y: V along z; normal z: V
// along y), segment by segment of V, face by face, block by block of columns.
__global__ void __launch_bounds__(kThreads, 1) pattern_kernel(const __grid_constant__ Box box, const unsigned char* B,
                                                             const float* power, const double* omega, int nf,
                                                             const float4* dirs, int D, float* out, unsigned* err,
                                                             int polls) {
    extern __shared__ __align__(1024) unsigned char sm[];
    uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kBarOff);
    uint64_t *full = bars, *empty = bars + kStages, *a_full = bars + 2 * kStages;  // a_full: A is written
    uint64_t *t_full = a_full + 1, *t_empty = t_full + 2;  // products of a block complete / contracted
    volatile int* abort = reinterpret_cast<volatile int*>(bars + 16);
    uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + 17);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) mbar_init(full + s, 1), mbar_init(empty + s, 1);
        mbar_init(a_full, 32 * kComputeWarps);
        for (int s = 0; s < 2; ++s) mbar_init(t_full + s, 1), mbar_init(t_empty + s, 32 * kComputeWarps);
        mbar_init(bars + 15, 1);  // the tensor core's last commit
        *abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(saddr(tslot)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tslot;
    const int dtiles = (D + kDirs - 1) / kDirs, items = nf * dtiles;
    bool ok = true;

    if (warp == kComputeWarps) {
        if (lane == 0) {  // ---- B tiles, one bulk copy each ----
            uint32_t n = 0;  // copies issued
            for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
                const size_t base = (size_t)(item / dtiles) * box.tiles;
                for (int set = 0; ok && set < 2; ++set)
                    for (int seg = 0; ok && seg < box.f[4 * set].segs; ++seg)
                        for (int f = 4 * set; ok && f < (set ? 6 : 4); ++f) {
                            const Face& q = box.f[f];
                            const int count = q.blocks * q.kc * 2;  // a segment's tiles are contiguous
                            const unsigned char* src = B + (base + q.tile0 + (size_t)seg * count) * kTile;
                            for (int t = 0; t < count; ++t, ++n) {
                                const uint32_t s = n % kStages, use = n / kStages;
                                if (use > 0 && !(ok = mbar_wait(empty + s, (use - 1) & 1, abort, polls))) break;
                                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(full + s)),
                                             "r"(kTile)
                                             : "memory");
                                asm volatile(
                                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                        saddr(sm + s * kTile)),
                                    "l"(src + (size_t)t * kTile), "r"(kTile), "r"(saddr(full + s))
                                    : "memory");
                            }
                        }
            }
            // the last copy into every stage lands before the CTA's shared memory goes
            for (uint32_t k = n > kStages ? n - kStages : 0; k < n; ++k) drain(full + k % kStages, (k / kStages) & 1);
        }
        __syncwarp();
    } else if (warp == kComputeWarps + 1) {
        if (lane == 0) {  // ---- the tensor core ----
            uint32_t n = 0, gen = 0, blk = 0;
            for (int item = blockIdx.x; ok && item < items; item += gridDim.x)
                for (int set = 0; ok && set < 2; ++set)
                    for (int seg = 0; ok && seg < box.f[4 * set].segs; ++seg) {
                        if (!(ok = mbar_wait(a_full, gen++ & 1, abort, polls))) break;
                        for (int f = 4 * set; ok && f < (set ? 6 : 4); ++f)
                            for (int b = 0; ok && b < box.f[f].blocks; ++b, ++blk) {
                                const uint32_t half = blk & 1, use = blk >> 1, d = tmem + half * kN;
                                if (use > 0 && !(ok = mbar_wait(t_empty + half, (use - 1) & 1, abort, polls))) break;
                                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                                for (int kc = 0; ok && kc < box.f[f].kc; ++kc) {
                                    const unsigned char* a_hi = sm + kAOff + kc * kAPart;
                                    const unsigned char* a_lo = a_hi + kMaxKc * kAPart;
                                    for (int part = 0; part < 2; ++part, ++n) {  // B_hi, then B_lo
                                        const uint32_t s = n % kStages;
                                        if (!(ok = mbar_wait(full + s, (n / kStages) & 1, abort, polls))) break;
                                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                                        const unsigned char* bt = sm + s * kTile;
#pragma unroll
                                        for (int k = 0; k < kKc / 16; ++k) {
                                            const uint64_t bd = operand_desc(bt + k * 2 * kN * 16, kN * 16, 128);
                                            mma(d, operand_desc(a_hi + k * 2 * kDirs * 16, kDirs * 16, 128), bd,
                                                kc > 0 || part > 0 || k > 0);
                                            if (part == 0)
                                                mma(d, operand_desc(a_lo + k * 2 * kDirs * 16, kDirs * 16, 128), bd, true);
                                        }
                                        commit(empty + s);  // the stage may be refilled once these have read it
                                    }
                                }
                                commit(t_full + half);
                            }
                    }
            // The MMAs issued so far end before tensor and shared memory go: also where another role gave up its
            // wait for them after the last one was issued.
            commit(bars + 15);
            drain(bars + 15, 0);
        }
        __syncwarp();
    } else {
        // ---- A, the contraction over iu, and the result: thread = direction (lane quarter warp % 4) and half
        // of a block's columns (warp / 4) ----
        const int row = (warp & 3) * 32 + lane, half_cols = warp >> 2;
        uint32_t blk = 0;
        float* combine = reinterpret_cast<float*>(sm + kCombineOff) + row * 12;
        for (int item = blockIdx.x; ok && item < items; item += gridDim.x) {
            const int fq = item / dtiles, d = (item - fq * dtiles) * kDirs + row;
            const float4 r = dirs[min(d, D - 1)];
            const double kw = omega[fq];
            const Turns turns[3] = {turns_per_cell(kw, r.x), turns_per_cell(kw, r.y), turns_per_cell(kw, r.z)};
            float NL[2][3][2] = {};  // N, L: [component]{re, im}
            for (int set = 0; ok && set < 2; ++set) {
                const Turns tv = set ? turns[1] : turns[2];
                float step_s, step_c;  // folded row i lies at +-(half - i)
                twiddle(tv, -1.0f, step_s, step_c);
                const float pv0 = set ? box.half[1] : box.half[2];
                const int kcs = box.f[4 * set].kc, rows = (box.f[4 * set].nv1 + 1) / 2;
                for (int seg = 0; ok && seg < box.f[4 * set].segs; ++seg) {
                    // every MMA that read the last A has ended (its products were waited for): the rows of
                    // this segment, chunk by chunk, the two threads of a direction taking turns; anew from
                    // the phase every 16 rows, one complex product from row to row between
                    for (int kc = half_cols; kc < kcs; kc += 2) {
                        const int i0 = (seg * kcs + kc) * 16;
                        float s, c;
                        twiddle(tv, pv0 - (float)i0, s, c);
                        unsigned char* hi = sm + kAOff + kc * kAPart + row * 16;
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            uint32_t h[4], l[4];
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                const bool live = i0 + g * 4 + j < rows;
                                const float vc = live ? c : 0.0f, vs = live ? s : 0.0f;
                                h[j] = pack_bf16(vc, vs);
                                l[j] = pack_bf16(vc - bf16_part(vc), vs - bf16_part(vs));
                                const float c1 = fmaf(c, step_c, -s * step_s);
                                s = fmaf(s, step_c, c * step_s), c = c1;
                            }
                            *reinterpret_cast<uint4*>(hi + g * kDirs * 16) = make_uint4(h[0], h[1], h[2], h[3]);
                            *reinterpret_cast<uint4*>(hi + g * kDirs * 16 + kMaxKc * kAPart) = make_uint4(l[0], l[1], l[2], l[3]);
                        }
                    }
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // -> tensor-core reads
                    mbar_arrive(a_full);
                    for (int f = 4 * set; ok && f < (set ? 6 : 4); ++f) {
                        const int a = f >> 1;
                        const Turns tu = a == 0 ? turns[1] : turns[0];
                        const float pu0 = -(a == 0 ? box.half[1] : box.half[0]);
                        float us, uc;
                        twiddle(tu, 1.0f, us, uc);
                        float g[4][2] = {};
                        for (int b = 0; b < box.f[f].blocks; ++b, ++blk) {
                            const uint32_t half = blk & 1;
                            // one verdict a warp, whatever its lanes saw (a lane may find the barrier complete and
                            // another the abort word): what follows is for whole warps
                            const bool landed = mbar_wait(t_full + half, (blk >> 1) & 1, abort, polls);
                            if (!(ok = __all_sync(0xffffffffu, landed))) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const int iu0 = b * kCols + half_cols * (kCols / 2);
                            float s, c;
                            twiddle(tu, pu0 + (float)iu0, s, c);
                            const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + half * kN + half_cols * (kN / 2);
#pragma unroll
                            for (int t = 0; t < 4; ++t) {  // four columns iu of eight products (the padding's are 0)
                                float v[32];
                                tmem_ld32(at + t * 32, v);
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
#pragma unroll
                                    for (int q = 0; q < 4; ++q) {
                                        const float re = v[i * 8 + 2 * q], im = v[i * 8 + 2 * q + 1];
                                        g[q][0] = fmaf(c, re, fmaf(-s, im, g[q][0]));
                                        g[q][1] = fmaf(s, re, fmaf(c, im, g[q][1]));
                                    }
                                    const float c1 = fmaf(c, uc, -s * us);
                                    s = fmaf(s, uc, c * us), c = c1;
                                }
                            }
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            mbar_arrive(t_empty + half);
                        }
                        // the plane's phase, then the face's share of N and L
                        float s, c;
                        twiddle(turns[a], box.f[f].sign * box.half[a], s, c);
                        float p[4][2];
#pragma unroll
                        for (int q = 0; q < 4; ++q) p[q][0] = c * g[q][0] - s * g[q][1], p[q][1] = s * g[q][0] + c * g[q][1];
#pragma unroll
                        for (int k = 0; k < 3; ++k)  // component k is the face's u or v
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const bool is_u = k == (a == 0 ? 1 : 0), is_v = k == (a == 2 ? 1 : 2);
                                NL[0][k][h] += is_u ? p[0][h] : (is_v ? p[1][h] : 0.0f);
                                NL[1][k][h] += is_u ? p[2][h] : (is_v ? p[3][h] : 0.0f);
                            }
                    }
                }
            }
            // the two halves of the columns, then ntff_reduce.comp:19-39
            if (half_cols)
#pragma unroll
                for (int k = 0; k < 12; ++k) combine[k] = (&NL[0][0][0])[k];
            {  // all of them leave after the same item: one that gave up takes the others along
                uint32_t failed;
                __syncwarp();
                asm volatile(
                    "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\t"
                    "selp.u32 %0, 1, 0, q;\n\t}"
                    : "=r"(failed)
                    : "r"(ok ? 0u : 1u), "n"(32 * kComputeWarps)
                    : "memory");
                ok = failed == 0;
            }
            if (!half_cols) {
#pragma unroll
                for (int k = 0; k < 12; ++k) (&NL[0][0][0])[k] += combine[k];
                const float rv[3] = {r.x, r.y, r.z};
                float F2 = 0.0f;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float N[3] = {NL[0][0][h], NL[0][1][h], NL[0][2][h]}, L[3] = {NL[1][0][h], NL[1][1][h], NL[1][2][h]};
                    const float dn = N[0] * rv[0] + N[1] * rv[1] + N[2] * rv[2];
                    const float F0 = (N[0] - dn * rv[0]) - (rv[1] * L[2] - L[1] * rv[2]);
                    const float F1 = (N[1] - dn * rv[1]) - (rv[2] * L[0] - L[2] * rv[0]);
                    const float Fz = (N[2] - dn * rv[2]) - (rv[0] * L[1] - L[0] * rv[1]);
                    F2 = F2 + (F0 * F0 + F1 * F1 + Fz * Fz);
                }
                if (ok && d < D) {
                    float P = 0.0f;
                    if (d == 0)
                        for (int k = 0; k < box.parts; ++k) P += power[(size_t)fq * box.parts + k];
                    float* o = out + ((size_t)fq * D + d) * 2;
                    o[0] = F2, o[1] = 0.5f * P;
                }
            }
            __syncwarp();
            asm volatile("bar.sync 1, %0;" ::"n"(32 * kComputeWarps) : "memory");  // `combine` is free again
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (tid == 0 && *abort) atomicOr(err, 4u);
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem) : "memory");
}

}  // namespace

extern "C" int emlab_ntff_dft_pattern_gemm(emlab_grid* g, int box, const float* directions, int n_dirs, float* out) {
    if (int rc = require_grid(g)) return rc;
    EMLAB_REQUIRE(g->dft_on, "no far-field DFT attached");
    EMLAB_REQUIRE(box >= 0 && box < g->dft_nbox, "no such far-field DFT box");
    EMLAB_REQUIRE(directions && out && n_dirs > 0 && n_dirs <= (1 << 20), "bad direction arguments");
    EMLAB_CUDA(cudaSetDevice(g->device));
    if (int rc = dft_fold_now(g)) return rc;
    const uint64_t samples = g->dft_samples;
    EMLAB_REQUIRE(samples > 0, "no far-field DFT samples yet");
    Box bx = make_box(g->dft_boxes.data() + (size_t)box * kDftBoxInts);
    const double scale = 2.0 / (double)samples;
    const int D = n_dirs, nf = g->dft_nf;
    long long most = 0;  // threads of the largest face
    for (const Face& q : bx.f) most = std::max(most, (long long)q.blocks * kCols * q.segs * q.kc * 4);
    const int field_blocks = (int)((most + kFieldThreads - 1) / kFieldThreads);
    bx.parts = 6 * field_blocks;
    // frequencies whose tiles take 256 MB together; the scratch grows to the largest request and stays
    const size_t per_f = (size_t)bx.tiles * kTile;
    const int group = (int)std::clamp<size_t>((256ull << 20) / per_f, 1, (size_t)nf);
    const size_t scratch = (group * per_f) / 4 + (size_t)group * bx.parts, outs = (size_t)nf * D * 2;
    if (g->d_spec_dirs.n < (size_t)D || g->d_spec_part.n < scratch || g->d_spec_out.n < outs)
        if (int rc = emlab_grid_synchronize(g, 0)) return rc;
    if (g->d_spec_dirs.n < (size_t)D) EMLAB_CUDA(g->d_spec_dirs.alloc((size_t)D));
    if (g->d_spec_part.n < scratch) EMLAB_CUDA(g->d_spec_part.alloc(scratch));
    if (g->d_spec_out.n < outs) EMLAB_CUDA(g->d_spec_out.alloc(outs));
    EMLAB_CUDA(cudaMemcpyAsync(g->d_spec_dirs.p, directions, (size_t)D * 16, cudaMemcpyHostToDevice, g->stream));
    int sms = 0;
    EMLAB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, g->device));
    EMLAB_CUDA(cudaFuncSetAttribute(pattern_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    unsigned char* B = reinterpret_cast<unsigned char*>(g->d_spec_part.p);
    float* power = g->d_spec_part.p + (group * per_f) / 4;
    const double2* X = reinterpret_cast<const double2*>(g->d_dft_x.p);
    for (int f0 = 0; f0 < nf; f0 += group) {
        const int n = std::min(group, nf - f0);
        face_tiles_kernel<<<dim3(field_blocks, 6 * n), kFieldThreads, 0, g->stream>>>(bx, X, g->dft_points, f0, scale, B, power);
        const int items = n * ((D + kDirs - 1) / kDirs);
        pattern_kernel<<<std::min(items, sms), kThreads, kSmem, g->stream>>>(
            bx, B, power, g->d_dft_omega.p + f0, n, g->d_spec_dirs.p, D, g->d_spec_out.p + (size_t)f0 * D * 2,
            const_cast<unsigned*>(g->h_err), wait_limit());
        count_launches(2);
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return fail(EMLAB_ERR_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
    }
    EMLAB_CUDA(cudaMemcpyAsync(out, g->d_spec_out.p, outs * 4, cudaMemcpyDeviceToHost, g->stream));
    return emlab_grid_synchronize(g, 0);
}
