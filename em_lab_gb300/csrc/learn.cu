// learn.cu - kernels of the learned ring-down extrapolator (training and inference, sm_103a).
//
// The network (em_lab_gb300/extrap.py) is a 1-D convolutional encoder of the early port V(t), I(t)
// and a 4-layer MLP head; every layer is a GEMM with BF16 operands and FP32 accumulation:
//  * nn_gemm: C[M][N] = sum_k A(m, k) B(n, k) on the tcgen05 tensor cores (kind::f16 with BF16
//    operands, FP32 accumulator in tensor memory). Any strides: the same kernel serves the forward
//    product X W^T and the backward products dZ W and dZ^T X. 64-wide K chunks are copied into a ring
//    of shared-memory stages in the no-swizzle core-matrix layout (K-major, or row-major where the
//    operand is contiguous along its rows), one thread issues four MMAs of K 16 per chunk and
//    commits them to the stage's mbarrier. Waits are bounded; on expiry the CTA records an error,
//    frees its tensor memory and leaves.
//  * elementwise kernels: bias + ReLU with the BF16 copy for the next layer, ReLU backward, bias
//    gradients, im2col / col2im of the strided convolutions, the MSE loss gradient, Adam (FP32
//    master weights, BF16 copies for the GEMMs).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "../../include/emlab_nn.h"
#include "emlab_internal.h"

namespace emlab {
namespace {

constexpr int kTM = 128, kTK = 64;  // tile rows, K chunk (tile columns: 64 or 128)
constexpr int kThreads = 256, kLoaders = kThreads - 32;  // warp 0 issues the MMAs, the others copy
// Core matrices (8 x 16 bytes, 128 bytes) of a chunk. K-major (a piece is 8 elements along K of one
// row): 144 bytes apart along K, 8 x 144 along the rows. Row-major (a piece is 8 rows of one k): 128
// apart along K, 8 x 128 + 16 along the rows. The padding puts the pieces that eight neighbouring
// threads copy into different banks.
constexpr int kLboK = 144, kSboK = 8 * kLboK, kLboR = 128, kSboR = 8 * kLboR + 16;
constexpr int kABytes = kTM / 8 * kSboK;  // the larger of the two
constexpr int kMaxStages = 6;

__device__ unsigned g_nn_err;  // nonzero: a bounded wait of nn_gemm expired

__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// start >> 4, leading (along K) offset >> 4 at bit 16, stride (along the rows) offset >> 4 at bit 32,
// descriptor version 1 at bit 46; no swizzle
__device__ __forceinline__ uint64_t operand_desc(const void* p, int lbo, int sbo) {
    const uint64_t a = saddr(p);
    return ((a & 0x3FFFFull) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9, 10-12 = 1), bit 15 /
// 16 set where A / B lies row-major (contiguous along M / N), N >> 3 at bits 17-22, M >> 4 at 24-28.
__host__ __device__ constexpr uint32_t bf16_idesc(int m, int n, bool a_rows, bool b_rows) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (a_rows ? 1u << 15 : 0u) | (b_rows ? 1u << 16 : 0u) |
           ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// 16 bytes, of which the first `bytes` are read and the rest is zero.
__device__ __forceinline__ void cp_async16(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(saddr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src, int bytes) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(saddr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ bool wait_bounded(uint64_t* bar, uint32_t parity) {
    for (int i = 0; i < (1 << 20); ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(saddr(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
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

// How an operand (rows x K, element strides s_row, s_k) is read: kRowsK, contiguous along K in
// 16-byte pieces; kColsK, contiguous along the rows in 16-byte pieces (the transposed products of the
// backward pass; the tensor core reads it row-major); kAny, element by element.
enum { kRowsK = 0, kColsK = 1, kAny = 2 };

// One operand's 64-wide K chunk from k0, ROWS rows from row0 of its `rows`, into `tile`, by the loading
// threads (t of kLoaders). Everything beyond the operand's rows or K is zero; pieces beyond the rows stay so
// in a stage once `fresh` wrote them.
template <int ROWS, int MODE>
__device__ __forceinline__ void stage_operand(int t, unsigned char* tile, const __nv_bfloat16* p, long long s_row,
                                              long long s_k, int row0, int rows, int k0, int K, bool fresh) {
#pragma unroll
    for (int i = 0; i < (ROWS * kTK / 8 + kLoaders - 1) / kLoaders; ++i) {
        const int q = t + i * kLoaders;
        if (q >= ROWS * kTK / 8) break;
        if (MODE == kColsK) {  // piece (k, row block): a warp copies 32 (or 16) neighbouring row blocks of a k
            const int block = q % (ROWS / 8), k = q / (ROWS / 8);
            const int r = row0 + block * 8;
            if (r >= rows && !fresh) continue;
            const int live = k0 + k < K ? max(0, min(8, rows - r)) : 0;
            cp_async16(tile + block * kSboR + (k >> 3) * kLboR + (k & 7) * 16,
                       live ? p + (long long)(k0 + k) * s_k + r : p, 2 * live);
        } else {  // piece (row, K block): eight threads copy a row's 128 bytes
            const int block = q & 7, r = q >> 3, k = k0 + block * 8;
            if (row0 + r >= rows && !fresh) continue;
            unsigned char* dst = tile + (r >> 3) * kSboK + block * kLboK + (r & 7) * 16;
            const int live = row0 + r < rows ? max(0, min(8, K - k)) : 0;
            const __nv_bfloat16* src = live ? p + (long long)(row0 + r) * s_row + (long long)k * s_k : p;
            if (MODE == kRowsK) {
                cp_async16(dst, src, 2 * live);
            } else {
                __align__(16) __nv_bfloat16 v[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) v[j] = j < live ? src[j * s_k] : __float2bfloat16(0.0f);
                *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(v);
            }
        }
    }
}

// What becomes of a product C. kStore: C itself. kBiasAct: z = C + bias to C, and its activation as BF16 for the
// next layer (`group` rows of C make one row there: the positions of a convolution). kActGrad: the first `cols`
// columns are the gradient after an activation whose argument was z; dz and its BF16 copy, contiguous.
// In the tile's epilogue each of these costs a few hundred nanoseconds where a launch of its own took 3.4 us
// on the device and 10 on the host; same arithmetic, element by element.
enum { kStore = 0, kBiasAct = 1, kActGrad = 2 };
struct Epilogue {
    int kind;
    float* C;
    long long ldc;
    const float* in;  // bias, or z
    __nv_bfloat16* bf;
    long long ldo;
    int off, group, relu, cols;
};

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

__device__ __forceinline__ void store_bf16(__nv_bfloat16* out, const float (&v)[32]) {
#pragma unroll
    for (int q = 0; q < 32; q += 8) {
        __align__(16) __nv_bfloat16 b[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) b[j] = __float2bfloat16(v[q + j]);
        *reinterpret_cast<uint4*>(out + q) = *reinterpret_cast<uint4*>(b);
    }
}

// 32 columns from nb of row m of an N-column product
__device__ __forceinline__ void store_row(const Epilogue& e, int m, int nb, int N, float (&d)[32]) {
    if (e.kind == kActGrad) {
        const long long at = (long long)m * e.cols + nb;
        const int n = min(N, e.cols) - nb;
        if (n >= 32 && e.cols % 8 == 0 && aligned16(e.C) && aligned16(e.in) && aligned16(e.bf)) {
            float z[32];
#pragma unroll
            for (int q = 0; q < 32; q += 4) *reinterpret_cast<float4*>(z + q) = *reinterpret_cast<const float4*>(e.in + at + q);
#pragma unroll
            for (int q = 0; q < 32; ++q)
                if (e.relu && !(z[q] > 0.0f)) d[q] = 0.0f;
#pragma unroll
            for (int q = 0; q < 32; q += 4)
                *reinterpret_cast<float4*>(e.C + at + q) = make_float4(d[q], d[q + 1], d[q + 2], d[q + 3]);
            store_bf16(e.bf + at, d);
            return;
        }
#pragma unroll
        for (int q = 0; q < 32; ++q)
            if (q < n) {
                if (e.relu && !(e.in[at + q] > 0.0f)) d[q] = 0.0f;
                e.C[at + q] = d[q];
                e.bf[at + q] = __float2bfloat16(d[q]);
            }
        return;
    }
    if (e.kind == kBiasAct) {
#pragma unroll
        for (int q = 0; q < 32; ++q)
            if (nb + q < N) d[q] = d[q] + (e.in ? e.in[nb + q] : 0.0f);
    }
    float* crow = e.C + (long long)m * e.ldc;
    if (nb + 32 <= N && e.ldc % 4 == 0 && aligned16(e.C)) {
#pragma unroll
        for (int q = 0; q < 32; q += 4)
            *reinterpret_cast<float4*>(crow + nb + q) = make_float4(d[q], d[q + 1], d[q + 2], d[q + 3]);
    } else {
#pragma unroll
        for (int q = 0; q < 32; ++q)
            if (nb + q < N) crow[nb + q] = d[q];
    }
    if (e.kind != kBiasAct || !e.bf) return;
#pragma unroll
    for (int q = 0; q < 32; ++q) d[q] = e.relu && d[q] < 0.0f ? 0.0f : d[q];
    __nv_bfloat16* out = e.bf + (long long)(m / e.group) * e.ldo + e.off + (long long)(m % e.group) * N + nb;
    if (nb + 32 <= N && aligned16(out)) {
        store_bf16(out, d);
        return;
    }
#pragma unroll
    for (int q = 0; q < 32; ++q)
        if (nb + q < N) out[q] = __float2bfloat16(d[q]);
}

template <int TN>
__host__ __device__ constexpr int gemm_stage() {
    return kABytes + TN / 8 * kSboK;
}

// The ring of a tile: warps 1 .. 7 copy `rounds` rounds of operands into STAGES stages (load(c, stage)), a lane of
// warp 0 hands each round that has landed to the tensor core (mma(c, stage)) and a commit frees its stage.
// A copying thread waits for nothing but a free stage: its copies arrive at the stage's barrier by themselves, and
// the proxy fence between them and the tensor core's reads is the issuing lane's. With the whole CTA at a
// barrier each round the copies of the next waited for the issue of this one: the first head layer (256 x 256,
// K 1344) took 29.6 us, 23.2 us this way.
// False if a wait ran out; every copy and MMA of the caller has ended on return.
template <int STAGES>
struct Ring {
    uint64_t full[STAGES], empty[STAGES];
};
template <int STAGES>
__device__ __forceinline__ void ring_init(Ring<STAGES>& ring) {  // one thread, before a barrier
    for (int i = 0; i < STAGES; ++i) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(saddr(&ring.full[i])), "r"(kLoaders) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&ring.empty[i])) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
template <int STAGES, bool kAsync, class Load, class Mma>
__device__ __forceinline__ bool ring_run(Ring<STAGES>& ring, int rounds, Load&& load, Mma&& mma) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    bool ok = true;
    if (warp == 0) {
        if (lane == 0) {
            int c = 0;
            for (; c < rounds; ++c) {
                ok = wait_bounded(&ring.full[c % STAGES], (c / STAGES) & 1);
                if (!ok) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies -> tensor-core reads
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                mma(c, c % STAGES);
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 saddr(&ring.empty[c % STAGES]))
                             : "memory");
            }
            // commits complete in order: the last one's barrier covers all
            if (c > 0 && !wait_bounded(&ring.empty[(c - 1) % STAGES], ((c - 1) / STAGES) & 1)) ok = false;
        }
        __syncwarp();
    } else {
        for (int c = 0; c < rounds; ++c) {
            // the warp leaves together, also if some lanes' waits just made it
            if (c >= STAGES) ok = wait_bounded(&ring.empty[c % STAGES], (c / STAGES - 1) & 1);
            if (!__all_sync(0xffffffffu, ok)) {
                ok = false;
                break;
            }
            load(c, c % STAGES);
            const uint32_t full = saddr(&ring.full[c % STAGES]);
            if (kAsync)  // arrives once this thread's copies so far have landed
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(full) : "memory");
            else
                asm volatile("{\n\t.reg .b64 t;\n\tmbarrier.arrive.shared::cta.b64 t, [%0];\n\t}" ::"r"(full) : "memory");
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    return ok;
}

// Tensor memory of a tile's accumulator, and the barriers before it is read and given back
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, int cols) {  // warp 0
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(slot)), "r"(cols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_sync() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(accumulate ? 1u : 0u)
        : "memory");
}
// The epilogue: warp w reads TMEM lanes 32 (w % 4) .. +31 (tile rows) of the columns of half w / 4.
template <int TN>
__device__ __forceinline__ void tile_out(bool ok, bool any, uint32_t tmem, int m0, int n0, int M, int N, const Epilogue& e) {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok)) {
        ok = false;
        if (threadIdx.x == 0) atomicOr(&g_nn_err, 1u);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int warp = threadIdx.x >> 5, m = m0 + (warp & 3) * 32 + (threadIdx.x & 31);
#pragma unroll
    for (int j = 0; j < TN / 64; ++j) {
        const int col = (warp >> 2) * (TN / 2) + j * 32;
        float d[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) d[q] = 0.0f;
        if (ok && any) tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col, d);
        if (ok && m < M && n0 + col < N) store_row(e, m, n0 + col, N, d);
    }
    tmem_sync();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN) : "memory");
}

// C[M][N] = sum_k A(m, k) B(n, k), a 128 x TN tile per CTA. What bounds it at the sizes of the network
// (256 rows: a few CTAs of 4 to 21 chunks) is the latency of a chunk's loads, so up to six chunks are in
// flight and tiles are narrow where the device is not full. Every layout is copied 16 bytes at a time.
// The K order of the sum is that of the chunks whatever the tile or the ring, so results do not depend
// on either.
template <int TN, int STAGES, int AM, int BM>
__device__ __forceinline__ void gemm_tile(unsigned char* sm, int m0, int n0, int M, int N, int K,
                                          const __nv_bfloat16* A, long long sam, long long sak,
                                          const __nv_bfloat16* B, long long sbn, long long sbk, const Epilogue& e) {
    __shared__ Ring<STAGES> ring;
    __shared__ uint32_t tslot;
    constexpr int STAGE = gemm_stage<TN>();
    constexpr bool ar = AM == kColsK, br = BM == kColsK;
    constexpr int la = ar ? kLboR : kLboK, sa = ar ? kSboR : kSboK, lb = br ? kLboR : kLboK, sb = br ? kSboR : kSboK;
    if (threadIdx.x == 0) ring_init(ring);
    if (threadIdx.x < 32) tmem_alloc(&tslot, TN);
    tmem_sync();
    const uint32_t tmem = tslot;
    constexpr uint32_t idesc = bf16_idesc(kTM, TN, ar, br);
    const int chunks = (K + kTK - 1) / kTK;
    const bool ok = ring_run<STAGES, AM != kAny && BM != kAny>(
        ring, chunks,
        [&](int c, int s) {
            unsigned char* st = sm + s * STAGE;
            const int t = threadIdx.x - 32;
            stage_operand<kTM, AM>(t, st, A, sam, sak, m0, M, c * kTK, K, c < STAGES);
            stage_operand<TN, BM>(t, st + kABytes, B, sbn, sbk, n0, N, c * kTK, K, c < STAGES);
        },
        [&](int c, int s) {
            unsigned char* st = sm + s * STAGE;
#pragma unroll
            for (int k = 0; k < kTK / 16; ++k)
                mma_bf16(tmem, operand_desc(st + k * 2 * la, la, sa), operand_desc(st + kABytes + k * 2 * lb, lb, sb), idesc,
                         c > 0 || k > 0);
        });
    tile_out<TN>(ok, chunks > 0, tmem, m0, n0, M, N, e);
}

template <int TN, int STAGES, int AM, int BM>
__global__ void __launch_bounds__(kThreads) nn_gemm_kernel(int M, int N, int K, const __nv_bfloat16* A, long long sam,
                                                           long long sak, const __nv_bfloat16* B, long long sbn,
                                                           long long sbk, const __grid_constant__ Epilogue e) {
    extern __shared__ __align__(1024) unsigned char sm[];
    gemm_tile<TN, STAGES, AM, BM>(sm, blockIdx.x * kTM, blockIdx.y * TN, M, N, K, A, sam, sak, B, sbn, sbk, e);
}

template <int TN, int STAGES, int AM, int BM>
cudaError_t launch_gemm(int M, int N, int K, const __nv_bfloat16* A, long long sam, long long sak,
                        const __nv_bfloat16* B, long long sbn, long long sbk, const Epilogue& e, cudaStream_t s) {
    auto kernel = nn_gemm_kernel<TN, STAGES, AM, BM>;
    static const cudaError_t sized =  // once, thread-safe
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, STAGES * gemm_stage<TN>());
    if (sized != cudaSuccess) return sized;
    kernel<<<dim3((M + kTM - 1) / kTM, (N + TN - 1) / TN), kThreads, STAGES * gemm_stage<TN>(), s>>>(
        M, N, K, A, sam, sak, B, sbn, sbk, e);
    return cudaGetLastError();
}

template <int TN, int STAGES>
cudaError_t launch_gemm_modes(int M, int N, int K, const __nv_bfloat16* A, long long sam, long long sak,
                              const __nv_bfloat16* B, long long sbn, long long sbk, const Epilogue& e, cudaStream_t s) {
    auto mode = [](const void* p, long long s_row, long long s_k) {
        if (reinterpret_cast<uintptr_t>(p) & 15) return (int)kAny;
        if (s_k == 1 && s_row % 8 == 0) return (int)kRowsK;
        return s_row == 1 && s_k % 8 == 0 ? (int)kColsK : (int)kAny;
    };
    const int am = mode(A, sam, sak), bm = mode(B, sbn, sbk);
    if (am == kRowsK && bm == kRowsK)
        return launch_gemm<TN, STAGES, kRowsK, kRowsK>(M, N, K, A, sam, sak, B, sbn, sbk, e, s);
    if (am == kRowsK && bm == kColsK)
        return launch_gemm<TN, STAGES, kRowsK, kColsK>(M, N, K, A, sam, sak, B, sbn, sbk, e, s);
    if (am == kColsK && bm == kColsK)
        return launch_gemm<TN, STAGES, kColsK, kColsK>(M, N, K, A, sam, sak, B, sbn, sbk, e, s);
    return launch_gemm<TN, STAGES, kAny, kAny>(M, N, K, A, sam, sak, B, sbn, sbk, e, s);
}

// z[m][n] = c[m][n] + bias[n % bias_n] (in place); a = relu ? max(z, 0) : z, as BF16 at
// out[m * ldo + off + n]. bias_n < N serves a convolution whose rows hold several positions.
__global__ void nn_bias_act_kernel(float* z, const float* bias, int M, int N, int bias_n, int relu,
                                   __nv_bfloat16* out, long long ldo, int off) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)M * N) return;
    const int m = (int)(i / N), n = (int)(i - (long long)m * N);
    const float v = z[i] + (bias ? bias[n % bias_n] : 0.0f);
    z[i] = v;
    if (out) out[(long long)m * ldo + off + n] = __float2bfloat16(relu && v < 0.0f ? 0.0f : v);
}

// dz = dy * (z > 0) (relu) or dy; BF16 copy for the GEMMs
__global__ void nn_act_grad_kernel(const float* dy, long long ldy, int off, const float* z, int M, int N, int relu,
                                   float* dz, __nv_bfloat16* dz_bf) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= (long long)M * N) return;
    const int m = (int)(i / N), n = (int)(i - (long long)m * N);
    float g = dy[(long long)m * ldy + off + n];
    if (relu && !(z[i] > 0.0f)) g = 0.0f;
    dz[i] = g;
    dz_bf[i] = __float2bfloat16(g);
}

// out[n] = sum_m d[m][n], added in row order. One CTA per 32 columns: warps 1 .. 7 copy blocks of 128 rows
// into a ring, warp 0 adds them, one column per lane. The chain of additions is the floor (four cycles each:
// 34 us for the 16384 rows of the first convolution); 121 us with copies of four bytes a thread, 64 us
// with sixteen, 871 us when one thread per column loaded as it added.
constexpr int kSumRows = 128;
__host__ __device__ constexpr int sum_bytes(int stages) { return stages * kSumRows * 32 * 4; }
template <int kSumStages>
__device__ __forceinline__ void col_sum(float* ring, int n0, const float* d, int M, int N, float* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = n0 + lane;
    const int blocks = (M + kSumRows - 1) / kSumRows;
    const bool wide = N % 4 == 0 && aligned16(d);
    auto load = [&](int b) {  // warps 1 .. 7: four columns of a row a thread, or every seventh row a warp
        if (b < blocks && wide) {
            for (int q = threadIdx.x - 32; q < kSumRows * 8; q += kThreads - 32) {
                const int r = q >> 3, c = (q & 7) * 4, m = b * kSumRows + r;
                const bool live = m < M && n0 + c < N;
                cp_async16(ring + ((b % kSumStages) * kSumRows + r) * 32 + c, live ? d + (long long)m * N + n0 + c : d,
                           live ? 16 : 0);
            }
        } else if (b < blocks)
            for (int r = warp - 1; r < kSumRows; r += 7) {
                const int m = b * kSumRows + r;
                const bool live = m < M && n < N;
                cp_async4(ring + ((b % kSumStages) * kSumRows + r) * 32 + lane, live ? d + (long long)m * N + n : d,
                          live ? 4 : 0);
            }
        cp_commit();
    };
    if (warp)
        for (int b = 0; b < kSumStages - 1; ++b) load(b);
    float s = 0.0f;
    for (int b = 0; b < blocks; ++b) {
        if (warp) cp_wait<kSumStages - 2>();
        __syncthreads();  // block b is there; warp 0 is done with block b - 1, whose place block b + 2 takes
        if (warp) {
            load(b + kSumStages - 1);
        } else {
            const float* v = ring + (b % kSumStages) * kSumRows * 32 + lane;
            const int rows = min(kSumRows, M - b * kSumRows);
            if (rows == kSumRows) {
#pragma unroll
                for (int r = 0; r < kSumRows; ++r) s += v[r * 32];
            } else {
                for (int r = 0; r < rows; ++r) s += v[r * 32];
            }
        }
    }
    if (warp) cp_wait<0>();
    else if (n < N) out[n] = s;
}

__global__ void __launch_bounds__(kThreads) nn_col_sum_kernel(const float* d, int M, int N, float* out) {
    __shared__ __align__(16) float ring[sum_bytes(3) / 4];  // what a launch gets without asking
    col_sum<3>(ring, blockIdx.x * 32, d, M, N, out);
}

// The product of two operands contiguous along their rows (kColsK) where at most 64 rows of A are left:
// gw = dz^T x of a convolution sums thousands of rows into one small tile, and what a round costs beside its
// data (a chunk of the ring above: 0.9 us) bounds it. A chunk holds only the rows there are, so `group`
// chunks share a round: the first convolution (32 x 16, 16384 rows) takes 43 rounds of six instead of 256,
// 70 us instead of 242 by itself. The MMAs still read 128 rows and a multiple of 16 columns; what they
// find beyond the operand's rows is other data of the ring and ends in accumulator rows and columns that
// are not stored. Same K order.
constexpr int kNarrowStages = 4;
__device__ __forceinline__ void narrow_tile(unsigned char* sm, int smem, int m0, int n0, int M, int N, int K,
                                            const __nv_bfloat16* A, const __nv_bfloat16* B, const Epilogue& e) {
    __shared__ Ring<kNarrowStages> ring;
    __shared__ uint32_t tslot;
    const int ra = (min(kTM, M - m0) + 7) / 8, rb = (min(64, N - n0) + 7) / 8;  // row blocks
    const int chunk = (ra + rb) * kSboR;
    // the last chunk's MMAs read 16 row blocks of A and up to eight of B from its start on: inside the ring
    const int slots = (smem - (max(16, ra + 8) * kSboR - chunk)) / chunk;
    const int group = min(8, slots / kNarrowStages), stage = group * chunk;
    if (threadIdx.x == 0) ring_init(ring);
    if (threadIdx.x < 32) tmem_alloc(&tslot, 64);
    tmem_sync();
    const uint32_t tmem = tslot;
    const int chunks = (K + kTK - 1) / kTK, rounds = (chunks + group - 1) / group;
    // this thread's pieces (k, row block) of a chunk, the same in every chunk: up to three of each operand
    struct Piece {
        const __nv_bfloat16* src;
        int dst, k, bytes;  // k: kTK and more where there is no piece
    };
    constexpr int kPieces = (8 * kTK + kLoaders - 1) / kLoaders;
    Piece piece[2 * kPieces];
#pragma unroll
    for (int i = 0; i < 2 * kPieces; ++i) {
        const bool of_a = i < kPieces;
        const int blocks = of_a ? ra : rb, q = max(0, (int)threadIdx.x - 32) + i % kPieces * kLoaders;
        const int block = q % blocks, k = q / blocks, rows = of_a ? M : N, row = (of_a ? m0 : n0) + block * 8;
        piece[i] = {(of_a ? A : B) + (long long)min(k, K - 1) * rows + row,
                    (of_a ? 0 : ra * kSboR) + block * kSboR + (k >> 3) * kLboR + (k & 7) * 16, k, 2 * min(8, rows - row)};
    }
    // columns beyond the rows there are (to a multiple of 16) need not be formed
    const uint32_t idesc = bf16_idesc(kTM, (rb + 1) / 2 * 16, true, true);
    const bool ok = ring_run<kNarrowStages, true>(
        ring, rounds,
        [&](int c, int s) {
            for (int g = 0; g < group && c * group + g < chunks; ++g) {
                unsigned char* st = sm + s * stage + g * chunk;
                const int k0 = (c * group + g) * kTK;
#pragma unroll
                for (int i = 0; i < 2 * kPieces; ++i) {
                    if (piece[i].k >= kTK) continue;
                    const bool live = k0 + piece[i].k < K;
                    cp_async16(st + piece[i].dst, live ? piece[i].src + (long long)k0 * (i < kPieces ? M : N) : piece[i].src,
                               live ? piece[i].bytes : 0);
                }
            }
        },
        [&](int c, int s) {
            for (int g = 0; g < group && c * group + g < chunks; ++g) {
                unsigned char* st = sm + s * stage + g * chunk;
#pragma unroll
                for (int k = 0; k < kTK / 16; ++k)
                    mma_bf16(tmem, operand_desc(st + k * 2 * kLboR, kLboR, kSboR),
                             operand_desc(st + ra * kSboR + k * 2 * kLboR, kLboR, kSboR), idesc, c > 0 || g > 0 || k > 0);
            }
        });
    tile_out<64>(ok, chunks > 0, tmem, m0, n0, M, N, e);
}

// The weight and bias gradients of several layers in one launch: gW = dz^T x (M x N, K rows of dz and x)
// and gb = the column sums of dz. They depend on nothing but the layers' dz, so the long chains (the
// first convolution sums 16384 rows in one tile) run beside all the others instead of after them.
constexpr int kMaxGrads = 16, kGradSumStages = 9;
struct GradItem {
    int M, N, K, first;  // first: the layer's first CTA; its tiles, then its column sums
    const __nv_bfloat16 *dz_bf, *x;
    const float* dz;
    float *gw, *gb;
};
struct GradList {
    GradItem g[kMaxGrads];
    int n;
};
__global__ void __launch_bounds__(kThreads) nn_weight_grads_kernel(const __grid_constant__ GradList list) {
    extern __shared__ __align__(1024) unsigned char sm[];
    int i = list.n - 1;
    while (i > 0 && (int)blockIdx.x < list.g[i].first) --i;
    const GradItem& g = list.g[i];
    const int cols = (g.N + 63) / 64, tiles = (g.M + kTM - 1) / kTM * cols, t = (int)blockIdx.x - g.first;
    const Epilogue e = {kStore, g.gw, g.N, nullptr, nullptr, 0, 0, 1, 0, 0};
    const int m0 = t / cols * kTM, n0 = t % cols * 64;
    // up to 64 rows the ring holds at least two chunks a round; more rows and the six single chunks serve
    if (t < tiles && g.M - m0 <= 64)
        narrow_tile(sm, kMaxStages * gemm_stage<64>(), m0, n0, g.M, g.N, g.K, g.dz_bf, g.x, e);
    else if (t < tiles)
        gemm_tile<64, kMaxStages, kColsK, kColsK>(sm, m0, n0, g.M, g.N, g.K, g.dz_bf, 1, g.M, g.x, 1, g.N, e);
    else
        col_sum<kGradSumStages>(reinterpret_cast<float*>(sm), (t - tiles) * 32, g.dz, g.K, g.M, g.gb);
}

// x: [B][Lin][C] (position-major); cols: [B * Lout][k * C], column (j, c) = x[b][l * stride - pad + j][c]
__global__ void nn_im2col_kernel(const __nv_bfloat16* x, int B, int Lin, int Cc, int k, int stride, int pad,
                                 int Lout, __nv_bfloat16* cols) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = (long long)B * Lout * k * Cc;
    if (i >= total) return;
    const int c = (int)(i % Cc);
    const int j = (int)((i / Cc) % k);
    const long long bl = i / ((long long)Cc * k);
    const int l = (int)(bl % Lout), b = (int)(bl / Lout);
    const int p = l * stride - pad + j;
    cols[i] = (p >= 0 && p < Lin) ? x[((long long)b * Lin + p) * Cc + c] : __float2bfloat16(0.0f);
}

// dx[b][p][c] = sum over (l, j) with l * stride - pad + j = p of dcols[(b, l)][(j, c)] (FP32)
// With z: the gradient after the activation whose argument was z, and its BF16 copy.
__global__ void nn_col2im_kernel(const float* dcols, int B, int Lin, int Cc, int k, int stride, int pad, int Lout,
                                 float* dx, const float* z, __nv_bfloat16* dz_bf) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const long long total = (long long)B * Lin * Cc;
    if (i >= total) return;
    const int c = (int)(i % Cc);
    const int p = (int)((i / Cc) % Lin);
    const int b = (int)(i / ((long long)Cc * Lin));
    float s = 0.0f;
    for (int j = 0; j < k; ++j) {
        const int q = p + pad - j;
        if (q < 0 || q % stride) continue;
        const int l = q / stride;
        if (l >= Lout) continue;
        s += dcols[((long long)b * Lout + l) * ((long long)k * Cc) + (long long)j * Cc + c];
    }
    if (z && !(z[i] > 0.0f)) s = 0.0f;
    dx[i] = s;
    if (z) dz_bf[i] = __float2bfloat16(s);
}

// mean squared error over n values: dy = 2 (y - t) / n, loss += sum (y - t)^2 / n (per block, atomic). With
// dy_bf: its BF16 copy, and zeros in both from n to total.
__global__ void nn_mse_kernel(const float* y, const float* t, long long n, long long total, float* dy, __nv_bfloat16* dy_bf,
                              float* loss) {
    __shared__ float red[256];
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    float e = 0.0f;
    if (i < total) {
        const float d = i < n ? y[i] - t[i] : 0.0f, g = i < n ? 2.0f * d / (float)n : 0.0f;
        dy[i] = g;
        if (dy_bf) dy_bf[i] = __float2bfloat16(g);
        if (i < n) e = d * d / (float)n;
    }
    red[threadIdx.x] = e;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0 && loss && (long long)blockIdx.x * blockDim.x < n) atomicAdd(loss, red[0]);
}

// Adam (FP32 master weights); the BF16 copy is refreshed for the next GEMMs. Several tensors in one
// launch (a launch costs more than most of them): tensor i takes the blocks from first[i] on.
constexpr int kMaxAdam = 32;
struct AdamList {
    emlab_nn_param p[kMaxAdam];
    int first[kMaxAdam];
    int n;
};
__global__ void nn_adam_kernel(const __grid_constant__ AdamList list, float lr, float b1, float b2, float eps, float bc1,
                               float bc2) {
    int t = list.n - 1;
    while (t > 0 && (int)blockIdx.x < list.first[t]) --t;
    const emlab_nn_param& p = list.p[t];
    const long long i = ((int)blockIdx.x - list.first[t]) * (long long)blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float gi = p.g[i];
    const float mi = b1 * p.m[i] + (1.0f - b1) * gi;
    const float vi = b2 * p.v[i] + (1.0f - b2) * gi * gi;
    p.m[i] = mi, p.v[i] = vi;
    const float wi = p.w[i] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
    p.w[i] = wi;
    if (p.w_bf16) static_cast<__nv_bfloat16*>(p.w_bf16)[i] = __float2bfloat16(wi);
}

// The first `given` of n values are read, the rest is zero.
__global__ void nn_to_bf16_kernel(const float* x, long long given, long long n, __nv_bfloat16* out, long long ldo,
                                  int cols, int off) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long r = i / cols, c = i - r * cols;
    out[r * ldo + off + c] = __float2bfloat16(i < given ? x[i] : 0.0f);
}

inline unsigned blocks(long long n, int t = 256) { return (unsigned)((n + t - 1) / t); }

}  // namespace
}  // namespace emlab

using namespace emlab;

#define NN_STREAM(s) reinterpret_cast<cudaStream_t>(s)
#define NN_CHECK()                                                                          \
    do {                                                                                    \
        const cudaError_t e_ = cudaGetLastError();                                          \
        if (e_ != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(e_)); \
    } while (0)


namespace {
int gemm(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn, long long sbk,
         const Epilogue& e, void* stream) {
    if (M <= 0 || N <= 0 || K < 0 || !A || !B) return report_error(EMLAB_ERR_INVALID, "bad GEMM arguments");
    const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(A);
    const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>(B);
    // 128-column tiles once they fill the device (each operand row is then read half as often), with
    // three chunks in the ring so that two CTAs share an SM; below that narrow tiles and all six chunks
    const long long wide = (long long)((M + kTM - 1) / kTM) * ((N + 127) / 128);
    const cudaError_t err =
        wide >= 2 * sm_count() ? launch_gemm_modes<128, 3>(M, N, K, a, sam, sak, b, sbn, sbk, e, NN_STREAM(stream))
                        : launch_gemm_modes<64, kMaxStages>(M, N, K, a, sam, sak, b, sbn, sbk, e, NN_STREAM(stream));
    if (err != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(err));
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}
}  // namespace

extern "C" {

int emlab_nn_gemm(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                  long long sbk, float* C, long long ldc, void* stream) {
    if (!C) return report_error(EMLAB_ERR_INVALID, "bad GEMM arguments");
    return gemm(M, N, K, A, sam, sak, B, sbn, sbk, {kStore, C, ldc, nullptr, nullptr, 0, 0, 1, 0, 0}, stream);
}

int emlab_nn_gemm_bias_act(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                           long long sbk, float* Z, long long ldz, const float* bias, int relu, void* out_bf16,
                           long long ldo, int off, int group, void* stream) {
    if (!Z || group < 1) return report_error(EMLAB_ERR_INVALID, "bad GEMM arguments");
    return gemm(M, N, K, A, sam, sak, B, sbn, sbk,
                {kBiasAct, Z, ldz, bias, static_cast<__nv_bfloat16*>(out_bf16), ldo, off, group, relu, 0}, stream);
}

int emlab_nn_gemm_act_grad(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                           long long sbk, const float* z, int cols, int relu, float* dz, void* dz_bf16, void* stream) {
    if (!z || !dz || !dz_bf16 || cols < 1 || cols > N) return report_error(EMLAB_ERR_INVALID, "bad GEMM arguments");
    return gemm(M, N, K, A, sam, sak, B, sbn, sbk,
                {kActGrad, dz, 0, z, static_cast<__nv_bfloat16*>(dz_bf16), 0, 0, 1, relu, cols}, stream);
}

int emlab_nn_status(void* stream) {
    unsigned err = 0;
    if (cudaStreamSynchronize(NN_STREAM(stream)) != cudaSuccess ||
        cudaMemcpyFromSymbol(&err, g_nn_err, 4) != cudaSuccess)
        return report_error(EMLAB_ERR_CUDA, "nn status read failed");
    if (err) {
        const unsigned zero = 0;
        cudaMemcpyToSymbol(g_nn_err, &zero, 4);
        return report_error(EMLAB_ERR_TIMEOUT, "a tensor-core GEMM gave up a bounded wait on the device");
    }
    return EMLAB_OK;
}

int emlab_nn_bias_act(float* z, const float* bias, int M, int N, int bias_n, int relu, void* out_bf16, long long ldo,
                      int off, void* stream) {
    if (bias_n <= 0) return report_error(EMLAB_ERR_INVALID, "bias length must be positive");
    nn_bias_act_kernel<<<blocks((long long)M * N), 256, 0, NN_STREAM(stream)>>>(
        z, bias, M, N, bias_n, relu, static_cast<__nv_bfloat16*>(out_bf16), ldo, off);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_act_grad(const float* dy, long long ldy, int off, const float* z, int M, int N, int relu, float* dz,
                      void* dz_bf16, void* stream) {
    nn_act_grad_kernel<<<blocks((long long)M * N), 256, 0, NN_STREAM(stream)>>>(
        dy, ldy, off, z, M, N, relu, dz, static_cast<__nv_bfloat16*>(dz_bf16));
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_col_sum(const float* d, int M, int N, float* out, void* stream) {
    nn_col_sum_kernel<<<(N + 31) / 32, kThreads, 0, NN_STREAM(stream)>>>(d, M, N, out);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_im2col(const void* x, int B, int Lin, int C, int k, int stride, int pad, int Lout, void* cols,
                    void* stream) {
    nn_im2col_kernel<<<blocks((long long)B * Lout * k * C), 256, 0, NN_STREAM(stream)>>>(
        static_cast<const __nv_bfloat16*>(x), B, Lin, C, k, stride, pad, Lout, static_cast<__nv_bfloat16*>(cols));
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_col2im(const float* dcols, int B, int Lin, int C, int k, int stride, int pad, int Lout, float* dx,
                    void* stream) {
    nn_col2im_kernel<<<blocks((long long)B * Lin * C), 256, 0, NN_STREAM(stream)>>>(dcols, B, Lin, C, k, stride, pad,
                                                                                    Lout, dx, nullptr, nullptr);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_mse(const float* y, const float* t, long long n, float* dy, float* loss, void* stream) {
    nn_mse_kernel<<<blocks(n), 256, 0, NN_STREAM(stream)>>>(y, t, n, n, dy, nullptr, loss);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_mse_grad(const float* y, const float* t, long long n, long long total, float* dy, void* dy_bf16, float* loss,
                      void* stream) {
    if (!y || !t || !dy || !dy_bf16 || n < 1 || total < n)
        return report_error(EMLAB_ERR_INVALID, "bad loss arguments");
    nn_mse_kernel<<<blocks(total), 256, 0, NN_STREAM(stream)>>>(y, t, n, total, dy, static_cast<__nv_bfloat16*>(dy_bf16),
                                                                loss);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_col2im_act_grad(const float* dcols, int B, int Lin, int C, int k, int stride, int pad, int Lout,
                             const float* z, float* dz, void* dz_bf16, void* stream) {
    if (!z || !dz || !dz_bf16) return report_error(EMLAB_ERR_INVALID, "bad gradient arguments");
    nn_col2im_kernel<<<blocks((long long)B * Lin * C), 256, 0, NN_STREAM(stream)>>>(
        dcols, B, Lin, C, k, stride, pad, Lout, dz, z, static_cast<__nv_bfloat16*>(dz_bf16));
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_adam(float* w, float* m, float* v, const float* g, long long n, float lr, float b1, float b2, float eps,
                  int t, void* w_bf16, void* stream) {
    const emlab_nn_param p = {w, m, v, g, n, w_bf16};
    return emlab_nn_adam_all(&p, 1, lr, b1, b2, eps, t, stream);
}

int emlab_nn_adam_all(const emlab_nn_param* params, int count, float lr, float b1, float b2, float eps, int t,
                      void* stream) {
    if (count < 0 || (count && !params)) return report_error(EMLAB_ERR_INVALID, "bad Adam arguments");
    const float bc1 = 1.0f - powf(b1, (float)t), bc2 = 1.0f - powf(b2, (float)t);
    for (int base = 0; base < count; base += kMaxAdam) {
        AdamList list{};
        unsigned total = 0;
        for (int i = base; i < count && list.n < kMaxAdam; ++i) {
            if (params[i].n <= 0) continue;
            list.p[list.n] = params[i];
            list.first[list.n++] = (int)total;
            total += blocks(params[i].n);
        }
        if (!total) continue;
        nn_adam_kernel<<<total, 256, 0, NN_STREAM(stream)>>>(list, lr, b1, b2, eps, bc1, bc2);
        count_launches(1);
        NN_CHECK();
    }
    return EMLAB_OK;
}

int emlab_nn_weight_grads(const emlab_nn_grad* grads, int count, void* stream) {
    if (count < 0 || (count && !grads)) return report_error(EMLAB_ERR_INVALID, "bad gradient arguments");
    auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    GradList list{};
    int total = 0;
    for (int i = 0; i < count; ++i) {
        const emlab_nn_grad& q = grads[i];
        if (q.out_features <= 0 || q.in_features <= 0 || q.rows < 0 || !q.dz_bf16 || !q.x_bf16 || !q.dz || !q.gw || !q.gb)
            return report_error(EMLAB_ERR_INVALID, "bad gradient arguments");
        const int M = q.out_features, N = q.in_features;
        if (list.n < kMaxGrads && M % 8 == 0 && N % 8 == 0 && aligned(q.dz_bf16) && aligned(q.x_bf16)) {
            list.g[list.n++] = {M, N, q.rows, total, static_cast<const __nv_bfloat16*>(q.dz_bf16),
                                static_cast<const __nv_bfloat16*>(q.x_bf16), q.dz, q.gw, q.gb};
            total += (M + kTM - 1) / kTM * ((N + 63) / 64) + (M + 31) / 32;
            continue;
        }
        // rows the tensor core cannot copy 16 bytes at a time: the separate products
        if (int rc = emlab_nn_gemm(M, N, q.rows, q.dz_bf16, 1, M, q.x_bf16, 1, N, q.gw, N, stream)) return rc;
        if (int rc = emlab_nn_col_sum(q.dz, q.rows, M, q.gb, stream)) return rc;
    }
    if (!total) return EMLAB_OK;
    constexpr int smem = kMaxStages * gemm_stage<64>();
    static_assert(smem >= sum_bytes(kGradSumStages), "the column sums' ring fits the tile's stages");
    static const cudaError_t sized =
        cudaFuncSetAttribute(nn_weight_grads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (sized != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(sized));
    nn_weight_grads_kernel<<<total, kThreads, smem, NN_STREAM(stream)>>>(list);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_to_bf16(const float* x, long long n, void* out, long long ldo, int cols, int off, void* stream) {
    return emlab_nn_pad_to_bf16(x, n, n, out, ldo, cols, off, stream);
}

int emlab_nn_pad_to_bf16(const float* x, long long given, long long n, void* out, long long ldo, int cols, int off,
                         void* stream) {
    nn_to_bf16_kernel<<<blocks(n), 256, 0, NN_STREAM(stream)>>>(x, given, n, static_cast<__nv_bfloat16*>(out), ldo, cols,
                                                                off);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

}  // extern "C"
