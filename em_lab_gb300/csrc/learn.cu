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
constexpr int kThreads = 256;
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

// One operand's 64-wide K chunk from k0, ROWS rows from row0 of its `rows`, into `tile`. Everything beyond
// the operand's rows or K is zero; pieces beyond the rows stay so in a stage once `fresh` wrote them.
template <int ROWS, int MODE>
__device__ __forceinline__ void stage_operand(unsigned char* tile, const __nv_bfloat16* p, long long s_row,
                                              long long s_k, int row0, int rows, int k0, int K, bool fresh) {
    const int t = threadIdx.x;
    if (MODE == kColsK) {  // piece (k, row block): a warp copies 32 (or 16) neighbouring row blocks of a k
#pragma unroll
        for (int i = 0; i < ROWS * kTK / 8 / kThreads; ++i) {
            const int q = t + i * kThreads, block = q % (ROWS / 8), k = q / (ROWS / 8);
            const int r = row0 + block * 8;
            if (r >= rows && !fresh) continue;
            const int live = k0 + k < K ? max(0, min(8, rows - r)) : 0;
            cp_async16(tile + block * kSboR + (k >> 3) * kLboR + (k & 7) * 16,
                       live ? p + (long long)(k0 + k) * s_k + r : p, 2 * live);
        }
    } else {  // piece (row, K block): eight threads copy a row's 128 bytes
#pragma unroll
        for (int i = 0; i < ROWS * kTK / 8 / kThreads; ++i) {
            const int q = t + i * kThreads, block = q & 7, r = q >> 3, k = k0 + block * 8;
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

template <int TN>
__host__ __device__ constexpr int gemm_stage() {
    return kABytes + TN / 8 * kSboK;
}

// C[M][N] = sum_k A(m, k) B(n, k), a 128 x TN tile per CTA. What bounds it at the sizes of the network
// (256 rows: a few CTAs of 4 to 21 chunks; the convolutions' weight gradients, one or four CTAs of 64
// and 256) is the latency of a chunk's loads, so up to six chunks are in flight (asynchronous copies
// into a ring, one mbarrier per stage that the MMAs reading it complete) and tiles are narrow where the
// device is not full. Every layout is copied 16 bytes at a time. The K order of the sum is that of
// the chunks whatever the tile or the ring, so results do not depend on either.
template <int TN, int AM, int BM>
__device__ __forceinline__ void gemm_tile(unsigned char* sm, int m0, int n0, int M, int N, int K,
                                          const __nv_bfloat16* A, long long sam, long long sak,
                                          const __nv_bfloat16* B, long long sbn, long long sbk, float* C,
                                          long long ldc, int stages) {
    __shared__ uint64_t bar[kMaxStages];  // the MMAs that read stage s have finished
    __shared__ uint32_t tslot;
    // 1 + the chunk whose barrier everyone leaves after, once a wait ran out (a thread late to read it
    // after one barrier may already see the next chunk's)
    __shared__ volatile int stop;
    constexpr int STAGE = gemm_stage<TN>();
    constexpr bool ar = AM == kColsK, br = BM == kColsK;
    constexpr int la = ar ? kLboR : kLboK, sa = ar ? kSboR : kSboK, lb = br ? kLboR : kLboK, sb = br ? kSboR : kSboK;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int i = 0; i < stages; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(&bar[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(saddr(&tslot)), "r"(TN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const int chunks = (K + kTK - 1) / kTK;
    auto load = [&](int c) {  // one group of copies per chunk, empty past the last
        if (c < chunks) {
            unsigned char* st = sm + (c % stages) * STAGE;
            stage_operand<kTM, AM>(st, A, sam, sak, m0, M, c * kTK, K, c < stages);
            stage_operand<TN, BM>(st + kABytes, B, sbn, sbk, n0, N, c * kTK, K, c < stages);
        }
        cp_commit();
    };
    for (int c = 0; c < kMaxStages - 2; ++c)
        if (c < stages - 2) load(c);
        else cp_commit();
    if (tid == 0) stop = 0;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tslot;
    constexpr uint32_t idesc = bf16_idesc(kTM, TN, ar, br);

    bool ok = true;
    int issued = 0;  // chunks handed to the tensor core
    for (int c = 0; c < chunks; ++c) {
        // chunk c - 2's stage takes chunk c - 2 + stages once its MMAs have read it (two chunks back, so
        // that the wait is over when it is reached)
        if (c >= 2 && c - 2 + stages < chunks && !wait_bounded(&bar[(c - 2) % stages], ((c - 2) / stages) & 1)) stop = c + 1;
        load(c - 2 + stages);
        // this thread's copies of chunk c have landed: those of at most stages - 2 later ones are open
        if (stages == kMaxStages) cp_wait<kMaxStages - 2>();
        else cp_wait<1>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies -> tensor-core reads
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (stop == c + 1) {
            ok = false;
            break;
        }
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            unsigned char* st = sm + (c % stages) * STAGE;
#pragma unroll
            for (int s = 0; s < kTK / 16; ++s) {
                const uint64_t ad = operand_desc(st + s * 2 * la, la, sa), bd = operand_desc(st + kABytes + s * 2 * lb, lb, sb);
                const uint32_t acc = (c > 0 || s > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             saddr(&bar[c % stages]))
                         : "memory");
        }
        ++issued;
    }
    cp_wait<0>();
    // every MMA has ended (commits complete in order: the last one's barrier covers all)
    if (issued > 0 && !wait_bounded(&bar[(issued - 1) % stages], ((issued - 1) / stages) & 1)) ok = false;
    if (__syncthreads_or(!ok)) {
        ok = false;
        if (tid == 0) atomicOr(&g_nn_err, 1u);
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    // warp w reads TMEM lanes 32 (w % 4) .. +31 (tile rows) of the columns of half w / 4
    const int m = m0 + (warp & 3) * 32 + lane;
    const bool vec_c = (ldc % 4) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
    for (int j = 0; j < TN / 64; ++j) {
        const int col = (warp >> 2) * (TN / 2) + j * 32;
        float d[32];
#pragma unroll
        for (int q = 0; q < 32; ++q) d[q] = 0.0f;
        if (ok && issued > 0) tmem_ld32(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col, d);
        const int nb = n0 + col;
        if (!ok || m >= M) continue;
        float* crow = C + (long long)m * ldc;
        if (nb + 32 <= N && vec_c) {
#pragma unroll
            for (int q = 0; q < 32; q += 4)
                *reinterpret_cast<float4*>(crow + nb + q) = make_float4(d[q], d[q + 1], d[q + 2], d[q + 3]);
            continue;
        }
#pragma unroll
        for (int q = 0; q < 32; ++q)
            if (nb + q < N) crow[nb + q] = d[q];
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TN) : "memory");
}

template <int TN, int AM, int BM>
__global__ void __launch_bounds__(kThreads) nn_gemm_kernel(int M, int N, int K, const __nv_bfloat16* A, long long sam,
                                                           long long sak, const __nv_bfloat16* B, long long sbn,
                                                           long long sbk, float* C, long long ldc, int stages) {
    extern __shared__ __align__(1024) unsigned char sm[];
    gemm_tile<TN, AM, BM>(sm, blockIdx.x * kTM, blockIdx.y * TN, M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, stages);
}

template <int TN, int AM, int BM>
cudaError_t launch_gemm(int M, int N, int K, const __nv_bfloat16* A, long long sam, long long sak,
                        const __nv_bfloat16* B, long long sbn, long long sbk, float* C, long long ldc, int stages,
                        cudaStream_t s) {
    auto kernel = nn_gemm_kernel<TN, AM, BM>;
    static const cudaError_t sized =  // once, thread-safe
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxStages * gemm_stage<TN>());
    if (sized != cudaSuccess) return sized;
    kernel<<<dim3((M + kTM - 1) / kTM, (N + TN - 1) / TN), kThreads, stages * gemm_stage<TN>(), s>>>(
        M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, stages);
    return cudaGetLastError();
}

template <int TN>
cudaError_t launch_gemm_modes(int M, int N, int K, const __nv_bfloat16* A, long long sam, long long sak,
                              const __nv_bfloat16* B, long long sbn, long long sbk, float* C, long long ldc, int stages,
                              cudaStream_t s) {
    auto mode = [](const void* p, long long s_row, long long s_k) {
        if (reinterpret_cast<uintptr_t>(p) & 15) return (int)kAny;
        if (s_k == 1 && s_row % 8 == 0) return (int)kRowsK;
        return s_row == 1 && s_k % 8 == 0 ? (int)kColsK : (int)kAny;
    };
    const int am = mode(A, sam, sak), bm = mode(B, sbn, sbk);
    if (am == kRowsK && bm == kRowsK)
        return launch_gemm<TN, kRowsK, kRowsK>(M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, stages, s);
    if (am == kRowsK && bm == kColsK)
        return launch_gemm<TN, kRowsK, kColsK>(M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, stages, s);
    if (am == kColsK && bm == kColsK)
        return launch_gemm<TN, kColsK, kColsK>(M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, stages, s);
    return launch_gemm<TN, kAny, kAny>(M, N, K, A, sam, sak, B, sbn, sbk, C, ldc, stages, s);
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
// into a ring of three, warp 0 adds them, one column per lane. Bound by the chain of additions (16384
// rows of the first convolution), which the loads no longer interrupt: 871 us before, when one thread
// per column loaded as it added.
constexpr int kSumRows = 128, kSumStages = 3;
constexpr int kSumBytes = kSumStages * kSumRows * 32 * 4;
__device__ __forceinline__ void col_sum(float* ring, int n0, const float* d, int M, int N, float* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = n0 + lane;
    const int blocks = (M + kSumRows - 1) / kSumRows;
    auto load = [&](int b) {  // warps 1 .. 7: every seventh row
        if (b < blocks)
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
    __shared__ __align__(16) float ring[kSumBytes / 4];
    col_sum(ring, blockIdx.x * 32, d, M, N, out);
}

// The weight and bias gradients of several layers in one launch: gW = dz^T x (M x N, K rows of dz and x)
// and gb = the column sums of dz. They depend on nothing but the layers' dz, so the long chains (the
// first convolution sums 16384 rows in one tile) run beside all the others instead of after them.
constexpr int kMaxGrads = 16;
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
    if (t < tiles)
        gemm_tile<64, kColsK, kColsK>(sm, t / cols * kTM, t % cols * 64, g.M, g.N, g.K, g.dz_bf, 1, g.M, g.x, 1, g.N,
                                      g.gw, g.N, kMaxStages);
    else
        col_sum(reinterpret_cast<float*>(sm), (t - tiles) * 32, g.dz, g.K, g.M, g.gb);
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
__global__ void nn_col2im_kernel(const float* dcols, int B, int Lin, int Cc, int k, int stride, int pad, int Lout,
                                 float* dx) {
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
    dx[i] = s;
}

// mean squared error over n values: dy = 2 (y - t) / n, loss += sum (y - t)^2 / n (per block, atomic)
__global__ void nn_mse_kernel(const float* y, const float* t, long long n, float* dy, float* loss) {
    __shared__ float red[256];
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    float e = 0.0f;
    if (i < n) {
        const float d = y[i] - t[i];
        dy[i] = 2.0f * d / (float)n;
        e = d * d / (float)n;
    }
    red[threadIdx.x] = e;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0 && loss) atomicAdd(loss, red[0]);
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

__global__ void nn_to_bf16_kernel(const float* x, long long n, __nv_bfloat16* out, long long ldo, int cols, int off) {
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long r = i / cols, c = i - r * cols;
    out[r * ldo + off + c] = __float2bfloat16(x[i]);
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

extern "C" {

int emlab_nn_gemm(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                  long long sbk, float* C, long long ldc, void* stream) {
    if (M <= 0 || N <= 0 || K < 0 || !A || !B || !C) return report_error(EMLAB_ERR_INVALID, "bad GEMM arguments");
    const __nv_bfloat16* a = static_cast<const __nv_bfloat16*>(A);
    const __nv_bfloat16* b = static_cast<const __nv_bfloat16*>(B);
    // 128-column tiles once they fill the device (each operand row is then read half as often), with
    // three chunks in the ring so that two CTAs share an SM; below that narrow tiles and all six chunks
    const long long wide = (long long)((M + kTM - 1) / kTM) * ((N + 127) / 128);
    const cudaError_t e =
        wide >= 2 * 152 ? launch_gemm_modes<128>(M, N, K, a, sam, sak, b, sbn, sbk, C, ldc, 3, NN_STREAM(stream))
                        : launch_gemm_modes<64>(M, N, K, a, sam, sak, b, sbn, sbk, C, ldc, kMaxStages, NN_STREAM(stream));
    if (e != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(e));
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
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
                                                                                    Lout, dx);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_mse(const float* y, const float* t, long long n, float* dy, float* loss, void* stream) {
    nn_mse_kernel<<<blocks(n), 256, 0, NN_STREAM(stream)>>>(y, t, n, dy, loss);
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
    static_assert(smem >= kSumBytes, "the column sums' ring fits the tile's stages");
    static const cudaError_t sized =
        cudaFuncSetAttribute(nn_weight_grads_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (sized != cudaSuccess) return report_error(EMLAB_ERR_CUDA, cudaGetErrorString(sized));
    nn_weight_grads_kernel<<<total, kThreads, smem, NN_STREAM(stream)>>>(list);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

int emlab_nn_to_bf16(const float* x, long long n, void* out, long long ldo, int cols, int off, void* stream) {
    nn_to_bf16_kernel<<<blocks(n), 256, 0, NN_STREAM(stream)>>>(x, n, static_cast<__nv_bfloat16*>(out), ldo, cols, off);
    count_launches(1);
    NN_CHECK();
    return EMLAB_OK;
}

}  // extern "C"
