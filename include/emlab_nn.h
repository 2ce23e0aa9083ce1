/* emlab_nn.h - kernels of the learned ring-down extrapolator (no reference counterpart: the
 * reference has no learned component; the learned antenna-sweep workload).
 *
 * Device pointers and sizes only; `stream` is a cudaStream_t (NULL = the legacy default stream).
 * BF16 operands are __nv_bfloat16 arrays, everything else FP32. Return EMLAB_OK or an error code
 * with emlab_last_error() set. */
#ifndef EMLAB_NN_H
#define EMLAB_NN_H

#ifdef __cplusplus
extern "C" {
#endif

/* C[m * ldc + n] = sum_k A(m, k) B(n, k), A(m, k) = A[m * sam + k * sak], B(n, k) = B[n * sbn + k * sbk]
 * (BF16), FP32 accumulation on the tensor cores (tcgen05, 128 x 64 or 128 x 128 tiles). */
int emlab_nn_gemm(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                  long long sbk, float* C, long long ldc, void* stream);
/* As emlab_nn_gemm, then as emlab_nn_bias_act on its result Z[m * ldz + n] with bias[n] (may be NULL);
 * out_bf16 (may be NULL): out_bf16[(m / group) * ldo + off + (m % group) * N + n]. */
int emlab_nn_gemm_bias_act(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                           long long sbk, float* Z, long long ldz, const float* bias, int relu, void* out_bf16,
                           long long ldo, int off, int group, void* stream);
/* As emlab_nn_act_grad on the first `cols` columns of the product, which itself is not stored: z, dz and
 * dz_bf16 are M x cols. */
int emlab_nn_gemm_act_grad(int M, int N, int K, const void* A, long long sam, long long sak, const void* B, long long sbn,
                           long long sbk, const float* z, int cols, int relu, float* dz, void* dz_bf16, void* stream);
/* Synchronises the stream; EMLAB_ERR_TIMEOUT if a GEMM gave up a bounded wait since the last call. */
int emlab_nn_status(void* stream);
/* z[m][n] += bias[n % bias_n] in place; out_bf16[m * ldo + off + n] = relu ? max(z, 0) : z (BF16). */
int emlab_nn_bias_act(float* z, const float* bias, int M, int N, int bias_n, int relu, void* out_bf16, long long ldo,
                      int off, void* stream);
/* dz = dy[m * ldy + off + n] * (relu ? z > 0 : 1), with a BF16 copy. */
int emlab_nn_act_grad(const float* dy, long long ldy, int off, const float* z, int M, int N, int relu, float* dz,
                      void* dz_bf16, void* stream);
/* out[n] = sum_m d[m][n]. */
int emlab_nn_col_sum(const float* d, int M, int N, float* out, void* stream);
/* x (B, Lin, C) BF16 -> cols (B * Lout, k * C): column (j, c) of row (b, l) = x[b][l * stride - pad + j][c]. */
int emlab_nn_im2col(const void* x, int B, int Lin, int C, int k, int stride, int pad, int Lout, void* cols,
                    void* stream);
/* The adjoint of emlab_nn_im2col on FP32: dx (B, Lin, C) from dcols (B * Lout, k * C). */
int emlab_nn_col2im(const float* dcols, int B, int Lin, int C, int k, int stride, int pad, int Lout, float* dx,
                    void* stream);
/* The same through a ReLU whose argument was z (B, Lin, C), with a BF16 copy. */
int emlab_nn_col2im_act_grad(const float* dcols, int B, int Lin, int C, int k, int stride, int pad, int Lout,
                             const float* z, float* dz, void* dz_bf16, void* stream);
/* dy = 2 (y - t) / n; *loss += sum (y - t)^2 / n. */
int emlab_nn_mse(const float* y, const float* t, long long n, float* dy, float* loss, void* stream);
/* The same with a BF16 copy of dy; dy and the copy are zero from n to total. */
int emlab_nn_mse_grad(const float* y, const float* t, long long n, long long total, float* dy, void* dy_bf16, float* loss,
                      void* stream);
/* One Adam step at time t (>= 1) on n FP32 weights; w_bf16 (optional) receives their BF16 copy. */
int emlab_nn_adam(float* w, float* m, float* v, const float* g, long long n, float lr, float b1, float b2, float eps,
                  int t, void* w_bf16, void* stream);
/* out_bf16[r * ldo + off + c] = x[r * cols + c] for the n = rows * cols values. */
int emlab_nn_to_bf16(const float* x, long long n, void* out, long long ldo, int cols, int off, void* stream);
/* The same, reading only the first `given` values; the rest are zero. */
int emlab_nn_pad_to_bf16(const float* x, long long given, long long n, void* out, long long ldo, int cols, int off,
                         void* stream);

/* Adam of several tensors in one launch (each as emlab_nn_adam does it; tensors of no elements are
 * skipped). */
typedef struct emlab_nn_param {
    float *w, *m, *v;
    const float* g;
    long long n;
    void* w_bf16; /* may be NULL */
} emlab_nn_param;
int emlab_nn_adam_all(const emlab_nn_param* params, int count, float lr, float b1, float b2, float eps, int t,
                      void* stream);
/* Weight and bias gradients of several layers in one launch: gw[o][i] = sum over rows of dz_bf16[r][o]
 * x_bf16[r][i] (as emlab_nn_gemm), gb[o] = sum over rows of dz[r][o] in row order (as emlab_nn_col_sum). */
typedef struct emlab_nn_grad {
    int out_features, in_features, rows;
    const void *dz_bf16, *x_bf16;
    const float* dz;
    float *gw, *gb;
} emlab_nn_grad;
int emlab_nn_weight_grads(const emlab_nn_grad* grads, int count, void* stream);

#ifdef __cplusplus
}
#endif
#endif
