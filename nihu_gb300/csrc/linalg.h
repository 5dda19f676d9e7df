// Internal launchers of the dense linear algebra kernels (linalg.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nihu {

// number of column splits of a matvec (partial buffer holds splits * m complex128);
// sum_warps: warps among which the sum over the splits of a row is divided
int gemv_splits(int64_t m, int64_t n, int dtype, int sum_warps = 1);
constexpr int GMRES_SUM_WARPS = 8;  // of the GMRES step
cudaError_t launch_gemv(int dtype, const void *A, int64_t m, int64_t n, int64_t lda, const double2 *x, double2 *y,
                        double are, double aim, double bre, double bim, double2 *partial, int splits, cudaStream_t s);

// batch members b = 0..batch-1: y_b = alpha A_b x_b + beta y_b with
// A_b = A + b * a_stride (elements), x_b = x + b * n, y_b = y + b * m;
// partial holds batch * splits * m complex128; active (device, may be NULL)
// skips members whose flag is 0 (their y is left untouched)
cudaError_t launch_gemv_batched(int dtype, const void *A, int64_t m, int64_t n, int64_t lda, int64_t a_stride,
                                int batch, const double2 *x, double2 *y, double are, double aim, double bre,
                                double bim, double2 *partial, int splits, cudaStream_t s, const int *active);
cudaError_t launch_add_identity_batched(int n, double are, double aim, int dtype, void *out, int64_t ld, int64_t stride,
                                        int batch, cudaStream_t s);
// segment t: dst[dst_off[t] + i] = src[src_off[t] + i] for i < len[t]
// (device tables of count entries; max_len bounds every len[t])
cudaError_t launch_permute_segments(const double2 *src, double2 *dst, const int64_t *src_off, const int64_t *dst_off,
                                    const int *len, int count, int max_len, cudaStream_t s);

// the matvec's partial sums alone (splits x n); active (device, may be NULL):
// nothing is done when it is 0
cudaError_t launch_gemv_partial(int dtype, const void *A, int64_t m, int64_t n, int64_t lda, const double2 *x,
                                double2 *partial, int splits, cudaStream_t s, const int *active);

// gmres_step.cu ---------------------------------------------------------
// what the host watches (mapped memory): seq is written last
constexpr int GMRES_GO = 0, GMRES_CYCLE = 1, GMRES_STOP = 2, GMRES_ZERO = 3;
struct GmresHost {
    volatile double rel;
    volatile int iters, flag, seq;
};
struct GmresState {
    double r0, rel;
    int iters, kdone;
};
struct GmresStep {
    int64_t n = 0;
    int restart = 0, k = 0, first = 0, max_iters = 0, splits = 0, seq = 0;
    double tol = 0.0;
    const double2 *partial = nullptr;  // of A V_k, or (b set) of A x
    const double2 *b = nullptr;        // set: begin a cycle from b - A x (first: of the solve)
    double2 *V = nullptr;              // restart + 1 vectors
    double2 *small = nullptr;          // H [(restart + 1) x restart], cs, sn [restart], g [restart + 1]
    double2 *sums = nullptr;           // 2 x (restart + 1) x plan.ctas
    GmresState *state = nullptr;
    int *active = nullptr;  // 1 while the cycle runs
    GmresHost *host = nullptr;
};
struct GmresPlan {
    int ctas = 0;
    size_t smem = 0;
};
inline size_t gmres_small_entries(int m) { return (size_t)(m + 1) * m + 2 * m + (m + 1); }
// max_ctas: no more thread blocks than that (their partial sums are 32 (restart + 1) B each)
cudaError_t gmres_step_plan(int64_t n, int restart, int device, int max_ctas, GmresPlan *plan);
cudaError_t launch_gmres_step(const GmresStep &a, const GmresPlan &plan, cudaStream_t s);
// x += V H^{-1} g over the steps done
cudaError_t launch_gmres_update(const GmresStep &a, double2 *x, cudaStream_t s);

cudaError_t launch_lu_factor(double2 *A, int64_t n, int64_t lda, int *piv, int *info, int64_t *launches,
                             cudaStream_t s);
// lu32.cu: mixed-precision LU (FP32 factors of the FP64 matrix, refined by the
// caller): whether order n fits the kernels (smem_max: the device's per-block
// opt-in limit)
bool lu32_fits(int n, size_t smem_max);
// kernel attributes for order n (outside any stream capture)
cudaError_t lu32_prepare(int n, size_t smem_max);
// F (n x n complex64, leading dimension n) = A rounded to complex64, perm [n] = identity
cudaError_t launch_to_c64(const double2 *A, int64_t lda, int n, float2 *F, int *perm, cudaStream_t s);
// F in place = its FP32 LU factors with partial pivoting (perm: the row order; info =
// 1 + first zero pivot column), the diagonal blocks of 64 inverted; work: scratch of
// LU32_WORK_BYTES; stream-capturable
constexpr size_t LU32_WORK_BYTES = 192;
cudaError_t launch_lu32_factor(float2 *F, int n, int *perm, void *work, int *info, int64_t *launches, cudaStream_t s);
// d = (P^T L U)^{-1} r with the FP32 factors
cudaError_t launch_lu32_solve(const float2 *F, int n, const int *perm, const double2 *r, double2 *d, cudaStream_t s);
// x += d; sums[0] = |d|^2, sums[1] = |x|^2
cudaError_t launch_lu32_update_x(double2 *x, const double2 *d, int n, double *sums, cudaStream_t s);
cudaError_t launch_lu_solve(const double2 *A, int64_t n, int64_t lda, const int *piv, const double2 *b, double2 *x,
                            cudaStream_t s);

// multi.cu: complex GEMM on a real view of A (cuBLAS), batched vector kernels
cudaError_t launch_gemm_c64(void *cublas, int mode, const void *A, int64_t m, int64_t n, int64_t lda, const double2 *X,
                            int64_t ldx, int nrhs, double2 *Y, int64_t ldy, double are, double aim, double bre,
                            double bim, float *Xp, float *Z, cudaStream_t s, int *cublas_status);
// gemm_tc.cu: the same product on the tcgen05 tensor cores, split BF16 with
// FP32 accumulation (parts = 2: BF16x3, parts = 3: BF16x6, FP32-accurate).
// Needs a 16-byte aligned A with an even lda (TMA on the float view);
// scratch holds gemm_tc_scratch_bytes(); err receives a nonzero code if a
// pipeline wait ran out (the kernel then stops and frees its tensor memory).
bool gemm_tc_supported(const void *A, int64_t lda);
size_t gemm_tc_scratch_bytes(int parts, int64_t m, int64_t n, int64_t nrhs);
cudaError_t launch_gemm_tc(int parts, const void *A, int64_t m, int64_t n, int64_t lda, const double2 *X, int64_t ldx,
                           int64_t nrhs, double2 *Y, int64_t ldy, double are, double aim, double bre, double bim,
                           void *scratch, int *err, cudaStream_t s);
int bdot_blocks(int64_t n);
cudaError_t launch_bdot(const double2 *V, int nv, const double2 *W, int64_t n, int nrhs, double2 *part, double2 *out,
                        cudaStream_t s);
cudaError_t launch_bcombo(const double2 *V, int64_t n, int nrhs, int nv, const double2 *h, double sign, double2 *W,
                          cudaStream_t s);
// the same with products and partial sums in FP32 (the inner Arnoldi of a
// refinement); V32: the basis V rounded to FP32, or NULL (rounded as it is read)
cudaError_t launch_bdot32(const double2 *V, const float2 *V32, int nv, const double2 *W, int64_t n, int nrhs,
                          double2 *part, double2 *out, cudaStream_t s);
cudaError_t launch_bcombo32(const double2 *V, const float2 *V32, int64_t n, int nrhs, int nv, const double2 *h,
                            double sign, double2 *W, cudaStream_t s);
// dst = src * sc per right-hand side, and its FP32 copy dst32 (may be NULL)
cudaError_t launch_bscale(const double2 *src, double2 *dst, float2 *dst32, int64_t n, int nrhs, const double *sc,
                          cudaStream_t s);
cudaError_t launch_rsub(const double2 *B, double2 *R, size_t count, cudaStream_t s);

}  // namespace nihu
