// Multiple right-hand sides: complex GEMM on the tensor cores and the
// batched vector kernels of a lockstep multi-RHS GMRES.
//
// A complex64 matrix (column-major, m x n, lda) is, viewed as floats, a real
// 2m x n matrix whose even rows hold Re A and odd rows Im A.  With the
// right-hand sides split into planes Xp = [Re X | Im X] (n x 2 nrhs), ONE real
// GEMM Z = A_r Xp (2m x 2 nrhs) reads A once and yields every real product:
//   Re Y = Z[2i, r] - Z[2i+1, nrhs + r],  Im Y = Z[2i, nrhs + r] + Z[2i+1, r].
// The GEMM runs through cuBLAS (a plain library GEMM) in one of three modes:
// FP32 on the CUDA cores, TF32 tensor cores, or BF16x9 (each FP32 operand
// split into three BF16 parts, nine tensor-core products, FP32 accumulation:
// FP32-accurate at tensor-core speed).
#include <cublas_v2.h>

#include <type_traits>

#include "kernels.h"
#include "linalg.h"

namespace nihu {

// Xp[:, r] = Re X[:, r], Xp[:, nrhs + r] = Im X[:, r] (FP32)
__global__ void k_to_planar(const double2 *__restrict__ X, int64_t n, int64_t ldx, int nrhs, float *__restrict__ Xp)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int r = blockIdx.y;
    if (i >= n) return;
    double2 v = X[(int64_t)r * ldx + i];
    Xp[(int64_t)r * n + i] = (float)v.x;
    Xp[(int64_t)(nrhs + r) * n + i] = (float)v.y;
}

// Y = alpha * (complex product from Z) + beta * Y, FP64 accumulation
__global__ void k_combine(const float *__restrict__ Z, int64_t m, int nrhs, double2 *Y, int64_t ldy, double are,
                          double aim, double bre, double bim)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int r = blockIdx.y;
    if (i >= m) return;
    const int64_t ldz = 2 * m;
    double re = (double)Z[(int64_t)r * ldz + 2 * i] - (double)Z[(int64_t)(nrhs + r) * ldz + 2 * i + 1];
    double im = (double)Z[(int64_t)(nrhs + r) * ldz + 2 * i] + (double)Z[(int64_t)r * ldz + 2 * i + 1];
    double2 y = make_double2(0.0, 0.0);
    if (bre != 0.0 || bim != 0.0) y = Y[(int64_t)r * ldy + i];
    Y[(int64_t)r * ldy + i] = make_double2(are * re - aim * im + bre * y.x - bim * y.y,
                                           are * im + aim * re + bre * y.y + bim * y.x);
}

cublasComputeType_t compute_type(int mode)
{
    if (mode == 1) return CUBLAS_COMPUTE_32F_FAST_TF32;
    if (mode == 2) return CUBLAS_COMPUTE_32F_EMULATED_16BFX9;
    return CUBLAS_COMPUTE_32F;
}

cudaError_t launch_gemm_c64(void *cublas, int mode, const void *A, int64_t m, int64_t n, int64_t lda, const double2 *X,
                            int64_t ldx, int nrhs, double2 *Y, int64_t ldy, double are, double aim, double bre,
                            double bim, float *Xp, float *Z, cudaStream_t s, int *cublas_status)
{
    *cublas_status = 0;
    if (m == 0 || nrhs == 0) return cudaSuccess;
    dim3 gx((unsigned)((n + 255) / 256), nrhs);
    if (n > 0) k_to_planar<<<gx, 256, 0, s>>>(X, n, ldx, nrhs, Xp);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    cublasHandle_t h = (cublasHandle_t)cublas;
    cublasSetStream(h, s);
    const float one = 1.0f, zero = 0.0f;
    cublasStatus_t cs;
    if (n > 0) {
        cs = cublasGemmEx(h, CUBLAS_OP_N, CUBLAS_OP_N, (int)(2 * m), 2 * nrhs, (int)n, &one, A, CUDA_R_32F,
                          (int)(2 * lda), Xp, CUDA_R_32F, (int)n, &zero, Z, CUDA_R_32F, (int)(2 * m),
                          compute_type(mode), CUBLAS_GEMM_DEFAULT);
    } else {
        cs = CUBLAS_STATUS_SUCCESS;
        cudaMemsetAsync(Z, 0, sizeof(float) * 2 * m * 2 * nrhs, s);
    }
    if (cs != CUBLAS_STATUS_SUCCESS) {
        *cublas_status = (int)cs;
        return cudaSuccess;
    }
    dim3 gy((unsigned)((m + 255) / 256), nrhs);
    k_combine<<<gy, 256, 0, s>>>(Z, m, nrhs, Y, ldy, are, aim, bre, bim);
    return cudaGetLastError();
}

// ------------------------------------------------------------------ batched
// Vectors are columns of n x nrhs complex128 blocks (leading dimension n);
// a Krylov basis V is (m + 1) such blocks stored back to back.

constexpr int BT = 256;

// part[((v * nrhs + r) * blocks + b)] = sum over the block's rows of conj(V_v[:, r]) . W[:, r];
// F32: products and the thread's and warp's sums in FP32 (the block's in FP64),
// NV basis vectors to a block, which convert W once.  V2: float2 reads a copy
// of the basis that was rounded once, with the same products: the conversions
// of the FP64 one, four a point and vector on the narrow FP64 pipe, bounded the
// Gram-Schmidt passes (15 680 unknowns, 64 right-hand sides, 16 steps: the
// solve 15.5 ms, here 14.0).
template <bool F32, int NV, class V2>
__global__ void __launch_bounds__(BT) k_bdot(const V2 *__restrict__ V, const double2 *__restrict__ W, int64_t n,
                                             int nrhs, int nv, double2 *part)
{
    __shared__ double sr[NV][BT / 32], si[NV][BT / 32];
    const int v0 = blockIdx.z * NV, r = blockIdx.y;
    const V2 *a = V + ((int64_t)v0 * nrhs + r) * n;
    const double2 *b = W + (int64_t)r * n;
    const int64_t next = (int64_t)nrhs * n;
    using T = std::conditional_t<F32, float, double>;
    T ar[NV] = {}, ai[NV] = {};
    for (int64_t i = (int64_t)blockIdx.x * BT + threadIdx.x; i < n; i += (int64_t)gridDim.x * BT) {
        const double2 y = b[i];
        const T yr = (T)y.x, yi = (T)y.y;
#pragma unroll
        for (int u = 0; u < NV; ++u) {
            if (v0 + u >= nv) break;
            const V2 x = a[u * next + i];
            const T xr = (T)x.x, xi = (T)x.y;
            ar[u] += xr * yr + xi * yi;
            ai[u] += xr * yi - xi * yr;
        }
    }
#pragma unroll
    for (int u = 0; u < NV; ++u) {
        const T wr = warp_sum(ar[u]), wi = warp_sum(ai[u]);
        if ((threadIdx.x & 31) == 0) { sr[u][threadIdx.x >> 5] = wr; si[u][threadIdx.x >> 5] = wi; }
    }
    __syncthreads();
    const int u = threadIdx.x;
    if (u < NV && v0 + u < nv) {
        double tr = 0.0, ti = 0.0;
        for (int k = 0; k < BT / 32; ++k) { tr += sr[u][k]; ti += si[u][k]; }
        part[((int64_t)(v0 + u) * nrhs + r) * gridDim.x + blockIdx.x] = make_double2(tr, ti);
    }
}

// out[v * nrhs + r] = sum_b part[(v * nrhs + r) * blocks + b]
__global__ void k_bdot_reduce(const double2 *__restrict__ part, int count, int blocks, double2 *out)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    double sr = 0.0, si = 0.0;
    for (int b = 0; b < blocks; ++b) {
        double2 p = part[(int64_t)t * blocks + b];
        sr += p.x;
        si += p.y;
    }
    out[t] = make_double2(sr, si);
}

// W[:, r] += sign * sum_{v < nv} V_v[:, r] h[v * nrhs + r]; F32: the sum in FP32
template <bool F32>
__global__ void k_bcombo(const double2 *__restrict__ V, int64_t n, int nrhs, int nv, const double2 *__restrict__ h,
                         double sign, double2 *W)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int r = blockIdx.y;
    if (i >= n) return;
    using T = std::conditional_t<F32, float, double>;
    T sr = 0, si = 0;
    for (int v = 0; v < nv; ++v) {
        const double2 a = V[((int64_t)v * nrhs + r) * n + i], c = h[v * nrhs + r];
        const T ar = (T)a.x, ai = (T)a.y, cr = (T)c.x, ci = (T)c.y;
        sr += ar * cr - ai * ci;
        si += ar * ci + ai * cr;
    }
    double2 acc = W[(int64_t)r * n + i];
    acc.x += sign * (double)sr;
    acc.y += sign * (double)si;
    W[(int64_t)r * n + i] = acc;
}

// the same from the FP32 copy of the basis, the coefficients rounded once a block
__global__ void __launch_bounds__(256) k_bcombo32(const float2 *__restrict__ V, int64_t n, int nrhs, int nv,
                                                  const double2 *__restrict__ h, double sign, double2 *W)
{
    constexpr int TILE = 64;  // coefficients staged at a time
    __shared__ float2 hs[TILE];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    float sr = 0, si = 0;
    for (int v0 = 0; v0 < nv; v0 += TILE) {
        const int nt = min(TILE, nv - v0);
        __syncthreads();
        if (threadIdx.x < nt) {
            const double2 c = h[(v0 + threadIdx.x) * nrhs + r];
            hs[threadIdx.x] = make_float2((float)c.x, (float)c.y);
        }
        __syncthreads();
        if (i < n)
#pragma unroll 4
            for (int v = 0; v < nt; ++v) {
                const float2 a = V[((int64_t)(v0 + v) * nrhs + r) * n + i], c = hs[v];
                sr += a.x * c.x - a.y * c.y;
                si += a.x * c.y + a.y * c.x;
            }
    }
    if (i >= n) return;
    double2 acc = W[(int64_t)r * n + i];
    acc.x += sign * (double)sr;
    acc.y += sign * (double)si;
    W[(int64_t)r * n + i] = acc;
}

// dst[:, r] = src[:, r] * s[r], and its FP32 copy dst32 (may be NULL)
__global__ void k_bscale(const double2 *__restrict__ src, double2 *dst, float2 *dst32, int64_t n,
                         const double *__restrict__ s)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    int r = blockIdx.y;
    if (i >= n) return;
    double2 v = src[(int64_t)r * n + i];
    double f = s[r];
    v = make_double2(v.x * f, v.y * f);
    dst[(int64_t)r * n + i] = v;
    if (dst32) dst32[(int64_t)r * n + i] = make_float2((float)v.x, (float)v.y);
}

// R = B - R (element-wise, count complex values)
__global__ void k_rsub(const double2 *__restrict__ B, double2 *R, size_t count)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    double2 b = B[i], r = R[i];
    R[i] = make_double2(b.x - r.x, b.y - r.y);
}

cudaError_t launch_rsub(const double2 *B, double2 *R, size_t count, cudaStream_t s)
{
    if (count == 0) return cudaSuccess;
    k_rsub<<<(unsigned)((count + 255) / 256), 256, 0, s>>>(B, R, count);
    return cudaGetLastError();
}

int bdot_blocks(int64_t n)
{
    int64_t b = (n + BT * 8 - 1) / (BT * 8);
    return (int)max((int64_t)1, min(b, (int64_t)16));
}

static cudaError_t bdot_reduce(const double2 *part, int count, int blocks, double2 *out, cudaStream_t s)
{
    k_bdot_reduce<<<(count + 255) / 256, 256, 0, s>>>(part, count, blocks, out);
    return cudaGetLastError();
}

cudaError_t launch_bdot(const double2 *V, int nv, const double2 *W, int64_t n, int nrhs, double2 *part, double2 *out,
                        cudaStream_t s)
{
    const int blocks = bdot_blocks(n);
    k_bdot<false, 1><<<dim3(blocks, nrhs, nv), BT, 0, s>>>(V, W, n, nrhs, nv, part);
    return bdot_reduce(part, nv * nrhs, blocks, out, s);
}

cudaError_t launch_bdot32(const double2 *V, const float2 *V32, int nv, const double2 *W, int64_t n, int nrhs,
                          double2 *part, double2 *out, cudaStream_t s)
{
    const int blocks = bdot_blocks(n);
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // four vectors a block where that still makes two blocks per SM (10 580 unknowns,
    // seven right-hand sides: a solve 10.28 ms with four, 10.08 with one)
    const dim3 g4(blocks, nrhs, (nv + 3) / 4), g1(blocks, nrhs, nv);
    const bool four = (int64_t)blocks * nrhs * g4.z >= 2 * (int64_t)sms;
    if (V32 && four) k_bdot<true, 4><<<g4, BT, 0, s>>>(V32, W, n, nrhs, nv, part);
    else if (V32) k_bdot<true, 1><<<g1, BT, 0, s>>>(V32, W, n, nrhs, nv, part);
    else k_bdot<true, 1><<<g1, BT, 0, s>>>(V, W, n, nrhs, nv, part);
    return bdot_reduce(part, nv * nrhs, blocks, out, s);
}

cudaError_t launch_bcombo(const double2 *V, int64_t n, int nrhs, int nv, const double2 *h, double sign, double2 *W,
                          cudaStream_t s)
{
    k_bcombo<false><<<dim3((unsigned)((n + 255) / 256), nrhs), 256, 0, s>>>(V, n, nrhs, nv, h, sign, W);
    return cudaGetLastError();
}

cudaError_t launch_bcombo32(const double2 *V, const float2 *V32, int64_t n, int nrhs, int nv, const double2 *h,
                            double sign, double2 *W, cudaStream_t s)
{
    const dim3 g((unsigned)((n + 255) / 256), nrhs);
    if (V32) k_bcombo32<<<g, 256, 0, s>>>(V32, n, nrhs, nv, h, sign, W);
    else k_bcombo<true><<<g, 256, 0, s>>>(V, n, nrhs, nv, h, sign, W);
    return cudaGetLastError();
}

cudaError_t launch_bscale(const double2 *src, double2 *dst, float2 *dst32, int64_t n, int nrhs, const double *sc,
                          cudaStream_t s)
{
    dim3 g((unsigned)((n + 255) / 256), nrhs);
    k_bscale<<<g, 256, 0, s>>>(src, dst, dst32, n, sc);
    return cudaGetLastError();
}

}  // namespace nihu
