// Mixed-precision LU of one complex system: FP32 factors of the FP64 matrix with
// partial pivoting, and the solves with them.  The FP64 caller refines the
// solution (residual b - A x in FP64, corrections from these factors), so the
// FP32 factors set the speed and the FP64 residual the accuracy.
//
// Factorisation, a panel of up to 16 columns at a time, two kernels each:
//   k_lu32_panel   the panel with its rows in registers (one cluster)
//   k_lu32_trail   its row exchanges on all other columns, the panel's rows of
//                  U (unit-lower triangular solve), the trailing matrix's update
// and k_lu32_diag, which puts the inverses of the factors' 64 x 64 diagonal blocks in
// their place, so that k_lu32_solve's block steps are products.
//
// Order 1280: the factorisation 4.36 -> 2.31 ms, one solve 650 -> 72 us.
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.h"
#include "linalg.h"

namespace nihu {

namespace cg = cooperative_groups;

constexpr int LU32_NB = 16;     // columns of a panel
constexpr int LU32_T = 512;     // threads of a solve's CTA, at most of a panel's
constexpr int LU32_CTAS = 8;    // CTAs of the solve's cluster, at most of the panel's
constexpr int LU32_BLK = 64;    // rows of the solve's blocks
constexpr int LU32_LEFT = 8;    // columns left of a panel to a warp

// the exchange of one panel, relative to its first row j0: row r < nb of the
// result comes from row src[r]; row dst[q] (not below nb) from row from[q], -1: none
struct Lu32Moves {
    int src[LU32_NB], dst[LU32_NB], from[LU32_NB];
};
static_assert(sizeof(Lu32Moves) <= LU32_WORK_BYTES, "the factorisation's scratch");

__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void csubf(float2 &v, float2 a, float2 b)
{
    v.x = fmaf(-a.x, b.x, v.x);
    v.y = fmaf(-a.x, b.y, v.y);
    v.x = fmaf(a.y, b.y, v.x);
    v.y = fmaf(-a.y, b.x, v.y);
}

// F (n x n, leading dimension n) = A rounded to complex64; perm = identity
__global__ void k_to_c64(const double2 *__restrict__ A, int64_t lda, int n, float2 *__restrict__ F, int *__restrict__ perm)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if (i >= n) return;
    const double2 v = A[(int64_t)j * lda + i];
    F[(int64_t)j * n + i] = make_float2((float)v.x, (float)v.y);
    if (j == 0) perm[i] = i;
}

// Panel [j0, j0 + nb) of F, rows j0 .. n: thread t of CTA c holds rows
// c T R + q T + t (q < R) in registers.  A column's step: each warp's largest
// entry (two warp reductions over the bits of |a|^2; the lowest row on ties), a
// barrier, the largest of the warps; its owner writes the row to every CTA of the
// cluster, a second barrier (of the cluster, if there are several CTAs), and every
// thread scales and updates its rows by itself.  The owner of the pivot's row
// takes the diagonal row and the reverse, together with the number of the row
// that it came from.
//
// Bound by the chain of barriers and reductions per column: about 1 us a column,
// nearly whatever the number of rows (16 columns of 512 rows 20 us; with the panel
// in shared memory, a rank-1 pass over it and four barriers a column, 28).
// Unrolled over the columns, whose code is then fetched for one use each, 29 us.
template <int NB, int R, int T>
__global__ void __launch_bounds__(T) k_lu32_panel(float2 *__restrict__ F, int n, int j0, int nb,
                                                       Lu32Moves *__restrict__ moves, int *__restrict__ info)
{
    struct Row {
        float4 v[NB / 2];  // two columns each
    };
    __shared__ int2 s_key[2][T / 32];                // the warps' candidates: |a|^2 bits, row
    __shared__ __align__(16) Row s_u[2][LU32_CTAS];      // the CTAs': their rows, finished columns zero,
    __shared__ __align__(16) Row s_row[2][LU32_CTAS];    // (CTA 0:) with them
    __shared__ __align__(16) float4 s_inv[2][LU32_CTAS]; // (1 / pivot, -, -)
    __shared__ __align__(16) int4 s_slot[2][LU32_CTAS];  // |a|^2 bits, row, origin
    __shared__ __align__(16) Row s_diag[2];              // the diagonal row (CTA 0)
    __shared__ int s_dorig[2];
    __shared__ Lu32Moves s_mv;
    cg::cluster_group cl = cg::this_cluster();
    // every CTA of the cluster has started before its memory is written (waited for
    // behind the loads)
    cg::cluster_group::arrival_token started = cl.barrier_arrive();
    const int C = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = n - j0, row0 = rank * T * R + tid;
    constexpr int NONE = 0x7fffffff;
    float2 *G = F + (int64_t)j0 * n + j0;
    float2 a[R][NB];
    int orig[R], last[R];
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int r = row0 + q * T;
#pragma unroll
        for (int c = 0; c < NB; ++c) a[q][c] = r < m && c < nb ? G[(int64_t)c * n + r] : make_float2(0.0f, 0.0f);
        orig[q] = r;
        last[q] = -1;
    }
    if (rank == 0 && tid < LU32_NB) s_mv.dst[tid] = -1;
    cl.barrier_wait(std::move(started));
    // one body for all columns (unrolled, every instruction would be fetched for
    // one use): the current column is position 0, a step moves all
    // positions down by one, so that after NB steps they are in place again
#pragma unroll 1
    for (int kk = 0; kk < NB; ++kk) {
        if (kk >= nb) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const float2 t = a[q][0];
#pragma unroll
                for (int c = 1; c < NB; ++c) a[q][c - 1] = a[q][c];
                a[q][NB - 1] = t;
            }
            continue;
        }
        const int buf = kk & 1;
        // the thread's candidate; NaN counts as zero
        unsigned key = 0;
        int best = NONE;
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = row0 + q * T;
            const float v = a[q][0].x * a[q][0].x + a[q][0].y * a[q][0].y;
            const unsigned k = v > 0.0f ? __float_as_uint(v) : 0u;
            if (r >= kk && r < m && (best == NONE || k > key)) {
                key = k;
                best = r;
            }
        }
        const unsigned wk = __reduce_max_sync(0xffffffffu, key);
        const int wr = __reduce_min_sync(0xffffffffu, key == wk ? best : NONE);
        if (lane == 0) s_key[buf][warp] = make_int2((int)wk, wr);
        if (rank == 0 && tid == kk) {
            s_dorig[buf] = orig[0];
#pragma unroll
            for (int c = 0; c < NB; c += 2) s_diag[buf].v[c / 2] = make_float4(a[0][c].x, a[0][c].y, a[0][c + 1].x, a[0][c + 1].y);
        }
        __syncthreads();
        const int2 e = s_key[buf][lane & (T / 32 - 1)];
        unsigned bk = __reduce_max_sync(0xffffffffu, (unsigned)e.x);
        int p = __reduce_min_sync(0xffffffffu, (unsigned)e.x == bk ? e.y : NONE);
        // the owner of the CTA's candidate (no row left: thread 0 says so)
        if (p == NONE ? tid == 0 : ((p - rank * T * R) & (T - 1)) == tid) {
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (p == NONE ? q == 0 : row0 + q * T == p) {
                    const float2 d = a[q][0];
                    const float den = d.x * d.x + d.y * d.y;
                    const float4 inv = den > 0.0f ? make_float4(d.x / den, -d.y / den, 0.0f, 0.0f)
                                                  : make_float4(1.0f, 0.0f, 0.0f, 0.0f);
                    for (int t = 0; t < C; ++t) {
                        Row *u = C > 1 ? cl.map_shared_rank(&s_u[buf][rank], t) : &s_u[buf][rank];
#pragma unroll
                        for (int c = 0; c < NB; c += 2) {
                            const float2 x = c < NB - kk ? a[q][c] : make_float2(0.0f, 0.0f);
                            const float2 y = c + 1 < NB - kk ? a[q][c + 1] : make_float2(0.0f, 0.0f);
                            u->v[c / 2] = make_float4(x.x, x.y, y.x, y.y);
                        }
                        *(C > 1 ? cl.map_shared_rank(&s_inv[buf][rank], t) : &s_inv[buf][rank]) = inv;
                        *(C > 1 ? cl.map_shared_rank(&s_slot[buf][rank], t) : &s_slot[buf][rank]) =
                            make_int4((int)bk, p, orig[q], 0);
                    }
                    Row *f = C > 1 ? cl.map_shared_rank(&s_row[buf][rank], 0) : &s_row[buf][rank];
#pragma unroll
                    for (int c = 0; c < NB; c += 2) f->v[c / 2] = make_float4(a[q][c].x, a[q][c].y, a[q][c + 1].x, a[q][c + 1].y);
                }
            }
        }
        int from = 0;  // the CTA that has the pivot
        if (C > 1) {
            cl.sync();
            const int4 o = lane < C ? s_slot[buf][lane] : make_int4(0, NONE, 0, 0);
            bk = __reduce_max_sync(0xffffffffu, (unsigned)o.x);
            p = __reduce_min_sync(0xffffffffu, (unsigned)o.x == bk ? o.y : NONE);
            from = __ffs(__ballot_sync(0xffffffffu, (unsigned)o.x == bk && o.y == p)) - 1;
        } else {
            __syncthreads();
        }
        if (bk == 0 && rank == 0 && tid == 0 && *info == 0) *info = j0 + kk + 1;
        const float2 inv = *reinterpret_cast<const float2 *>(&s_inv[buf][from]);
        float2 fin[R], l[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int r = row0 + q * T;
            if (p != kk) {
                if (r == p) {
                    const Row *diag = rank == 0 ? &s_diag[buf] : cl.map_shared_rank(&s_diag[buf], 0);
                    const int *dorig = rank == 0 ? &s_dorig[buf] : cl.map_shared_rank(&s_dorig[buf], 0);
#pragma unroll
                    for (int c = 0; c < NB; c += 2) {
                        const float4 v = diag->v[c / 2];
                        a[q][c] = make_float2(v.x, v.y);
                        a[q][c + 1] = make_float2(v.z, v.w);
                    }
                    orig[q] = *dorig;
                    last[q] = kk;
                } else if (r == kk) {
#pragma unroll
                    for (int c = 0; c < NB; c += 2) {
                        const float4 v = s_row[buf][from].v[c / 2];
                        a[q][c] = make_float2(v.x, v.y);
                        a[q][c + 1] = make_float2(v.z, v.w);
                    }
                    orig[q] = s_slot[buf][from].z;
                }
            }
            fin[q] = a[q][0];
            l[q] = make_float2(0.0f, 0.0f);
            if (r > kk && r < m) {
                fin[q] = cmulf(fin[q], inv);
                l[q] = fin[q];
            }
        }
        const Row &u = s_u[buf][from];
#pragma unroll
        for (int c = 0; c < NB; c += 2) {
            const float4 v = u.v[c / 2];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                if (c > 0) {
                    a[q][c > 0 ? c - 1 : 0] = a[q][c];
                    csubf(a[q][c > 0 ? c - 1 : 0], l[q], make_float2(v.x, v.y));
                }
                a[q][c] = a[q][c + 1];
                csubf(a[q][c], l[q], make_float2(v.z, v.w));
            }
        }
#pragma unroll
        for (int q = 0; q < R; ++q) a[q][NB - 1] = fin[q];
    }
#pragma unroll
    for (int q = 0; q < R; ++q) {
        const int r = row0 + q * T;
        if (r < m) {
#pragma unroll
            for (int c = 0; c < NB; ++c)
                if (c < nb) G[(int64_t)c * n + r] = a[q][c];
        }
        if (r < nb) s_mv.src[r] = orig[q];  // CTA 0
        else if (last[q] >= 0 && orig[q] != r) {
            Lu32Moves *mv = cl.map_shared_rank(&s_mv, 0);
            mv->dst[last[q]] = r;
            mv->from[last[q]] = orig[q];
        }
    }
    cl.sync();  // the moves are complete, and no CTA leaves while its memory is read
    if (rank == 0 && tid < LU32_NB) {
        moves->src[tid] = tid < nb ? s_mv.src[tid] : tid;
        moves->dst[tid] = s_mv.dst[tid];
        moves->from[tid] = s_mv.from[tid];
    }
}

// The panel's row exchanges on every other column, U12 = L11^{-1} A12 and
// A22 -= L21 U12 in one launch: a block takes W columns right of the panel over
// all rows.  All rows that an exchange moves are read before any is written
// (2 nb independent loads a column); 16 lanes solve a column's triangle;
// then a thread takes whole rows, L21 from L2 into registers, U12 from shared memory.
// The blocks after the strips exchange the columns left of the panel, and perm.
//
// Bound by FP32 issue on the first panels, by the launch on the last.  W: 8 up to
// two strips an SM, 16 beyond (half the reads of L21).  Order 1280, mean of
// the panels: 8 us; exchange, triangle and 64 x 64 tiles as kernels of their own 14.
template <int W>
__global__ void __launch_bounds__(W * 2 * LU32_NB, W == 8 ? 2 : 1) k_lu32_trail(float2 *__restrict__ F, int n, int j0, int nb, int strips,
                                                       const Lu32Moves *__restrict__ moves, int *__restrict__ perm)
{
    constexpr int T = W * 2 * LU32_NB;  // a thread per moved entry
    __shared__ Lu32Moves mv;
    __shared__ float2 L[LU32_NB][LU32_NB + 1];
    __shared__ __align__(16) float2 U[LU32_NB][W];
    const int tid = threadIdx.x;
    if (tid < 3 * LU32_NB) (&mv.src[0])[tid] = (&moves->src[0])[tid];
    if ((int)blockIdx.x >= strips) {
        __syncthreads();
        // a warp a column, a lane an entry
        const int r = tid & 31, q = r & (LU32_NB - 1);
        const bool top = r < LU32_NB, in = top ? r < nb : mv.dst[q] >= 0;
        const int from = in ? (top ? mv.src[q] : mv.from[q]) : 0, to = top ? r : mv.dst[q];
        const int t0 = ((int)blockIdx.x - strips) * LU32_LEFT * W + (tid >> 5);
        float2 v[LU32_LEFT];
#pragma unroll
        for (int k = 0; k < LU32_LEFT; ++k)
            if (in && t0 + k * W < j0) v[k] = F[(int64_t)(t0 + k * W) * n + j0 + from];
        const bool last = t0 == 0 && in;  // perm, by the first block's first warp
        const int x = last ? perm[j0 + from] : 0;
        __syncwarp();
#pragma unroll
        for (int k = 0; k < LU32_LEFT; ++k)
            if (in && t0 + k * W < j0) F[(int64_t)(t0 + k * W) * n + j0 + to] = v[k];
        if (last) perm[j0 + to] = x;
        return;
    }
    if (tid < LU32_NB * LU32_NB) {
        const int r = tid % LU32_NB, c = tid / LU32_NB;
        L[r][c] = r < nb && c < nb ? F[(int64_t)(j0 + c) * n + j0 + r] : make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    const int jb = j0 + nb + (int)blockIdx.x * W, nw = min(W, n - jb);
    // lane r < 16 of a column: its row r of the result; r >= 16: a row below the panel
    const int w = tid / (2 * LU32_NB), r = tid % (2 * LU32_NB);
    const bool top = r < LU32_NB, in = w < nw && (top ? r < nb : mv.dst[r - LU32_NB] >= 0);
    float2 *col = F + (int64_t)(jb + w) * n + j0;
    float2 v = make_float2(0.0f, 0.0f);
    if (in) v = col[top ? mv.src[r] : mv.from[r - LU32_NB]];
    __syncthreads();
    if (in && !top) col[mv.dst[r - LU32_NB]] = v;
#pragma unroll
    for (int q = 0; q < LU32_NB - 1; ++q) {
        const float2 x = make_float2(__shfl_sync(0xffffffffu, v.x, q), __shfl_sync(0xffffffffu, v.y, q));
        if (top && r > q) csubf(v, L[r][q], x);
    }
    if (top) U[r][w] = v;  // zero beyond nb rows and nw columns
    if (in && top) col[r] = v;
    __syncthreads();
    for (int i = j0 + nb + tid; i < n; i += T) {
        float2 l[LU32_NB], c[W];
#pragma unroll
        for (int q = 0; q < LU32_NB; ++q) l[q] = q < nb ? F[(int64_t)(j0 + q) * n + i] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int t = 0; t < W; ++t) c[t] = t < nw ? F[(int64_t)(jb + t) * n + i] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < LU32_NB; ++q)
#pragma unroll
            for (int t = 0; t < W; ++t) csubf(c[t], l[q], U[q][t]);
#pragma unroll
        for (int t = 0; t < W; ++t)
            if (t < nw) F[(int64_t)(jb + t) * n + i] = c[t];
    }
}

// The factors' 64 x 64 diagonal blocks replaced by the inverses of their L
// (blockIdx.y 0, strictly below the diagonal, where the unit one is not stored) and
// U (1, the rest), eight lanes a column; the last block is filled up with the
// identity.  Each thread block reads only the triangle that it writes.
constexpr size_t LU32_DIAG_SMEM = 2 * sizeof(float2) * LU32_BLK * (LU32_BLK + 1);
__global__ void __launch_bounds__(8 * LU32_BLK) k_lu32_diag(float2 *__restrict__ F, int n)
{
    extern __shared__ float2 sm[];
    float2(*D)[LU32_BLK + 1] = reinterpret_cast<float2(*)[LU32_BLK + 1]>(sm);  // D[row][column]
    float2(*X)[LU32_BLK + 1] = reinterpret_cast<float2(*)[LU32_BLK + 1]>(sm + LU32_BLK * (LU32_BLK + 1));  // X[column][row]
    const int b0 = blockIdx.x * LU32_BLK, j = threadIdx.x >> 3, h = threadIdx.x & 7;
    const bool upper = blockIdx.y;
    float2 *G = F + (int64_t)b0 * n + b0;
    for (int t = threadIdx.x; t < LU32_BLK * LU32_BLK; t += 8 * LU32_BLK) {
        const int r = t % LU32_BLK, c = t / LU32_BLK;
        const bool own = b0 + c < n && b0 + r < n && (upper ? r <= c : r > c);
        D[r][c] = own ? G[(int64_t)c * n + r] : make_float2(c == r ? 1.0f : 0.0f, 0.0f);
        X[c][r] = make_float2(0.0f, 0.0f);
    }
    __syncthreads();
    // a row a step, 0.8 us each: the matrix's alone
    const int rows = min(LU32_BLK, n - b0);
    for (int s = 0; s < rows; ++s) {
        const int r = upper ? rows - 1 - s : s;
        float2 v = make_float2(h == 0 && r == j ? 1.0f : 0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < LU32_BLK; q += 8) csubf(v, D[r][q + h], X[j][q + h]);  // zero from row r on
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
            v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
            v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
        }
        if (upper) {
            const float2 u = D[r][r];
            const float den = u.x * u.x + u.y * u.y;
            v = make_float2((v.x * u.x + v.y * u.y) / den, (v.y * u.x - v.x * u.y) / den);
        }
        if (h == 0) X[j][r] = v;
        __syncwarp();
    }
    __syncthreads();
    for (int t = threadIdx.x; t < LU32_BLK * LU32_BLK; t += 8 * LU32_BLK) {
        const int r = t % LU32_BLK, c = t / LU32_BLK;
        if (b0 + c < n && b0 + r < n && (upper ? r <= c : r > c)) G[(int64_t)c * n + r] = X[c][r];
    }
}

// d = U^{-1} L^{-1} P r on one cluster.  The rows' blocks of 64 go round the
// CTAs.  A step has one block's result y, in every CTA's memory: the CTA that
// owns the next block takes y off its rows first, multiplies by the inverse of
// the diagonal block (both tiles were loaded a step ahead), and writes the
// result to all CTAs; the other rows follow between the two halves of the
// cluster barrier.  Thread (row, g) holds eight columns of a tile; its sums
// over the steps are its own (part) until the row is due.
//
// Bound by the chain of a barrier, two small products and the write to the
// other CTAs per block; one CTA, whose thread 0 also ran through the pivots,
// read the factors at 0.1 TB/s (order 1280: 650 us, here 72; without tiles loaded ahead 115).
__global__ void __cluster_dims__(LU32_CTAS, 1, 1) __launch_bounds__(LU32_T)
    k_lu32_solve(const float2 *__restrict__ F, int n, const int *__restrict__ perm, const double2 *__restrict__ r,
                 double2 *__restrict__ d)
{
    extern __shared__ float2 part[];  // [8][own rows]
    __shared__ float2 s_y[4][LU32_BLK], s_red[8][LU32_BLK], s_raw[LU32_BLK];
    cg::cluster_group cl = cg::this_cluster();
    // every CTA has started before its memory is written (waited for behind the gather)
    cg::cluster_group::arrival_token started = cl.barrier_arrive();
    const int rank = (int)cl.block_rank();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = (warp & 1) * 32 + lane, g = warp >> 1;
    const int nblk = (n + LU32_BLK - 1) / LU32_BLK;
    const int own = (nblk - rank + LU32_CTAS - 1) / LU32_CTAS;  // blocks of this CTA
    float2 *mine = part + (size_t)g * own * LU32_BLK + row;     // entry of own block q at q 64
    for (int q = 0; q < own; ++q) {
        const int i = (rank + q * LU32_CTAS) * LU32_BLK + row;
        float2 v = make_float2(0.0f, 0.0f);
        if (g == 0 && i < n) {
            const double2 x = r[perm[i]];
            v = make_float2((float)x.x, (float)x.y);
        }
        mine[q * LU32_BLK] = v;
    }
    cl.barrier_wait(std::move(started));
    // eight columns of the tile (row block rb, column block cb)
    auto load_tile = [&](int rb, int cb, float2 t[8]) {
        const int i = rb * LU32_BLK + row;
        const int j = cb * LU32_BLK + g * 8;
#pragma unroll
        for (int c = 0; c < 8; ++c)
            t[c] = i < n && j + c < n ? __ldg(F + (int64_t)(j + c) * n + i) : make_float2(0.0f, 0.0f);
    };
    // the same of the diagonal block's inverse, of U's or of the unit-lower L's
    auto load_inv = [&](int b, int upper, float2 t[8]) {
        load_tile(b, b, t);
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int j = g * 8 + c;
            if (upper ? row > j : row <= j) t[c] = make_float2(!upper && row == j ? 1.0f : 0.0f, 0.0f);
        }
    };
    auto take_off = [&](float2 &v, const float2 t[8], const float2 *y) {
#pragma unroll
        for (int c = 0; c < 8; ++c) csubf(v, t[c], y[g * 8 + c]);
    };
    // block b's result (by its owner, all threads): the parts' sum times the
    // inverse, into slot of every CTA
    auto finish = [&](int b, const float2 ti[8], int slot, bool last) {
        const int q = b / LU32_CTAS;
        __syncthreads();  // the parts of this block
        if (tid < LU32_BLK) {
            float2 v = part[q * LU32_BLK + tid];
#pragma unroll
            for (int h = 1; h < 8; ++h) {
                const float2 u = part[((size_t)h * own + q) * LU32_BLK + tid];
                v.x += u.x;
                v.y += u.y;
            }
            s_raw[tid] = v;
        }
        __syncthreads();
        float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < 8; ++c) csubf(v, ti[c], s_raw[g * 8 + c]);
        s_red[g][row] = v;
        __syncthreads();
        v = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int h = 0; h < 8; ++h) {
            v.x -= s_red[h][row].x;
            v.y -= s_red[h][row].y;
        }
        cl.map_shared_rank(&s_y[slot][0], g)[row] = v;
        mine[q * LU32_BLK] = g == 0 ? v : make_float2(0.0f, 0.0f);
        const int i = b * LU32_BLK + row;
        if (last && g == 0 && i < n) d[i] = make_double2((double)v.x, (double)v.y);
    };
    // tiles loaded a step ahead: of the next block and of the first two own
    // blocks beyond it
    float2 tl[8], ti[8], t0[8], t1[8];
    // pass 0: blocks up, L; pass 1: blocks down, U
    for (int pass = 0; pass < 2; ++pass) {
        const int step = pass ? -1 : 1, first = pass ? nblk - 1 : 0;
        // own blocks [begin, end) beyond block b
        auto begin = [&](int b) { return pass ? 0 : (b + 1 - rank + LU32_CTAS - 1) / LU32_CTAS; };
        auto end = [&](int b) { return pass ? (b - rank + LU32_CTAS - 1) / LU32_CTAS : own; };
        // the tiles of the step that has block b's result
        auto ahead = [&](int b) {
            const int next = b + step;
            if (next % LU32_CTAS == rank) {
                load_tile(next, b, tl);
                load_inv(next, pass, ti);
            }
            const int q = begin(next), q1 = end(next);
            if (q < q1) load_tile(rank + q * LU32_CTAS, b, t0);
            if (q + 1 < q1) load_tile(rank + (q + 1) * LU32_CTAS, b, t1);
        };
        if (first % LU32_CTAS == rank) {
            load_inv(first, pass, ti);
            finish(first, ti, 0, pass);
        }
        if (nblk > 1) ahead(first);
        cl.sync();
        for (int s = 0; s + 1 < nblk; ++s) {
            const int b = first + s * step, next = b + step;
            const float2 *y = s_y[s & 3];
            if (next % LU32_CTAS == rank) {
                take_off(mine[next / LU32_CTAS * LU32_BLK], tl, y);
                finish(next, ti, (s + 1) & 3, pass);
            }
            cg::cluster_group::arrival_token token = cl.barrier_arrive();
            int q = begin(next);
            const int q1 = end(next);
            if (q < q1) take_off(mine[q * LU32_BLK], t0, y);
            if (q + 1 < q1) take_off(mine[(q + 1) * LU32_BLK], t1, y);
            for (q += 2; q < q1; q += 2) {
                load_tile(rank + q * LU32_CTAS, b, t0);
                if (q + 1 < q1) load_tile(rank + (q + 1) * LU32_CTAS, b, t1);
                take_off(mine[q * LU32_BLK], t0, y);
                if (q + 1 < q1) take_off(mine[(q + 1) * LU32_BLK], t1, y);
            }
            if (s + 2 < nblk) ahead(next);
            cl.barrier_wait(std::move(token));
        }
        cl.sync();  // slot 0 is free for the next pass
    }
}

// the same for one diagonal block (n <= 64): no cluster to launch and to wait for
// (order 1, the whole solve: 167 -> 150 us)
__global__ void __launch_bounds__(LU32_T) k_lu32_solve_block(const float2 *__restrict__ F, int n, const int *__restrict__ perm,
                                                             const double2 *__restrict__ r, double2 *__restrict__ d)
{
    __shared__ float2 s_y[LU32_BLK], s_red[8][LU32_BLK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = (warp & 1) * 32 + lane, g = warp >> 1;
    if (tid < LU32_BLK) {
        const double2 x = tid < n ? r[perm[tid]] : make_double2(0.0, 0.0);
        s_y[tid] = make_float2((float)x.x, (float)x.y);
    }
    for (int upper = 0; upper < 2; ++upper) {
        float2 t[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int j = g * 8 + c;
            const bool own = row < n && j < n && (upper ? row <= j : row > j);
            t[c] = own ? __ldg(F + (int64_t)j * n + row) : make_float2(!upper && row == j ? 1.0f : 0.0f, 0.0f);
        }
        __syncthreads();
        float2 v = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int c = 0; c < 8; ++c) csubf(v, t[c], s_y[g * 8 + c]);
        s_red[g][row] = v;
        __syncthreads();
        if (g == 0) {
            v = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                v.x -= s_red[h][row].x;
                v.y -= s_red[h][row].y;
            }
            s_y[row] = v;
            if (upper && row < n) d[row] = make_double2((double)v.x, (double)v.y);
        }
    }
}

// x += d; sums[0] = |d|^2, sums[1] = |x|^2 (one block, fixed order)
__global__ void __launch_bounds__(1024) k_lu32_update_x(double2 *x, const double2 *__restrict__ d, int n, double *sums)
{
    __shared__ double sd[32], sx[32];
    double ad = 0.0, ax = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double2 di = d[i];
        double2 xi = x[i];
        xi.x += di.x;
        xi.y += di.y;
        x[i] = xi;
        ad += di.x * di.x + di.y * di.y;
        ax += xi.x * xi.x + xi.y * xi.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        ad += __shfl_xor_sync(0xffffffffu, ad, o);
        ax += __shfl_xor_sync(0xffffffffu, ax, o);
    }
    if ((threadIdx.x & 31) == 0) {
        sd[threadIdx.x >> 5] = ad;
        sx[threadIdx.x >> 5] = ax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double td = 0.0, tx = 0.0;
        for (int w = 0; w < (int)(blockDim.x / 32); ++w) {
            td += sd[w];
            tx += sx[w];
        }
        sums[0] = td;
        sums[1] = tx;
    }
}

static int lu32_blocks(int n) { return (n + LU32_BLK - 1) / LU32_BLK; }

// the solve's shared memory: eight parts of the rows of the CTA that has most
static size_t lu32_solve_smem(int n)
{
    return 8 * sizeof(float2) * LU32_BLK * (size_t)((lu32_blocks(n) + LU32_CTAS - 1) / LU32_CTAS);
}

bool lu32_fits(int n, size_t smem_max)
{
    if (n < 1 || n > LU32_T * 8 * LU32_CTAS) return false;  // the panel's registers (4 columns, 8 rows a thread)
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, k_lu32_solve) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return lu32_solve_smem(n) + fa.sharedSizeBytes <= smem_max;
}

cudaError_t lu32_prepare(int n, size_t smem_max)
{
    if (!lu32_fits(n, smem_max)) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(k_lu32_diag, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LU32_DIAG_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_lu32_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lu32_solve_smem(n));
    return e;
}

cudaError_t launch_to_c64(const double2 *A, int64_t lda, int n, float2 *F, int *perm, cudaStream_t s)
{
    k_to_c64<<<dim3((n + 255) / 256, n), 256, 0, s>>>(A, lda, n, F, perm);
    return cudaGetLastError();
}

template <int NB, int R, int T>
static cudaError_t launch_panel(float2 *F, int n, int j0, int *nb, Lu32Moves *moves, int *info, cudaStream_t s)
{
    int ctas = 1;
    while (ctas * T * R < n - j0) ctas *= 2;
    *nb = std::min(NB, n - j0);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(T);
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = ctas > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k_lu32_panel<NB, R, T>, F, n, j0, *nb, moves, info);
}

template <int W>
static void launch_trail(float2 *F, int n, int j0, int nb, const Lu32Moves *moves, int *perm, cudaStream_t s)
{
    const int strips = (n - j0 - nb + W - 1) / W;
    const int left = j0 / (LU32_LEFT * W) + 1;  // blocks for the columns left of the panel and perm
    k_lu32_trail<W><<<strips + left, W * 2 * LU32_NB, 0, s>>>(F, n, j0, nb, strips, moves, perm);
}

cudaError_t launch_lu32_factor(float2 *F, int n, int *perm, void *work, int *info, int64_t *launches, cudaStream_t s)
{
    Lu32Moves *moves = (Lu32Moves *)work;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    for (int j0 = 0, nb; j0 < n; j0 += nb) {
        // rows a thread and columns a panel as the registers of eight CTAs hold
        // them; few rows a CTA while they last (order 1280, all panels: 256 threads of
        // one row 2.31 ms, of two 2.43, 128 of two 2.35, of four 2.64, 512 of one 2.40)
        const int m = n - j0;
        cudaError_t e;
        if (m <= 256 * LU32_CTAS) e = launch_panel<16, 1, 256>(F, n, j0, &nb, moves, info, s);
        else if (m <= 256 * 2 * LU32_CTAS) e = launch_panel<16, 2, 256>(F, n, j0, &nb, moves, info, s);
        else if (m <= 512 * 2 * LU32_CTAS) e = launch_panel<16, 2, 512>(F, n, j0, &nb, moves, info, s);
        else if (m <= 512 * 4 * LU32_CTAS) e = launch_panel<8, 4, 512>(F, n, j0, &nb, moves, info, s);
        else e = launch_panel<4, 8, 512>(F, n, j0, &nb, moves, info, s);
        if (e != cudaSuccess) return e;
        if (m - nb <= 16 * sms) launch_trail<8>(F, n, j0, nb, moves, perm, s);
        else launch_trail<16>(F, n, j0, nb, moves, perm, s);
        *launches += 2;
    }
    k_lu32_diag<<<dim3(lu32_blocks(n), 2), 8 * LU32_BLK, LU32_DIAG_SMEM, s>>>(F, n);
    *launches += 1;
    return cudaGetLastError();
}

cudaError_t launch_lu32_solve(const float2 *F, int n, const int *perm, const double2 *r, double2 *d, cudaStream_t s)
{
    if (n <= LU32_BLK) k_lu32_solve_block<<<1, LU32_T, 0, s>>>(F, n, perm, r, d);
    else k_lu32_solve<<<LU32_CTAS, LU32_T, lu32_solve_smem(n), s>>>(F, n, perm, r, d);
    return cudaGetLastError();
}

cudaError_t launch_lu32_update_x(double2 *x, const double2 *d, int n, double *sums, cudaStream_t s)
{
    k_lu32_update_x<<<1, 1024, 0, s>>>(x, d, n, sums);
    return cudaGetLastError();
}

}  // namespace nihu
