// The vector part of one GMRES step of a single dense system, on the device:
// the sum of the matvec's partial products, classical Gram-Schmidt with one
// reorthogonalisation (CGS2, FP64), the new basis vector, the Givens rotations
// and the stopping decision (nihu/fmm/GMRES.h:57-205 semantics), in one
// cooperative launch.
//
// The step was eight launches and three host round trips (two projections and
// a norm, each read back for the rotations), 60 us beside a matvec of 46 us
// on 5120 unknowns.  The vectors are small, but their FP64 sums want every SM
// (2 FP64 operations per SM and cycle: on one cluster of 8 SMs the step took
// 79 us): CTA c of a cooperative launch owns a slice of the rows and keeps its
// part of w in shared memory; dot products and norms are formed per CTA and
// added in a fixed order by every CTA after a grid barrier (three per step).
// The host only watches a status word in mapped memory, one step behind, to
// stop enqueuing; steps enqueued past the end find `active` = 0 and return.
// 5120 unknowns, assembly and 8 steps: 1.38 -> 0.91 ms (the step 29 us beside a
// matvec of 35 us); 320 unknowns, 3 steps: 0.57 -> 0.23 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "common.cuh"
#include "linalg.h"

namespace cg = cooperative_groups;

namespace nihu {
namespace {

constexpr int GS_THREADS = 256;
constexpr int GS_WARPS = GS_THREADS / 32;
static_assert(GS_WARPS == GMRES_SUM_WARPS, "the partial products are summed by every warp");
constexpr int GS_ROWS = 32;  // fewest rows per CTA
// basis vectors from which on each thread takes one (its product with w, its sum
// over the CTAs): a warp's sum over its lanes, 20 FP64 additions a vector, is then
// most of the step (2000 unknowns, GMRES(256), 256 steps: 69.7 -> 44.0 ms; eight
// launches a step, before the cooperative one, 60.2)
constexpr int GS_LONG = 64;

__device__ __forceinline__ double2 cmul2(double2 a, double2 b)
{
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cmulc(double2 a, double2 b)  // conj(a) b
{
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// LONG: a step of GS_LONG basis vectors or more
template <bool LONG>
__global__ void __launch_bounds__(GS_THREADS) k_gmres_step(GmresStep a)
{
    cg::grid_group grid = cg::this_grid();
    const int G = (int)gridDim.x, rank = (int)blockIdx.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m = a.restart, k = a.k;
    const int64_t n = a.n;
    // written by the launches before this one only, and by this one's CTA 0
    // after its last barrier
    if (!*reinterpret_cast<volatile int *>(a.active)) {
        if (rank == 0 && tid == 0) a.host->seq = a.seq;
        return;
    }
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2 *h = reinterpret_cast<double2 *>(smem_raw);  // [m + 2]
    double2 *h2 = h + (m + 2);                            // [m + 1]
    double2 *part = h2 + (m + 1);                         // [GS_WARPS][32], then [2 m + 1]
    double2 *w = part + (size_t)GS_WARPS * 32 + 2 * m + 1;  // the slice
    const int64_t i0 = n * rank / G, i1 = n * (rank + 1) / G;
    const int rows = (int)(i1 - i0);
    double2 *V = a.V;  // basis vector v at V + v * n
    int buf = 0;

    // out[v] = sum over the CTAs of part(v) (this CTA's, a warp at a time), v < cnt:
    // lane c % 32 adds CTAs c, c + 32, ... and the lanes are added as a tree
    auto reduce = [&](int cnt, double2 *out, auto &&part) {
        double2 *all = a.sums + (size_t)buf * (m + 1) * G;
        for (int v = warp; v < cnt; v += GS_WARPS) {
            const double2 p = part(v);
            if (lane == 0) __stcg(all + (size_t)v * G + rank, p);
        }
        grid.sync();
        for (int v = warp; v < cnt; v += GS_WARPS) {
            double sr = 0.0, si = 0.0;
            for (int c = lane; c < G; c += 32) {
                const double2 t = __ldcg(all + (size_t)v * G + c);
                sr += t.x;
                si += t.y;
            }
            sr = warp_sum(sr);
            si = warp_sum(si);
            if (lane == 0) out[v] = make_double2(sr, si);
        }
        buf ^= 1;
        __syncthreads();
    };
    auto norm = [&]() -> double {
        reduce(1, h + (m + 1), [&](int) {
            double s = 0.0;
            for (int i = lane; i < rows; i += 32) s += w[i].x * w[i].x + w[i].y * w[i].y;
            return make_double2(warp_sum(s), 0.0);
        });
        return sqrt(h[m + 1].x);
    };

    // CTA 0 rotates at the end: the earlier rotations and g into shared memory now
    double2 *rot = part + (size_t)GS_WARPS * 32;  // cs [k], sn [k], g[k]
    const double2 *cs0 = a.small + (size_t)(m + 1) * m;
    if (rank == 0 && !a.b)
        for (int t = tid; t <= 2 * k; t += GS_THREADS)
            rot[t] = t < k ? cs0[t] : (t < 2 * k ? cs0[m + t - k] : cs0[2 * m + k]);

    // w = (b -) A v from the matvec's partial sums: 32 rows at a time, every
    // eighth split per warp, the warps added in order
    for (int r0 = 0; r0 < rows; r0 += 32) {
        const int i = r0 + lane;
        double sr = 0.0, si = 0.0;
        if (i < rows) {
            const double2 *p = a.partial + i0 + i;
#pragma unroll 8
            for (int s = warp; s < a.splits; s += GS_WARPS) {
                const double2 t = __ldcs(p + (int64_t)s * n);
                sr += t.x;
                si += t.y;
            }
        }
        part[warp * 32 + lane] = make_double2(sr, si);
        __syncthreads();
        if (warp == 0 && i < rows) {
            sr = si = 0.0;
            for (int q = 0; q < GS_WARPS; ++q) {
                sr += part[q * 32 + lane].x;
                si += part[q * 32 + lane].y;
            }
            if (a.b) {
                const double2 bi = a.b[i0 + i];
                sr = bi.x - sr;
                si = bi.y - si;
            }
            w[i] = make_double2(sr, si);
        }
        __syncthreads();
    }

    GmresState *st = a.state;
    double2 *H = a.small, *cs = H + (size_t)(m + 1) * m, *sn = cs + m, *g = sn + m;
    if (a.b) {
        // a new cycle from the residual: V_0 = r / |r|, g = |r| e_1
        const double beta = norm();
        const double s = beta > 0.0 ? 1.0 / beta : 0.0;
        for (int i = tid; i < rows; i += GS_THREADS) V[i0 + i] = make_double2(w[i].x * s, w[i].y * s);
        if (rank == 0 && tid == 0) {
            if (a.first) {
                st->r0 = beta;
                st->iters = 0;
                st->rel = 0.0;
            }
            st->kdone = 0;
            g[0] = make_double2(beta, 0.0);
            // a zero residual: solved
            const int flag = beta == 0.0 ? GMRES_ZERO : GMRES_GO;
            if (flag != GMRES_GO) *a.active = 0;
            a.host->rel = beta == 0.0 ? 0.0 : st->rel;
            a.host->iters = st->iters;
            a.host->flag = flag;
            __threadfence_system();
            a.host->seq = a.seq;
        }
        return;
    }

    // out[v] = V_v^H w, v <= k: a vector a thread
    auto project_long = [&](double2 *out) {
        double2 *all = a.sums + (size_t)buf * (m + 1) * G;
        for (int v = tid; v <= k; v += GS_THREADS) {
            const double2 *Vv = V + (int64_t)v * n + i0;
            double sr = 0.0, si = 0.0;
#pragma unroll 4
            for (int i = 0; i < rows; ++i) {
                const double2 q = cmulc(Vv[i], w[i]);
                sr += q.x;
                si += q.y;
            }
            __stcg(all + (size_t)rank * (m + 1) + v, make_double2(sr, si));
        }
        grid.sync();
        for (int v = tid; v <= k; v += GS_THREADS) {
            double sr = 0.0, si = 0.0;
#pragma unroll 8
            for (int c = 0; c < G; ++c) {
                const double2 t = __ldcg(all + (size_t)c * (m + 1) + v);
                sr += t.x;
                si += t.y;
            }
            out[v] = make_double2(sr, si);
        }
        buf ^= 1;
        __syncthreads();
    };

    // CGS2: h = V^H w, w -= V h, twice (the second time h2)
    for (int pass = 0; pass < 2; ++pass) {
        double2 *hp = pass ? h2 : h;
        if constexpr (LONG) {
            project_long(hp);
            // 32 rows at a time, every eighth vector per warp, the warps subtracted in order
            for (int r0 = 0; r0 < rows; r0 += 32) {
                const int i = r0 + lane;
                double sr = 0.0, si = 0.0;
                if (i < rows) {
                    const double2 *Vi = V + i0 + i;
#pragma unroll 4
                    for (int v = warp; v <= k; v += GS_WARPS) {
                        const double2 q = cmul2(__ldcg(Vi + (int64_t)v * n), hp[v]);
                        sr += q.x;
                        si += q.y;
                    }
                }
                part[warp * 32 + lane] = make_double2(sr, si);
                __syncthreads();
                if (warp == 0 && i < rows) {
                    double2 x = w[i];
                    for (int q = 0; q < GS_WARPS; ++q) {
                        x.x -= part[q * 32 + lane].x;
                        x.y -= part[q * 32 + lane].y;
                    }
                    w[i] = x;
                }
                __syncthreads();
            }
            continue;
        }
        reduce(k + 1, hp, [&](int v) {
            const double2 *Vv = V + (int64_t)v * n + i0;
            double sr = 0.0, si = 0.0;
            for (int i = lane; i < rows; i += 32) {
                const double2 q = cmulc(__ldcg(Vv + i), w[i]);
                sr += q.x;
                si += q.y;
            }
            return make_double2(warp_sum(sr), warp_sum(si));
        });
        for (int i = tid; i < rows; i += GS_THREADS) {
            double2 x = w[i];
            const double2 *Vi = V + i0 + i;
#pragma unroll 4
            for (int v = 0; v <= k; ++v) {
                const double2 q = cmul2(__ldcg(Vi + (int64_t)v * n), hp[v]);
                x.x -= q.x;
                x.y -= q.y;
            }
            w[i] = x;
        }
        __syncthreads();
    }
    const double hn = norm();
    if (hn > 0.0) {
        const double s = 1.0 / hn;
        double2 *Vn = V + (int64_t)(k + 1) * n + i0;
        for (int i = tid; i < rows; i += GS_THREADS) Vn[i] = make_double2(w[i].x * s, w[i].y * s);
    }
    if (rank != 0) return;
    // the column of H is the sum of both projections; a cycle may have more
    // steps than the block threads
    for (int v = tid; v <= k; v += GS_THREADS) h[v] = make_double2(h[v].x + h2[v].x, h[v].y + h2[v].y);
    __syncthreads();
    if (tid == 0) {
        // the previous rotations, then a new one zeroing the subdiagonal
        double2 *Hk = H + (size_t)k * (m + 1);
        h[k + 1] = make_double2(hn, 0.0);
        for (int i = 0; i < k; ++i) {
            const double2 ci = rot[i], si = rot[k + i];
            const double2 a0 = h[i], a1 = h[i + 1], u = cmulc(ci, a0), v = cmulc(si, a1);
            const double2 p = cmul2(ci, a1), q = cmul2(si, a0);
            h[i] = make_double2(u.x + v.x, u.y + v.y);
            h[i + 1] = make_double2(p.x - q.x, p.y - q.y);
        }
        const double2 a0 = h[k], a1 = h[k + 1];
        const double den = sqrt(a0.x * a0.x + a0.y * a0.y + a1.x * a1.x + a1.y * a1.y), id = 1.0 / den;
        const double2 c = den == 0.0 ? make_double2(1.0, 0.0) : make_double2(a0.x * id, a0.y * id);
        const double2 s = den == 0.0 ? make_double2(0.0, 0.0) : make_double2(a1.x * id, a1.y * id);
        cs[k] = c;
        sn[k] = s;
        const double2 u = cmulc(c, a0), v = cmulc(s, a1);
        h[k] = make_double2(u.x + v.x, u.y + v.y);
        for (int i = 0; i <= k; ++i) Hk[i] = h[i];
        const double2 g0 = rot[2 * k], gk = cmulc(c, g0), gn = cmul2(s, g0);
        g[k] = gk;
        g[k + 1] = make_double2(-gn.x, -gn.y);
        const double rel = sqrt(gn.x * gn.x + gn.y * gn.y) / st->r0;
        const int iters = st->iters + 1;
        st->iters = iters;
        st->rel = rel;
        st->kdone = k + 1;
        const bool stop = rel < a.tol || iters >= a.max_iters || hn == 0.0 || k + 1 == n;
        const int flag = stop ? GMRES_STOP : (k + 1 == m ? GMRES_CYCLE : GMRES_GO);
        if (flag != GMRES_GO) *a.active = 0;
        a.host->rel = rel;
        a.host->iters = iters;
        a.host->flag = flag;
        __threadfence_system();
        a.host->seq = a.seq;
    }
}

// y = H^{-1} g over kdone steps (every block repeats it), x += V y
__global__ void __launch_bounds__(256) k_gmres_update(GmresStep a, double2 *x)
{
    extern __shared__ double2 y[];
    const int m = a.restart, kd = a.state->kdone;
    const double2 *H = a.small, *g = H + (size_t)(m + 1) * m + 2 * m;
    // column by column: y_j, then its share of the rows above
    for (int i = threadIdx.x; i < kd; i += blockDim.x) y[i] = g[i];
    __syncthreads();
    for (int j = kd - 1; j >= 0; --j) {
        const double2 d = H[(size_t)j * (m + 1) + j], t = y[j];
        const double q = d.x * d.x + d.y * d.y;
        const double2 yj = make_double2((t.x * d.x + t.y * d.y) / q, (t.y * d.x - t.x * d.y) / q);
        __syncthreads();
        if (threadIdx.x == 0) y[j] = yj;
        for (int i = threadIdx.x; i < j; i += blockDim.x) {
            const double2 p = cmul2(H[(size_t)j * (m + 1) + i], yj);
            y[i].x -= p.x;
            y[i].y -= p.y;
        }
        __syncthreads();
    }
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    double2 acc = x[i];
#pragma unroll 4
    for (int v = 0; v < kd; ++v) {
        const double2 p = cmul2(a.V[(int64_t)v * a.n + i], y[v]);
        acc.x += p.x;
        acc.y += p.y;
    }
    x[i] = acc;
}

}  // namespace

cudaError_t gmres_step_plan(int64_t n, int restart, int device, int max_ctas, GmresPlan *plan)
{
    int optin = 0, sms = 0, per_sm = 0;
    cudaError_t e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_gmres_step<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e == cudaSuccess && restart >= GS_LONG)
        e = cudaFuncSetAttribute(k_gmres_step<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
    if (e != cudaSuccess) return e;
    plan->ctas = (int)std::max<int64_t>(1, std::min<int64_t>((n + GS_ROWS - 1) / GS_ROWS, std::min(sms, max_ctas)));
    plan->smem = sizeof(double2) * (2 * (size_t)restart + 3 + GS_WARPS * 32 + 2 * (size_t)restart + 1 +
                                    (size_t)((n + plan->ctas - 1) / plan->ctas));
    if (plan->smem > (size_t)optin) return cudaErrorInvalidValue;
    e = restart >= GS_LONG
            ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gmres_step<true>, GS_THREADS, plan->smem)
            : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_gmres_step<false>, GS_THREADS, plan->smem);
    if (e == cudaSuccess && per_sm < 1) e = cudaErrorInvalidConfiguration;
    return e;
}

cudaError_t launch_gmres_step(const GmresStep &a, const GmresPlan &plan, cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(plan.ctas);
    cfg.blockDim = dim3(GS_THREADS);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return !a.b && a.k + 1 >= GS_LONG ? cudaLaunchKernelEx(&cfg, k_gmres_step<true>, a)
                                      : cudaLaunchKernelEx(&cfg, k_gmres_step<false>, a);
}

cudaError_t launch_gmres_update(const GmresStep &a, double2 *x, cudaStream_t s)
{
    k_gmres_update<<<(unsigned)((a.n + 255) / 256), 256, sizeof(double2) * (size_t)a.restart, s>>>(a, x);
    return cudaGetLastError();
}

}  // namespace nihu
