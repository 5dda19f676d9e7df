// Regular (far-field) collocational entries: fused SLP + DLP over all
// (test, trial) element pairs, in FP32 (default) or FP64.
//
// Restates nihu/core/double_integral.hpp:445-467 (sum_q w_q K(x_i, y_q) J_q
// with the accelerator of the selected degree, :557-585) for the Helmholtz and
// Laplace 3D SLP/DLP kernels (nihu/library/helmholtz_kernel.hpp:180-195,
// laplace_kernel.hpp:137-147, normal_derivative_kernel.hpp:131-175).
//
// Work layout (k_regular): a block owns REG_THREADS consecutive test rows and up
// to REG_COLS consecutive trial columns.  A thread owns one row; for each column it
// classifies the pair (classify.cuh), evaluates the selected rule(s) and
// writes the entry.  Writes of a warp are 32 consecutive entries of one
// column of the column-major matrix (256 B for complex64), so the dominant
// cost -- storing 2 x 8 bytes per pair -- streams at full HBM width.
// Self and nearly singular pairs are skipped (assemble_singular.cu writes
// them), so every entry is written exactly once.
//
// Right-hand-side mode (frequency batches, RegularArgs::rhs_part): the SLP
// entries are not stored; each thread sums SLP_f(i, j) q_f(j) over its
// block's columns per wave number in shared memory, the block writes one
// partial sum per (wave number, row), and k_rhs_reduce adds the partials and
// the FP64 kernel's nearly singular and self entries in a fixed order.  This
// is b = SLP q of the collocation system without the SLP matrix.
#include <algorithm>
#include <type_traits>

#include "classify.cuh"
#include "kernels.h"
#include "two_row.cuh"

namespace nihu {

constexpr int REG_THREADS = 256;
constexpr int REG_COLS = 32;

// k-independent part of one quadrature point (frequency batches): the
// distance and the SLP and DLP factors of eval_point
template <typename R>
struct PointGeom {
    R r, gs, fd;
};

template <typename R>
__device__ __forceinline__ PointGeom<R> point_geom(R rx, R ry, R rz, R wj, R nx, R ny, R nz, R ws, R wd)
{
    constexpr R INV4PI = R(1.0 / (4.0 * 3.14159265358979323846));
    R r2 = rx * rx + ry * ry + rz * rz;
    R rinv;
    if constexpr (sizeof(R) == 4) rinv = rsqrtf(r2);
    else rinv = rsqrt(r2);
    R g = wj * rinv * INV4PI;
    R rdn = (rx * nx + ry * ny + rz * nz) * rinv;
    return {r2 * rinv, g * ws, -g * rinv * rdn * wd};
}

// the k-dependent part: the same sums as eval_point
template <int FAM, typename R>
__device__ __forceinline__ void point_freq(const PointGeom<R> &p, R k, R &sr, R &si, R &dr, R &di)
{
    if constexpr (FAM == FAM_HELMHOLTZ) {
        R kr = k * p.r;
        R s, c;
        if constexpr (sizeof(R) == 4) sincos_reduced(kr, s, c);
        else sincos(kr, &s, &c);
        sr += p.gs * c;
        si -= p.gs * s;
        dr += p.fd * (c + kr * s);
        di += p.fd * (kr * c - s);
    } else {
        sr += p.gs;
        dr += p.fd;
    }
}

// wave numbers evaluated together per pass over a pair's points
constexpr int FREQ_TILE = 4;

template <typename Out, typename R>
__device__ __forceinline__ void store_entry(Out *p, R re, R im, R are, R aim, bool unit_alpha, int accumulate)
{
    R vr = re, vi = im;
    if (!unit_alpha) {
        vr = are * re - aim * im;
        vi = are * im + aim * re;
    }
    Out o;
    if (accumulate) {
        o = *p;
        o.x += vr;
        o.y += vi;
    } else {
        o.x = vr;
        o.y = vi;
    }
    *p = o;
}

// right-hand-side mode: wave numbers per block (the gridDim.z split keeps at
// most this many), which sizes the shared row sums and Neumann data
template <typename R>
__host__ __device__ constexpr int rhs_f_max() { return sizeof(R) == 4 ? 16 : 8; }

// the wave numbers per block a launch uses: RegularArgs::rhs_fmax within the
// cap that keeps the shared memory under 48 KB, else the default
template <typename R>
__host__ __device__ inline int rhs_fmax_of(const RegularArgs &a)
{
    constexpr int cap = sizeof(R) == 4 ? 20 : 10;
    return a.rhs_fmax > 0 ? (a.rhs_fmax < cap ? a.rhs_fmax : cap) : rhs_f_max<R>();
}

template <typename R>
using Cplx = std::conditional_t<sizeof(R) == 4, float2, double2>;

// acc += (sr + i si) q
template <typename R2, typename R>
__device__ __forceinline__ void rhs_add(R2 &acc, const R2 q, R sr, R si)
{
    acc.x += sr * q.x - si * q.y;
    acc.y += sr * q.y + si * q.x;
}

// frequency batches store plain entries (unit scale, no accumulation:
// launch_assemble_regular refuses anything else)
template <typename Out, typename R>
__device__ __forceinline__ void store_plain(Out *p, R re, R im)
{
    Out o;
    o.x = re;
    o.y = im;
    *p = o;
}

// the outputs of a frequency batch from wave number f on: a pointer that
// steps by mat_stride, or (TAB) the device table outs (separate matrices);
// the kernel picks the variant once, outside its wave number loops
template <typename Out, bool TAB>
struct BatchCursor {
    Out *p = nullptr;
    void *const *tab = nullptr;
    int64_t step, off;
    __device__ __forceinline__ BatchCursor(const RegularArgs &a, bool dlp, int f, int64_t off_)
        : step(a.mat_stride), off(off_)
    {
        if constexpr (TAB) {
            tab = a.outs + (dlp ? a.nk : 0) + f;
        } else {
            Out *base = reinterpret_cast<Out *>(dlp ? a.out_d : a.out_s);
            p = base ? base + (int64_t)f * a.mat_stride + off : nullptr;
        }
    }
    __device__ __forceinline__ Out *get() const
    {
        if constexpr (TAB) return reinterpret_cast<Out *>(*tab) + off;
        else return p;
    }
    __device__ __forceinline__ void next()
    {
        if constexpr (TAB) ++tab;
        else p += step;
    }
};

// Squared distance ratio above which a pair is certainly regular with the
// 1-point rule for both SLP (x >= 9.1) and DLP (x >= 15.8): 15.8^2 with a
// relative margin far larger than the FP32 error of the plain centre
// difference of a far pair.
constexpr float Q_FAR = 249.64f * (1.0f + 1e-4f);

// BATCH: frequency batch (a.nk > 1), a separate instantiation so that the
// single wave number kernel carries none of its code
// RHS: right-hand-side mode (BATCH only; the SLP entries go into the row sums)
// PLAIN: unit scale and no accumulation (single wave number, FP32), so the
// stores carry no run-time checks
// CK: a complex (lossy) wave number k + i k_im (single wave number, Helmholtz;
// its own instantiation, so the real-k kernels carry none of it)
template <typename R, typename Out, int FAM, int OPS, bool BATCH, bool RHS = false, bool PLAIN = false,
          bool CK = false>
__global__ void __launch_bounds__(REG_THREADS) k_regular(RegularArgs a)
{
    using R2 = Cplx<R>;
    __shared__ float4 s_hi[REG_COLS], s_lo[REG_COLS], s_p0[REG_COLS];
    __shared__ int s_nc[REG_COLS];
    // RHS: Neumann data [f - f_lo][c], then the row sums [f - f_lo][threadIdx.x]
    extern __shared__ __align__(16) unsigned char s_rhs[];
    R2 *s_q = reinterpret_cast<R2 *>(s_rhs);
    R2 *s_acc = s_q + rhs_fmax_of<R>(a) * REG_COLS;
    constexpr bool DO_S = (OPS & OP_SLP) != 0;
    constexpr bool DO_D = (OPS & OP_DLP) != 0;
    const DevMesh &test = a.test;
    const DevMesh &trial = a.trial;
    const int i = blockIdx.x * REG_THREADS + threadIdx.x;
    // the launch's split of the columns; frequency batches: whole column blocks (rhs_part)
    const int cpb = BATCH ? REG_COLS : (int)((a.j1 - a.j0 + gridDim.y - 1) / gridDim.y);
    const int jb = a.j0 + blockIdx.y * cpb;
    const int ncols = min(cpb, a.j1 - jb);
    // frequency batch: this block's wave numbers [f_lo, f_hi) (gridDim.z chunks)
    const int f_per = (a.nk + gridDim.z - 1) / gridDim.z;
    const int f_lo = min(a.nk, (int)blockIdx.z * f_per), f_hi = min(a.nk, f_lo + f_per);
    if (threadIdx.x < ncols) {
        s_hi[threadIdx.x] = trial.chi[jb + threadIdx.x];
        s_lo[threadIdx.x] = trial.clo[jb + threadIdx.x];
        s_nc[threadIdx.x] = trial.nc[jb + threadIdx.x];
        s_p0[threadIdx.x] = trial.p0[jb + threadIdx.x];
    }
    if constexpr (RHS) {
        const int nf = f_hi - f_lo;  // at most rhs_fmax_of (launch_assemble_regular)
        for (int t = threadIdx.x; t < nf * REG_COLS; t += REG_THREADS) {
            const int fl = t / REG_COLS, c = t - fl * REG_COLS;
            R2 v;
            v.x = 0;
            v.y = 0;
            if (c < ncols) {
                const double2 qv = a.rhs_q[(int64_t)(f_lo + fl) * trial.n + jb + c];
                v.x = R(qv.x);
                v.y = R(qv.y);
            }
            s_q[t] = v;
        }
        for (int fl = 0; fl < nf; ++fl) {
            R2 z;
            z.x = 0;
            z.y = 0;
            s_acc[fl * REG_THREADS + threadIdx.x] = z;
        }
    }
    __syncthreads();
    // whole warps beyond the last row leave; a partial last warp keeps its
    // out-of-range lanes (clamped to the last row, writes masked) so that
    // warp votes see every lane
    if ((i & ~31) >= test.n) return;
    const bool row_ok = i < test.n;
    const int ii = row_ok ? i : test.n - 1;

    const float4 ih = test.chi[ii], il = test.clo[ii];
    const int par = il.w != 0.0f ? 1 : 0;
    R k, are, aim, kim;
    if constexpr (sizeof(R) == 4) {
        kim = a.k_im32;
        k = a.k32;
        are = a.alpha_re32;
        aim = a.alpha_im32;
    } else {
        kim = a.k_im;
        k = a.k;
        are = a.alpha_re;
        aim = a.alpha_im;
    }
    (void)kim;
    // one quadrature point of the single wave number paths
    auto ev = [&](R rx, R ry, R rz, R wj, R nx, R ny, R nz, R ws, R wd, R &sr, R &si, R &dr, R &di) {
        if constexpr (CK) eval_point_ck<R>(rx, ry, rz, wj, nx, ny, nz, k, kim, ws, wd, sr, si, dr, di);
        else eval_point<FAM, R>(rx, ry, rz, wj, nx, ny, nz, k, ws, wd, sr, si, dr, di);
    };
    const bool unit_alpha = a.unit_alpha != 0;
    const int accumulate = a.accumulate;
    R x0, x1, x2;
    if constexpr (sizeof(R) == 8) {
        x0 = test.center[3 * (int64_t)ii];
        x1 = test.center[3 * (int64_t)ii + 1];
        x2 = test.center[3 * (int64_t)ii + 2];
    } else {
        x0 = ih.x + il.x;
        x1 = ih.y + il.y;
        x2 = ih.z + il.z;
    }
    Out *out_s = reinterpret_cast<Out *>(a.out_s);
    Out *out_d = reinterpret_cast<Out *>(a.out_d);
    // single wave number: this thread's entries of the current column, one
    // column (ld entries) further per step
    const int64_t ldo = a.ld;
    Out *ps = DO_S && !BATCH ? out_s + (int64_t)(jb - a.j0) * ldo + i : nullptr;
    Out *pd = DO_D && !BATCH ? out_d + (int64_t)(jb - a.j0) * ldo + i : nullptr;
    auto put = [&](Out *p, R re, R im) {
        if constexpr (PLAIN) store_plain(p, re, im);
        else store_entry(p, re, im, are, aim, unit_alpha, accumulate);
    };

    for (int c = 0; c < ncols; ++c, ps += DO_S && !BATCH ? ldo : 0, pd += DO_D && !BATCH ? ldo : 0) {
        const int j = jb + c;
        if constexpr (sizeof(R) == 4) {
            // far-field fast path, taken when every lane of the warp is a far
            // pair: one centroid point for both operators
            // the hi/lo centre difference: FP32 relative accuracy of r, which
            // the DLP's r.n of nearly coplanar far pairs needs
            const float4 h = s_hi[c], l = s_lo[c];
            const float fx = (h.x - ih.x) + (l.x - il.x), fy = (h.y - ih.y) + (l.y - il.y),
                        fz = (h.z - ih.z) + (l.z - il.z);
            const float q = (fx * fx + fy * fy + fz * fz) * h.w;
            if (__all_sync(0xffffffffu, q > Q_FAR)) {
                const float4 p = s_p0[c];
                if constexpr (BATCH) {
                    const int64_t off = (int64_t)(j - a.j0) * a.ld + i;
                    const PointGeom<float> gm = point_geom<float>(fx, fy, fz, p.x, p.y, p.z, p.w, R(DO_S), R(DO_D));
                    auto freqs = [&](auto tab) {
                        constexpr bool TAB = decltype(tab)::value;
                        BatchCursor<Out, TAB> cs(a, false, f_lo, off), cd(a, true, f_lo, off);
                        R2 *acc = s_acc + threadIdx.x;
                        const R2 *qc = s_q + c;
                        const float *kp = a.ks32 + f_lo;
                        for (int f = f_lo; f < f_hi; ++f) {
                            R sr = 0, si = 0, dr = 0, di = 0;
                            point_freq<FAM, float>(gm, *kp++, sr, si, dr, di);
                            if (row_ok) {
                                if constexpr (RHS) rhs_add(*acc, *qc, sr, si);
                                else if (DO_S) store_plain(cs.get(), sr, si);
                                if (DO_D) store_plain(cd.get(), dr, di);
                            }
                            if constexpr (RHS) {
                                acc += REG_THREADS;
                                qc += REG_COLS;
                            } else if (DO_S) {
                                cs.next();
                            }
                            if (DO_D) cd.next();
                        }
                    };
                    if (a.outs) freqs(std::true_type{});
                    else freqs(std::false_type{});
                } else {
                    R sr = 0, si = 0, dr = 0, di = 0;
                    ev(fx, fy, fz, p.x, p.y, p.z, p.w, R(DO_S), R(DO_D), sr, si, dr, di);
                    if (row_ok) {
                        if (DO_S) put(ps, sr, si);
                        if (DO_D) put(pd, dr, di);
                    }
                }
                continue;
            }
        }
        if constexpr (sizeof(R) == 4 && !BATCH && OPS == (OP_SLP | OP_DLP)) {
            // every lane certainly has the 1-point SLP rule (d/D >= 9.1) and a
            // certain DLP level, 0 (d/D >= 15.8) or 1 (below): the general
            // path's points in its order -- the centroid, then for level 1 the
            // DLP-only points -- without its per-lane dispatch.  "Certainly"
            // is classify_pair's FP32 guard band, so the levels are its own.
            const float4 jh = s_hi[c], jl = s_lo[c];
            const float mx = (jh.x - ih.x) + (jl.x - il.x), my = (jh.y - ih.y) + (jl.y - il.y),
                        mz = (jh.z - ih.z) + (jl.z - il.z);
            const float mq = (mx * mx + my * my + mz * mz) * jh.w;
            const float mlo = mq * (1.0f - 1e-5f), mhi = mq * (1.0f + 1e-5f);
            const bool d_far = mlo >= 249.64f;
            if (__all_sync(0xffffffffu, mlo >= 82.81f && (d_far || mhi < 249.64f))) {
                if (row_ok) {
                    const int64_t base = ((int64_t)j * 2 + par) * SLOTS;
                    R sr = 0, si = 0, dr = 0, di = 0;
                    const float4 yc = __ldg(trial.pts32 + 2 * base), nc = __ldg(trial.pts32 + 2 * base + 1);
                    ev(mx, my, mz, yc.w, nc.x, nc.y, nc.z, R(1), d_far ? R(1) : R(0), sr, si, dr, di);
                    if (!d_far) {
                        const int npd = level_npts(s_nc[c], par, 1);
                        for (int q = 0; q < npd; ++q) {
                            const int64_t sl = base + level_slot0(1) + q;
                            const float4 y = __ldg(trial.pts32 + 2 * sl), n = __ldg(trial.pts32 + 2 * sl + 1);
                            ev(mx + y.x, my + y.y, mz + y.z, y.w, n.x, n.y, n.z, R(0), R(1), sr, si, dr, di);
                        }
                    }
                    put(ps, sr, si);
                    put(pd, dr, di);
                }
                continue;
            }
        }
        int ls, ld;
        float dx, dy, dz;
        int kind = classify_pair(ih, il, s_hi[c], s_lo[c], ii, j, test.center, trial.center, trial.size,
                                 a.same_mesh, ls, ld, dx, dy, dz);
        if (kind != KIND_REGULAR || !row_ok) continue;
        if (!DO_S) ls = ld;
        if (!DO_D) ld = ls;
        // one uniform loop over this lane's points: SLP and DLP at the same
        // level share every point; otherwise the SLP points come first
        const int tnc = s_nc[c];
        const int nps = level_npts(tnc, par, ls);
        const int npd = level_npts(tnc, par, ld);
        const int n_eval = ls == ld ? nps : nps + npd;
        const int64_t base = ((int64_t)j * 2 + par) * SLOTS;
        if constexpr (BATCH) {
            // frequency batch: each point's geometry once per tile of wave numbers
            const int64_t off = (int64_t)(j - a.j0) * a.ld + i;
            auto tiles = [&](auto tab) {
                constexpr bool TAB = decltype(tab)::value;
                BatchCursor<Out, TAB> cs(a, false, f_lo, off), cd(a, true, f_lo, off);
                R2 *acc = s_acc + threadIdx.x;
                const R2 *qc = s_q + c;
                for (int f0 = f_lo; f0 < f_hi; f0 += FREQ_TILE) {
                    R kf[FREQ_TILE], sr[FREQ_TILE], si[FREQ_TILE], dr[FREQ_TILE], di[FREQ_TILE];
#pragma unroll
                    for (int u = 0; u < FREQ_TILE; ++u) {
                        if constexpr (sizeof(R) == 4) kf[u] = f0 + u < f_hi ? a.ks32[f0 + u] : 0.0f;
                        else kf[u] = f0 + u < f_hi ? a.ks[f0 + u] : 0.0;
                        sr[u] = si[u] = dr[u] = di[u] = 0;
                    }
                    for (int q = 0; q < n_eval; ++q) {
                        int slot;
                        R ws, wd;
                        if (ls == ld) { slot = level_slot0(ls) + q; ws = R(DO_S); wd = R(DO_D); }
                        else if (q < nps) { slot = level_slot0(ls) + q; ws = R(1); wd = R(0); }
                        else { slot = level_slot0(ld) + q - nps; ws = R(0); wd = R(1); }
                        PointGeom<R> gm;
                        if constexpr (sizeof(R) == 4) {
                            const float4 y = __ldg(trial.pts32 + 2 * (base + slot));
                            const float4 n = __ldg(trial.pts32 + 2 * (base + slot) + 1);
                            gm = point_geom<float>(dx + y.x, dy + y.y, dz + y.z, y.w, n.x, n.y, n.z, ws, wd);
                        } else {
                            const double *y = trial.pts64 + 8 * (base + slot);
                            gm = point_geom<double>(y[0] - x0, y[1] - x1, y[2] - x2, y[3], y[4], y[5], y[6], ws, wd);
                        }
#pragma unroll
                        for (int u = 0; u < FREQ_TILE; ++u) point_freq<FAM, R>(gm, kf[u], sr[u], si[u], dr[u], di[u]);
                    }
#pragma unroll
                    for (int u = 0; u < FREQ_TILE; ++u) {
                        if (f0 + u >= f_hi) break;
                        if constexpr (RHS) {
                            rhs_add(*acc, *qc, sr[u], si[u]);
                            acc += REG_THREADS;
                            qc += REG_COLS;
                        } else if (DO_S) {
                            store_plain(cs.get(), sr[u], si[u]);
                            cs.next();
                        }
                        if (DO_D) {
                            store_plain(cd.get(), dr[u], di[u]);
                            cd.next();
                        }
                    }
                }
            };
            if (a.outs) tiles(std::true_type{});
            else tiles(std::false_type{});
        } else {
            R sr = 0, si = 0, dr = 0, di = 0;
            for (int q = 0; q < n_eval; ++q) {
                int slot;
                R ws, wd;
                if (ls == ld) { slot = level_slot0(ls) + q; ws = R(DO_S); wd = R(DO_D); }
                else if (q < nps) { slot = level_slot0(ls) + q; ws = R(1); wd = R(0); }
                else { slot = level_slot0(ld) + q - nps; ws = R(0); wd = R(1); }
                if constexpr (sizeof(R) == 4) {
                    const float4 y = __ldg(trial.pts32 + 2 * (base + slot));
                    const float4 n = __ldg(trial.pts32 + 2 * (base + slot) + 1);
                    // r = (c_j - x) + (y - c_j): the hi/lo centre difference plus the
                    // point's offset from the trial centre
                    ev(dx + y.x, dy + y.y, dz + y.z, y.w, n.x, n.y, n.z, ws, wd, sr, si, dr, di);
                } else {
                    const double *y = trial.pts64 + 8 * (base + slot);
                    ev(y[0] - x0, y[1] - x1, y[2] - x2, y[3], y[4], y[5], y[6], ws, wd, sr, si, dr, di);
                }
            }
            if (DO_S) put(ps, sr, si);
            if (DO_D) put(pd, dr, di);
        }
    }
    if constexpr (RHS) {
        if (row_ok) {
            R2 *part = reinterpret_cast<R2 *>(a.rhs_part);
            for (int f = f_lo; f < f_hi; ++f) {
                R2 v = s_acc[(f - f_lo) * REG_THREADS + threadIdx.x];
                if (!unit_alpha) {
                    const R vr = are * v.x - aim * v.y;
                    v.y = are * v.y + aim * v.x;
                    v.x = vr;
                }
                part[((int64_t)f * gridDim.y + blockIdx.y) * test.n + i] = v;
            }
        }
    }
}

int regular_carveout_percent() { return TWO_ROW_CARVEOUT; }

// ------------------------------------------------- two rows per thread
// The FP32 kernel of a single wave number into complex64 matrices, through the
// column loop of two_row.cuh: a thread owns two rows, far columns take one
// vote and two centroid points, the other pairs are listed by rule,
//   0  9.1 <= d/D < 15.8: the centroid for the SLP, the level-1 points for the DLP
//   1  2.8 <= d/D < 9.1: the level-1 points for both
//   2  all others (closer, or within the FP32 guard band of a limit): classify_pair
// (with one operator: its own one-point limit is "far", the pairs down to its
// next limit list 1) and worked through one pair per lane, so that a pair
// costs its own points and not its warp's largest count.  Points, levels and
// their order are those of k_regular.
//
// Bound by FP32 issue, then by the stores (16 B a pair, 0.99 ms at the copy
// bandwidth).  Sphere of 20480 triangles, SLP and DLP, the whole step with the
// singular kernel beside it: 1.434 -> 1.386 ms against a form with scalar far
// rows, one list for everything below 9.1 D and 512 x 32 tiles; 320 triangles,
// this kernel: 110 -> 13 us (10 blocks before).  Tiles of 512 x 32 / 256 x 32 /
// 256 x 16 / 256 x 8 / 128 x 32 pairs: 1.458 / 1.430 / 1.382 / 1.416 / 1.436 ms: a
// block ends with its slowest warp, so small ones keep more warps running,
// until the staging shows.  Listed pairs packed in twos spill (1.54 ms).
// one point of the SLP (S_) and DLP (D_) kernels of two pairs, added to v:
// w4 = w J / (4 pi), rn = r.n; e^{-ikr} / (4 pi r) and
// -(1 + ikr) e^{-ikr} (r.n) / (4 pi r^3), CK: of a complex wave number k + i ki
struct Reg2Val {
    f2 sr, si, dr, di;
};
template <int FAM, bool CK, bool S_, bool D_>
__device__ __forceinline__ void reg2_point(f2 r2, f2 w4, f2 rn, float k, float ki, Reg2Val &v)
{
    const f2 rinv = f2_rsqrt(r2);
    const f2 g = w4 * rinv;
    f2 f{};  // g (r.n) / r^2: minus the DLP's factor
    if constexpr (D_) f = (g * (rinv * rinv)) * rn;
    if constexpr (FAM == FAM_HELMHOLTZ) {
        // with the sine of -kr: e^{-ikr} = cs + i sn; the DLP as -f (1 + ikr) e^{-ikr}
        const f2 r = r2 * rinv, nkr = r * f2_dup(-k);
        f2 sn, cs;
        f2_sincos_reduced(nkr, sn, cs);
        f2 na1 = f2_dup(-1.0f);
        if constexpr (CK) {
            float x, y;
            f2_unpack(r * f2_dup(ki), x, y);
            const f2 damp = f2_pack(expf(x), expf(y));
            cs = cs * damp;
            sn = sn * damp;
            na1 = f2_fma(r, f2_dup(ki), na1);
        }
        if constexpr (S_) {
            v.sr = f2_fma(g, cs, v.sr);
            v.si = f2_fma(g, sn, v.si);
        }
        if constexpr (D_) {
            // -(a1 + i kr)(cs + i sn) = (na1 cs + kr sn) + i (na1 sn - kr cs)
            const f2 kr = r * f2_dup(k);
            v.dr = f2_fma(f, f2_fma(kr, sn, na1 * cs), v.dr);
            v.di = f2_fma(f, f2_fma(nkr, cs, na1 * sn), v.di);
        }
    } else {
        if constexpr (S_) v.sr = v.sr + g;
        if constexpr (D_) v.dr = f2_fma(f, f2_dup(-1.0f), v.dr);
    }
}

// the same of one pair (the listed ones: packed in twos they need more
// registers than the loop leaves, and spill).  W4: w is w J / (4 pi), else w J: points
// of equal weights then round their products with 1 / (4 pi) one by one, which
// their sum averages
template <int FAM, bool CK, bool S_, bool D_, bool W4>
__device__ __forceinline__ void reg2_point1(float rx, float ry, float rz, float w, float rn, float k, float ki, float4 &o)
{
    constexpr float INV4PI = 0.0795774715459476679f;
    const float r2 = rx * rx + ry * ry + rz * rz;
    const float rinv = rsqrtf(r2);
    const float g = W4 ? w * rinv : w * rinv * INV4PI;
    if constexpr (FAM == FAM_HELMHOLTZ) {
        const float r = r2 * rinv, kr = k * r;
        float sn, cs, a1 = 1.0f;
        sincos_reduced(kr, sn, cs);
        if constexpr (CK) {
            const float damp = expf(ki * r);
            sn *= damp;
            cs *= damp;
            a1 = 1.0f - ki * r;
        }
        if constexpr (S_) {
            o.x += g * cs;
            o.y -= g * sn;
        }
        if constexpr (D_) {
            const float f = -g * (rinv * rinv) * rn;
            o.z += f * (a1 * cs + kr * sn);
            o.w += f * (kr * cs - a1 * sn);
        }
    } else {
        if constexpr (S_) o.x += g;
        if constexpr (D_) o.z -= g * (rinv * rinv) * rn;
    }
}

// list 2: one pair by the general dispatch (classify_pair, the uniform loop
// over the pair's points); false when it is not regular.  Not inlined, so that
// its registers are not the column loop's.
template <int FAM, int OPS, bool CK>
__device__ __noinline__ bool reg2_general(const RegularArgs &a, int i, int j, float4 &o)
{
    const DevMesh &test = a.test, &trial = a.trial;
    const float4 ih = test.chi[i], il = test.clo[i], jl = trial.clo[j];
    int ls, ld;
    float dx, dy, dz;
    if (classify_pair(ih, il, trial.chi[j], jl, i, j, test.center, trial.center, trial.size, a.same_mesh, ls, ld, dx, dy,
                      dz) != KIND_REGULAR)
        return false;
    if (!(OPS & OP_SLP)) ls = ld;
    if (!(OPS & OP_DLP)) ld = ls;
    const int par = il.w != 0.0f ? 1 : 0, tnc = jl.w != 0.0f ? 4 : 3;
    const float k = a.k32, ki = a.k_im32;
    const int nps = level_npts(tnc, par, ls), npd = level_npts(tnc, par, ld);
    const int n_eval = ls == ld ? nps : nps + npd;
    const int64_t base = ((int64_t)j * 2 + par) * SLOTS;
    o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int q = 0; q < n_eval; ++q) {
        int slot;
        float ws, wd;
        if (ls == ld) { slot = level_slot0(ls) + q; ws = wd = 1.0f; }
        else if (q < nps) { slot = level_slot0(ls) + q; ws = 1.0f; wd = 0.0f; }
        else { slot = level_slot0(ld) + q - nps; ws = 0.0f; wd = 1.0f; }
        const float4 y = __ldg(trial.pts32 + 2 * (base + slot));
        const float4 n = __ldg(trial.pts32 + 2 * (base + slot) + 1);
        // r = (c_j - x) + (y - c_j): the hi/lo centre difference plus the point's
        // offset from the trial centre
        if constexpr (CK)
            eval_point_ck<float>(dx + y.x, dy + y.y, dz + y.z, y.w, n.x, n.y, n.z, k, ki, ws, wd, o.x, o.y, o.z, o.w);
        else
            eval_point<FAM, float>(dx + y.x, dy + y.y, dz + y.z, y.w, n.x, n.y, n.z, k, ws, wd, o.x, o.y, o.z, o.w);
    }
    return true;
}

// PLAIN: unit scale and no accumulation, so the stores carry no run-time checks
template <int FAM, int OPS, bool CK, bool PLAIN>
struct Reg2Op {
    static constexpr int GENERAL_LANES = 1;
    static constexpr bool DO_S = (OPS & OP_SLP) != 0, DO_D = (OPS & OP_DLP) != 0;
    // (d/D)^2 of the one-point rule of every operator, and of the next limit
    // below which list 1 ends (both: the DLP's 2.8, above the SLP's 1.8)
    static constexpr float Q0 = DO_D ? 249.64f : 82.81f, Q1 = DO_D ? 7.84f : 3.24f;

    const RegularArgs &a;
    const TwoRowShared &sh;
    int jb;
    float2 *out_s, *out_d;  // of the block's first column
    float k, ki;

    struct Extra {};
    __device__ __forceinline__ Extra extra(int, int) const { return {}; }
    __device__ __forceinline__ bool far(const Extra &, int, float q, float) const { return q > Q0 * (1.0f + 1e-4f); }
    __device__ __forceinline__ int list(float q) const
    {
        // the FP32 guard band of classify_pair: outside it the class is the FP64 class
        const float lo = q * (1.0f - 1e-5f), hi = q * (1.0f + 1e-5f);
        if (hi < 2.25f) return -1;  // certainly nearly singular
        if (DO_S && DO_D && lo >= 82.81f && hi < Q0) return 0;
        if (lo >= Q1 && hi < (DO_S ? 82.81f : Q0)) return 1;
        return 2;
    }
    __device__ __forceinline__ void store(float2 *p, float re, float im) const
    {
        if constexpr (PLAIN) *p = make_float2(re, im);
        else store_entry(p, re, im, a.alpha_re32, a.alpha_im32, a.unit_alpha != 0, a.accumulate);
    }
    __device__ __forceinline__ void put_one(int i, int c, const float4 &o) const
    {
        const int64_t off = (int64_t)c * a.ld + i;
        if (DO_S) store(out_s + off, o.x, o.y);
        if (DO_D) store(out_d + off, o.z, o.w);
    }
    using Val = Reg2Val;  // SLP and DLP of both rows
    template <int H>
    __device__ __forceinline__ void put(const Val &v, int c, int i) const
    {
        float4 x, y;
        f2_unpack(v.sr, x.x, y.x);
        f2_unpack(v.si, x.y, y.y);
        f2_unpack(v.dr, x.z, y.z);
        f2_unpack(v.di, x.w, y.w);
        put_one(i, c, H == 0 ? x : y);
    }
    __device__ __forceinline__ static Val zero() { return {f2_dup(0.0f), f2_dup(0.0f), f2_dup(0.0f), f2_dup(0.0f)}; }
    // the one-point rule of both rows
    __device__ __forceinline__ void far_eval(const Extra &, int c, f2 dx, f2 dy, f2 dz, f2 r2, Val &v) const
    {
        const TwoRowCol &t = sh.col[c];
        v = zero();
        f2 rn{};
        if constexpr (DO_D) rn = f2_fma(dz, t.nz, f2_fma(dy, t.ny, dx * t.nx));
        reg2_point<FAM, CK, DO_S, DO_D>(r2, t.w4, rn, k, ki, v);
    }
    template <int LIST>
    __device__ __forceinline__ void pair(int i, int c) const
    {
        if constexpr (LIST == 1 || (DO_S && DO_D)) {
            constexpr bool PS = LIST == 1 && DO_S;  // the SLP at the level-1 points
            const TwoRowCol &t = sh.col[c];
            const float3 d = t.diff(a.test, i);
            const float4 p = t.p0();
            float4 o = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (LIST == 0) reg2_point1<FAM, CK, true, false, true>(d.x, d.y, d.z, p.x, 0.0f, k, ki, o);
            const int par = a.test.clo[i].w != 0.0f ? 1 : 0;
            const bool quad = a.trial.has_quad && a.trial.nc[jb + c] == 4;
            const float4 *pts = a.trial.pts32 + 2 * (((int64_t)(jb + c) * 2 + par) * SLOTS + level_slot0(1));
            const int np = level_npts(quad ? 4 : 3, par, 1);
            for (int q = 0; q < np; ++q) {
                const float4 v = __ldg(pts + 2 * q);
                const float px = d.x + v.x, py = d.y + v.y, pz = d.z + v.z;
                float rn = 0.0f;
                if constexpr (DO_D) {
                    // a flat triangle's points share the centre's normal (but not the
                    // rounding of r.n, which the rule's sum averages)
                    float4 n = make_float4(p.y, p.z, p.w, 0.0f);
                    if (quad) n = __ldg(pts + 2 * q + 1);
                    rn = px * n.x + py * n.y + pz * n.z;
                }
                reg2_point1<FAM, CK, PS, DO_D, false>(px, py, pz, v.w, rn, k, ki, o);
            }
            put_one(i, c, o);
        }
    }
    __device__ __forceinline__ void general(int i, int c) const
    {
        float4 o;
        if (reg2_general<FAM, OPS, CK>(a, i, jb + c, o)) put_one(i, c, o);
    }
};

// 64 registers, eight blocks an SM, six beside one block of the concurrent singular
// kernel
template <int FAM, int OPS, bool CK, bool PLAIN>
__global__ void __launch_bounds__(TWO_ROW_THREADS, 32 / TWO_ROW_WARPS) k_regular2(const __grid_constant__ RegularArgs a, int cols_per_block)
{
    __shared__ TwoRowShared sh;
    const int jb = a.j0 + blockIdx.y * cols_per_block;
    const int ncols = min(cols_per_block, a.j1 - jb);
    const int ib = blockIdx.x * TWO_ROW_ROWS;
    if (threadIdx.x < ncols) sh.stage(threadIdx.x, a.trial, jb + threadIdx.x);
    __syncthreads();
    if (ib + 64 * (int)(threadIdx.x >> 5) >= a.test.n) return;
    const int64_t off = (int64_t)(jb - a.j0) * a.ld;
    const Reg2Op<FAM, OPS, CK, PLAIN> op{a, sh, jb, reinterpret_cast<float2 *>(a.out_s) + off,
                                         reinterpret_cast<float2 *>(a.out_d) + off, a.k32, a.k_im32};
    if (ib + TWO_ROW_ROWS <= a.test.n) two_row_columns<true>(op, sh, a.test, ib, ncols);
    else two_row_columns<false>(op, sh, a.test, ib, ncols);
}

template <int FAM, int OPS, bool CK, bool PLAIN>
static cudaError_t launch_regular2(const RegularArgs &a, cudaStream_t s)
{
    int dev = 0;
    cudaGetDevice(&dev);
    static bool carveout_set[64] = {};
    if (dev >= 0 && dev < 64 && !carveout_set[dev]) {
        const cudaError_t e = cudaFuncSetAttribute(k_regular2<FAM, OPS, CK, PLAIN>,
                                                   cudaFuncAttributePreferredSharedMemoryCarveout,
                                                   regular_carveout_percent());
        if (e != cudaSuccess) return e;
        carveout_set[dev] = true;
    }
    return two_row_launches(a.test.n, a.j0, a.j1, [&](int j0, int j1, dim3 grid, int cols) {
        RegularArgs b = a;
        b.j0 = j0;
        b.j1 = j1;
        b.out_s = reinterpret_cast<float2 *>(a.out_s) + (int64_t)(j0 - a.j0) * a.ld;
        b.out_d = reinterpret_cast<float2 *>(a.out_d) + (int64_t)(j0 - a.j0) * a.ld;
        k_regular2<FAM, OPS, CK, PLAIN><<<grid, TWO_ROW_THREADS, 0, s>>>(b, cols);
    });
}

template <int FAM, bool CK, bool PLAIN>
static cudaError_t launch_regular2_ops(const RegularArgs &a, cudaStream_t s)
{
    if (a.ops == OP_SLP) return launch_regular2<FAM, OP_SLP, CK, PLAIN>(a, s);
    if (a.ops == OP_DLP) return launch_regular2<FAM, OP_DLP, CK, PLAIN>(a, s);
    return launch_regular2<FAM, OP_SLP | OP_DLP, CK, PLAIN>(a, s);
}

template <bool PLAIN>
static cudaError_t launch_regular2_fam(const RegularArgs &a, cudaStream_t s)
{
    if (a.family != FAM_HELMHOLTZ) return launch_regular2_ops<FAM_LAPLACE, false, PLAIN>(a, s);
    if (a.k_im != 0.0) return launch_regular2_ops<FAM_HELMHOLTZ, true, PLAIN>(a, s);
    return launch_regular2_ops<FAM_HELMHOLTZ, false, PLAIN>(a, s);
}

// partial sums of the same row added in FP32 before one FP64 addition
constexpr int RHS_GROUP = 8;

template <typename R2>
__global__ void __launch_bounds__(256) k_rhs_reduce(const R2 *__restrict__ part, int n_cb, int n, int64_t items,
                                                    const int64_t *__restrict__ row_ptr, const int2 *__restrict__ row_ent,
                                                    const double2 *__restrict__ near_slp, const double2 *__restrict__ q,
                                                    int qn, double2 *__restrict__ b)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int f = blockIdx.y;
    if (i >= n) return;
    using R = decltype(R2::x);
    double re = 0.0, im = 0.0;
    const R2 *p = part + (int64_t)f * n_cb * n + i;
    for (int cb0 = 0; cb0 < n_cb; cb0 += RHS_GROUP) {
        R gr = 0, gi = 0;
        const int cb1 = min(n_cb, cb0 + RHS_GROUP);
        for (int cb = cb0; cb < cb1; ++cb) {
            const R2 v = p[(int64_t)cb * n];
            gr += v.x;
            gi += v.y;
        }
        re += (double)gr;
        im += (double)gi;
    }
    const double2 *qf = q + (int64_t)f * qn;
    const double2 *sf = near_slp + (int64_t)f * items;
    R nr = 0, ni = 0;
    for (int64_t t = row_ptr[i]; t < row_ptr[i + 1]; ++t) {
        const int2 e = row_ent[t];
        const double2 sv = sf[e.x], qv = qf[e.y];
        const R sr = R(sv.x), si = R(sv.y), qr = R(qv.x), qi = R(qv.y);
        nr += sr * qr - si * qi;
        ni += sr * qi + si * qr;
    }
    b[(int64_t)f * n + i] = make_double2(re + (double)nr, im + (double)ni);
}

template <typename R, typename Out, int FAM, bool BATCH>
static void launch_ops(const RegularArgs &a, dim3 grid, cudaStream_t s)
{
    if constexpr (BATCH) {
        if (a.rhs_part) {
            const size_t smem = sizeof(Cplx<R>) * rhs_fmax_of<R>(a) * (REG_COLS + REG_THREADS);
            k_regular<R, Out, FAM, OP_SLP | OP_DLP, true, true><<<grid, REG_THREADS, smem, s>>>(a);
            return;
        }
    }
    if constexpr (!BATCH && FAM == FAM_HELMHOLTZ) {
        if (a.k_im != 0.0) {
            if (a.ops == OP_SLP) k_regular<R, Out, FAM, OP_SLP, false, false, false, true><<<grid, REG_THREADS, 0, s>>>(a);
            else if (a.ops == OP_DLP)
                k_regular<R, Out, FAM, OP_DLP, false, false, false, true><<<grid, REG_THREADS, 0, s>>>(a);
            else k_regular<R, Out, FAM, OP_SLP | OP_DLP, false, false, false, true><<<grid, REG_THREADS, 0, s>>>(a);
            return;
        }
    }
    if constexpr (!BATCH && sizeof(R) == 4) {
        if (a.unit_alpha && !a.accumulate) {
            if (a.ops == OP_SLP) k_regular<R, Out, FAM, OP_SLP, false, false, true><<<grid, REG_THREADS, 0, s>>>(a);
            else if (a.ops == OP_DLP) k_regular<R, Out, FAM, OP_DLP, false, false, true><<<grid, REG_THREADS, 0, s>>>(a);
            else k_regular<R, Out, FAM, OP_SLP | OP_DLP, false, false, true><<<grid, REG_THREADS, 0, s>>>(a);
            return;
        }
    }
    if (a.ops == OP_SLP) k_regular<R, Out, FAM, OP_SLP, BATCH><<<grid, REG_THREADS, 0, s>>>(a);
    else if (a.ops == OP_DLP) k_regular<R, Out, FAM, OP_DLP, BATCH><<<grid, REG_THREADS, 0, s>>>(a);
    else k_regular<R, Out, FAM, OP_SLP | OP_DLP, BATCH><<<grid, REG_THREADS, 0, s>>>(a);
}

template <typename R, typename Out>
static void launch_fam(const RegularArgs &a, dim3 grid, cudaStream_t s)
{
    const bool batch = a.nk > 1 || a.force_batch;
    constexpr bool SINGLE = sizeof(R) == 8 || sizeof(Out) == 16;  // FP32 into complex64: k_regular2
    if (a.family == FAM_HELMHOLTZ) {
        if (batch) launch_ops<R, Out, FAM_HELMHOLTZ, true>(a, grid, s);
        else if constexpr (SINGLE) launch_ops<R, Out, FAM_HELMHOLTZ, false>(a, grid, s);
    } else {
        if (batch) launch_ops<R, Out, FAM_LAPLACE, true>(a, grid, s);
        else if constexpr (SINGLE) launch_ops<R, Out, FAM_LAPLACE, false>(a, grid, s);
    }
}

cudaError_t launch_assemble_regular(const RegularArgs &a, cudaStream_t s)
{
    int ncols = a.j1 - a.j0;
    if (a.test.n == 0 || ncols <= 0) return cudaSuccess;
    if (a.precision == 0 && a.dtype == 0 && a.nk <= 1 && !a.force_batch)
        return a.unit_alpha && !a.accumulate ? launch_regular2_fam<true>(a, s) : launch_regular2_fam<false>(a, s);
    dim3 grid((a.test.n + REG_THREADS - 1) / REG_THREADS, (ncols + REG_COLS - 1) / REG_COLS);
    if (a.nk > 1 || a.force_batch) {
        // small meshes: split the wave numbers over gridDim.z (at least one tile of
        // FREQ_TILE each) until the grid holds about four blocks per SM
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const int64_t xy = (int64_t)grid.x * grid.y;
        const int64_t want = (4 * (int64_t)sms + xy - 1) / xy;
        const int most = (a.nk + FREQ_TILE - 1) / FREQ_TILE;
        if (a.accumulate || !a.unit_alpha) return cudaErrorInvalidValue;  // batches store plain entries
        grid.z = (unsigned)std::max<int64_t>(1, std::min<int64_t>(want, most));
        // right-hand-side mode: at most rhs_f_max wave numbers per block
        if (a.rhs_part) {
            const int fmax = a.precision == 0 ? rhs_fmax_of<float>(a) : rhs_fmax_of<double>(a);
            grid.z = std::max<unsigned>(grid.z, (unsigned)((a.nk + fmax - 1) / fmax));
        }
    } else {
        grid.y = column_blocks(grid.x, ncols, REG_COLS);
    }
    if (a.precision == 0) {
        if (a.dtype == 0) launch_fam<float, float2>(a, grid, s);
        else launch_fam<float, double2>(a, grid, s);
    } else {
        if (a.dtype == 0) launch_fam<double, float2>(a, grid, s);
        else launch_fam<double, double2>(a, grid, s);
    }
    return cudaGetLastError();
}

size_t rhs_part_bytes(const RegularArgs &a)
{
    const int64_t n_cb = (a.j1 - a.j0 + REG_COLS - 1) / REG_COLS;
    return (a.precision == 0 ? sizeof(float2) : sizeof(double2)) * (size_t)a.nk * n_cb * a.test.n;
}

cudaError_t launch_rhs_reduce(const RegularArgs &a, const NearList &near, double2 *b, cudaStream_t s)
{
    const int n = a.test.n;
    if (n == 0 || a.nk == 0) return cudaSuccess;
    const int n_cb = (a.j1 - a.j0 + REG_COLS - 1) / REG_COLS;
    const int64_t items = near.nnz + (a.same_mesh ? a.trial.n : 0);
    dim3 grid((n + 255) / 256, a.nk);
    if (a.precision == 0)
        k_rhs_reduce<float2><<<grid, 256, 0, s>>>((const float2 *)a.rhs_part, n_cb, n, items, near.row_ptr,
                                                  near.row_ent, a.near_slp, a.rhs_q, a.trial.n, b);
    else
        k_rhs_reduce<double2><<<grid, 256, 0, s>>>((const double2 *)a.rhs_part, n_cb, n, items, near.row_ptr,
                                                   near.row_ent, a.near_slp, a.rhs_q, a.trial.n, b);
    return cudaGetLastError();
}

}  // namespace nihu
