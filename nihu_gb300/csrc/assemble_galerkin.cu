// Galerkin formalism of the SLP and DLP operators on constant elements:
//   A(i, j) = int_{E_i} int_{E_j} K(x, y) dS_y dS_x
// (nihu/core/double_integral.hpp:143-384, the "general" formalism).
//
// Dispatch, as the reference: on one mesh an element pair that shares the
// element (face), two nodes (edge) or one node (corner) takes the singular
// Galerkin rule of its match type (nihu/core/element_match.hpp:60-90,
// nihu/core/singular_accelerator.hpp:220-310); every other pair takes the
// product of the regular rule of degree C + interval(d/D) on both elements
// (complexity_estimator.hpp:69-75, the dual accelerator of
// double_integral.hpp:300-312).  The singular rules are the 4D Gauss products
// (4 points per direction: the kernels' singular quadrature order 7) split
// into Duffy-type subdomains in coordinate differences
// (nihu/core/singular_galerkin_quadrature.hpp:200-420): face 3 subdomains
// (symmetric, 1536 points), edge 6 (1536), corner 1 (symmetric, 512).
//
// Work layout: k_galerkin_regular (FP32 default / FP64) owns the pairs at
// d/D >= 1.5 exactly as the collocation kernel does, with the test element's
// points in the same rule as the trial element's (a far pair is the
// collocation entry times the test element's area); k_galerkin_near (one warp
// per pair, lanes over the rule's points) owns the self pairs, the nearly
// singular list (d/D < 1.5: matched pairs, and unmatched ones with the
// degree-6/8 product rules) and the rare pairs beyond 1.5 D that still share
// a node (collected by the regular kernel).  The near kernel follows the
// regular quadrature's precision: FP64, or FP32 with r_vec formed from
// vectors relative to the common node (matched pairs) or to the element
// centres (unmatched pairs), which keeps FP32 relative accuracy as r -> 0.
#include <algorithm>
#include <initializer_list>
#include <mutex>
#include <vector>

#include "classify.cuh"
#include "kernels.h"
#include "singular_schemes.cuh"
#include "two_row.cuh"

namespace nihu {

constexpr int GAL_THREADS = 256;
constexpr int GAL_COLS = 32;
constexpr int GAL_WARPS = 4;
constexpr int GAL_GAUSS = 4;  // points per direction of the singular rules
constexpr int GAL_PER_DIM4 = GAL_GAUSS * GAL_GAUSS * GAL_GAUSS * GAL_GAUSS;
// points of the corner (0), edge (1) and face (2) rules
__host__ __device__ constexpr int gal_npts(int match) { return (match == 0 ? 2 : 6) * GAL_PER_DIM4; }
constexpr int GAL_TOTAL = gal_npts(0) + gal_npts(1) + gal_npts(2);

// the singular rules, (test xi, eta, trial xi, eta, w) per point: corner
// points first, then edge, then face; and in FP32 (test xi, eta, trial xi,
// eta, w, trial xi - test xi, trial eta - test eta, 0), the differences formed
// in FP64
__device__ double g_gal_rule[GAL_TOTAL * 5];

// the quad-quad rules (corner 1280, edge 1536, face 2048 points), the same layout
__host__ __device__ constexpr int galq_npts(int match) { return match == 0 ? 1280 : (match == 1 ? 1536 : 2048); }
__host__ __device__ constexpr int galq_offset(int match)
{
    return match == 0 ? 0 : (match == 1 ? galq_npts(0) : galq_npts(0) + galq_npts(1));
}
constexpr int GALQ_TOTAL = galq_npts(0) + galq_npts(1) + galq_npts(2);
__device__ double g_galq_rule[GALQ_TOTAL * 5];
__device__ __align__(16) float g_gal_rule32[GAL_TOTAL * 8];

__host__ __device__ constexpr int gal_offset(int match)
{
    return match == 0 ? 0 : (match == 1 ? gal_npts(0) : gal_npts(0) + gal_npts(1));
}

// one point of the 4D cube mapped into a subdomain of the match type: test
// point (a1, a2) and trial point (a1 + b1, a2 + b2) on 0 <= x2 <= x1 <= 1,
// weight times the subdomain Jacobian
static void gal_subdomain(int match, int sub, const double u[4], double &w, double out[4])
{
    double a1, a2, b1, b2;
    if (match == 2) {
        double jac;
        if (sub == 0) {
            b1 = u[0];
            b2 = u[0] * u[1];
            a1 = (1.0 - b1) * u[2];
            a2 = a1 * u[3];
            jac = (1.0 - b1) * a1;
        } else if (sub == 1) {
            b1 = u[0] * u[1];
            b2 = u[0] * (u[1] - 1.0);
            a1 = (1.0 - b1 + b2) * u[2] - b2;
            a2 = (a1 + b2) * u[3] - b2;
            jac = (1.0 - b1 + b2) * (a1 + b2);
        } else {
            b1 = u[0] * u[1];
            b2 = u[0];
            a1 = (1.0 - b2) * u[2] + b2 - b1;
            a2 = (a1 - b2 + b1) * u[3];
            jac = (1.0 - b2) * (a1 - b2 + b1);
        }
        w *= jac * u[0];
    } else if (match == 1) {
        const double p = u[0], q = u[1], r = u[2], s = u[3];
        switch (sub) {
        case 0: b1 = -p * q; b2 = -p * q * r; a1 = (1.0 - p) * s + p; a2 = p * (1.0 - q + q * r); break;
        case 1: b1 = p * q; b2 = p * q * r; a1 = (1.0 - p) * s + p * (1.0 - q); a2 = p * (1.0 - q); break;
        case 2: b1 = -p * q * r; b2 = p * q * (1.0 - r); a1 = (1.0 - p) * s + p; a2 = p * (1.0 - q); break;
        case 3: b1 = p * q * r; b2 = p * q * (r - 1.0); a1 = (1.0 - p) * s + p * (1.0 - q * r); a2 = p * (1.0 - q * r); break;
        case 4: b1 = -p * q * r; b2 = -p * q; a1 = (1.0 - p) * s + p; a2 = p; break;
        default: b1 = p * q * r; b2 = p * q; a1 = (1.0 - p) * s + p * (1.0 - q * r); a2 = p * (1.0 - q); break;
        }
        w *= q * p * p * (1.0 - p);
    } else {
        a1 = u[0];
        a2 = a1 * u[1];
        const double e1 = a1 * u[2], e2 = e1 * u[3];
        w *= u[2] * u[0] * u[0] * u[0];
        b1 = e1 - a1;
        b2 = e2 - a2;
    }
    out[0] = a1 - a2;
    out[1] = a2;
    out[2] = (a1 + b1) - (a2 + b2);
    out[3] = a2 + b2;
}

// every Dunavant rule in FP32, (xi, eta, w) per point at the offsets of quad_rules.h
struct TriF32 {
    float v[NIHU_TRI_DATA_LEN];
    constexpr TriF32() : v()
    {
        constexpr double d[NIHU_TRI_DATA_LEN] = NIHU_TRI_DATA;
        for (int q = 0; q < NIHU_TRI_DATA_LEN; ++q) v[q] = (float)d[q];
    }
};
__device__ constexpr TriF32 TRI_F32{};

// host generation of the three rules (the Gauss nodes come from the device
// tables' source, quad_rules.h)
static std::vector<double> gal_rules()
{
    static const double gdata[NIHU_GAUSS_DATA_LEN] = NIHU_GAUSS_DATA;
    static const int goff[NIHU_GAUSS_MAX_N] = NIHU_GAUSS_OFFSETS;
    double x[GAL_GAUSS], wt[GAL_GAUSS];
    for (int i = 0; i < GAL_GAUSS; ++i) {
        x[i] = (1.0 + gdata[2 * (goff[GAL_GAUSS - 1] + i)]) / 2.0;
        wt[i] = gdata[2 * (goff[GAL_GAUSS - 1] + i) + 1] / 2.0;
    }
    std::vector<double> out((size_t)GAL_TOTAL * 5);
    for (int match = 0; match < 3; ++match) {
        const int subs = match == 2 ? 3 : (match == 1 ? 6 : 1);
        const bool sym = match != 1;
        double *d = out.data() + 5 * (size_t)gal_offset(match);
        for (int i1 = 0; i1 < GAL_GAUSS; ++i1)
            for (int i2 = 0; i2 < GAL_GAUSS; ++i2)
                for (int i3 = 0; i3 < GAL_GAUSS; ++i3)
                    for (int i4 = 0; i4 < GAL_GAUSS; ++i4)
                        for (int sub = 0; sub < subs; ++sub) {
                            const double u[4] = {x[i1], x[i2], x[i3], x[i4]};
                            double w = wt[i1] * wt[i2] * wt[i3] * wt[i4], o[4];
                            gal_subdomain(match, sub, u, w, o);
                            d[0] = o[0]; d[1] = o[1]; d[2] = o[2]; d[3] = o[3]; d[4] = w;
                            d += 5;
                            if (sym) {
                                d[0] = o[2]; d[1] = o[3]; d[2] = o[0]; d[3] = o[1]; d[4] = w;
                                d += 5;
                            }
                        }
    }
    return out;
}

// Duffy quads of the coordinate difference mu for the quad-quad rules
// (nihu/library/lib_singular_galerkin_quadrature.cpp)
static const double QF[4][4][2] = {{{0, 0}, {0, 0}, {2, -2}, {2, 0}}, {{0, 0}, {0, 0}, {2, 0}, {2, 2}},
                                   {{0, 0}, {0, 0}, {2, 2}, {0, 2}}, {{0, 0}, {0, 0}, {0, 2}, {-2, 2}}};
static const double QE[6][4][2] = {{{0, 0}, {0, 0}, {-2, 0}, {-2, -2}}, {{0, 0}, {0, 0}, {-2, -2}, {0, -2}},
                                   {{0, 0}, {0, 0}, {0, -2}, {2, -2}},  {{0, 0}, {0, 0}, {2, -2}, {2, 0}},
                                   {{-2, -2}, {-2, -4}, {0, -4}, {0, -2}}, {{0, -2}, {0, -4}, {2, -4}, {2, -2}}};
static const double QC[5][4][2] = {{{0, 0}, {0, 0}, {-2, 0}, {-2, -2}}, {{0, 0}, {0, 0}, {-2, -2}, {0, -2}},
                                   {{-4, 0}, {-4, -2}, {-2, -2}, {-2, 0}}, {{-4, -2}, {-4, -4}, {-2, -4}, {-2, -2}},
                                   {{-2, -2}, {-2, -4}, {0, -4}, {0, -2}}};

// bilinear map of (u, v) in [-1,1]^2 onto the quad with corners C, signed Jacobian
static void quad_corner_map(const double C[4][2], double u, double v, double &x, double &y, double &det)
{
    const double N[4] = {(1 - u) * (1 - v) / 4, (1 + u) * (1 - v) / 4, (1 + u) * (1 + v) / 4, (1 - u) * (1 + v) / 4};
    const double du[4] = {-(1 - v) / 4, (1 - v) / 4, (1 + v) / 4, -(1 + v) / 4};
    const double dv[4] = {-(1 - u) / 4, -(1 + u) / 4, (1 + u) / 4, (1 - u) / 4};
    double j00 = 0, j01 = 0, j10 = 0, j11 = 0;
    x = y = 0;
    for (int c = 0; c < 4; ++c) {
        x += N[c] * C[c][0];
        y += N[c] * C[c][1];
        j00 += du[c] * C[c][0];
        j01 += du[c] * C[c][1];
        j10 += dv[c] * C[c][0];
        j11 += dv[c] * C[c][1];
    }
    det = j00 * j11 - j01 * j10;
}

// the trial point's reflection that sets the two squares side by side:
// none (face), (eta_0, -2 - eta_1) (edge), -2 - eta (corner)
static void quad_reflect(int match, double e0, double e1, double &o0, double &o1)
{
    o0 = match == 0 ? -2.0 - e0 : e0;
    o1 = match == 2 ? e1 : -2.0 - e1;
}

static std::vector<double> galq_rules()
{
    static const double gdata[NIHU_GAUSS_DATA_LEN] = NIHU_GAUSS_DATA;
    static const int goff[NIHU_GAUSS_MAX_N] = NIHU_GAUSS_OFFSETS;
    const double *g = gdata + 2 * goff[GAL_GAUSS - 1];
    std::vector<double> out((size_t)GALQ_TOTAL * 5);
    for (int match = 0; match < 3; ++match) {
        const int subs = match == 2 ? 4 : (match == 1 ? 6 : 5);
        const double (*tab)[4][2] = match == 2 ? QF : (match == 1 ? QE : QC);
        double lo[2], hi[2];
        quad_reflect(match, -1.0, -1.0, lo[0], lo[1]);
        quad_reflect(match, 1.0, 1.0, hi[0], hi[1]);
        for (int c = 0; c < 2; ++c)
            if (lo[c] > hi[c]) std::swap(lo[c], hi[c]);
        double *d = out.data() + 5 * (size_t)galq_offset(match);
        for (int sd = 0; sd < subs; ++sd)
            for (int a = 0; a < GAL_GAUSS; ++a)
                for (int b = 0; b < GAL_GAUSS; ++b) {
                    double mu0, mu1, det;
                    quad_corner_map(tab[sd], g[2 * a], g[2 * b], mu0, mu1, det);
                    const double wo = g[2 * a + 1] * g[2 * b + 1] * det;
                    auto clip = [](double v) { return std::min(1.0, std::max(-1.0, v)); };
                    const double x0 = clip(lo[0] - mu0), x1 = clip(hi[0] - mu0);
                    const double y0 = clip(lo[1] - mu1), y1 = clip(hi[1] - mu1);
                    const double R[4][2] = {{x0, y0}, {x1, y0}, {x1, y1}, {x0, y1}};
                    for (int c = 0; c < GAL_GAUSS; ++c)
                        for (int e = 0; e < GAL_GAUSS; ++e) {
                            double xi0, xi1, di;
                            quad_corner_map(R, g[2 * c], g[2 * e], xi0, xi1, di);
                            const double w = wo * g[2 * c + 1] * g[2 * e + 1] * di;
                            double et0, et1;
                            quad_reflect(match, mu0 + xi0, mu1 + xi1, et0, et1);
                            d[0] = xi0; d[1] = xi1; d[2] = et0; d[3] = et1; d[4] = w;
                            d += 5;
                            if (match == 2) {
                                d[0] = et0; d[1] = et1; d[2] = xi0; d[3] = xi1; d[4] = w;
                                d += 5;
                            }
                        }
                }
    }
    return out;
}

cudaError_t prepare_galerkin(cudaStream_t s)
{
    static std::mutex mu;
    static std::vector<int> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lock(mu);
    if ((int)done.size() > dev && done[dev]) return cudaSuccess;
    static const std::vector<double> rules = gal_rules();
    static const std::vector<float> rules32 = [] {
        std::vector<float> f((size_t)GAL_TOTAL * 8, 0.0f);
        for (size_t p = 0; p < (size_t)GAL_TOTAL; ++p) {
            const double *q = rules.data() + 5 * p;
            for (int c = 0; c < 5; ++c) f[8 * p + c] = (float)q[c];
            f[8 * p + 5] = (float)(q[2] - q[0]);
            f[8 * p + 6] = (float)(q[3] - q[1]);
        }
        return f;
    }();
    e = cudaMemcpyToSymbolAsync(g_gal_rule, rules.data(), rules.size() * sizeof(double), 0, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(g_gal_rule32, rules32.data(), rules32.size() * sizeof(float), 0,
                                    cudaMemcpyHostToDevice, s);
    static const std::vector<double> qrules = galq_rules();
    if (e == cudaSuccess)
        e = cudaMemcpyToSymbolAsync(g_galq_rule, qrules.data(), qrules.size() * sizeof(double), 0,
                                    cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return e;
    if ((int)done.size() <= dev) done.resize(dev + 1, 0);
    done[dev] = 1;
    return cudaSuccess;
}

// number of common corner nodes of two elements and, for triangles, the first
// common node of each in cyclic order (nihu/core/element.hpp:376-413)
__device__ __forceinline__ int common_nodes(int4 a, int na, int4 b, int nb, int &ind1, int &ind2)
{
    const int A[4] = {a.x, a.y, a.z, a.w}, B[4] = {b.x, b.y, b.z, b.w};
    int num = 0, s1 = 0, s2 = 0;
    for (int i = 0; i < na; ++i)
        for (int j = 0; j < nb; ++j) {
            if (A[i] != B[j]) continue;
            if (num == 0) {
                s1 = i;
                s2 = j;
            } else {
                if (i < s1 || (i == na - 1 && s1 == 0 && num == 1)) s1 = i;
                if (j < s2 || (j == nb - 1 && s2 == 0 && num == 1)) s2 = j;
            }
            ++num;
        }
    ind1 = s1;
    ind2 = s2;
    return num;
}

// PLAIN: unit scale and no accumulation (FP32): stores without run-time checks;
// CK: a complex (lossy) wave number (eval_point_ck)
template <typename R, typename Out, int FAM, int OPS, bool PLAIN = false, bool CK = false>
__global__ void __launch_bounds__(GAL_THREADS) k_galerkin_regular(GalArgs a)
{
    __shared__ float4 s_hi[GAL_COLS], s_lo[GAL_COLS], s_p0[GAL_COLS];
    __shared__ int4 s_nid[GAL_COLS];
    __shared__ int s_nc[GAL_COLS];
    constexpr bool DO_S = (OPS & OP_SLP) != 0;
    constexpr bool DO_D = (OPS & OP_DLP) != 0;
    const DevMesh &test = a.test;
    const DevMesh &trial = a.trial;
    const int i = blockIdx.x * GAL_THREADS + threadIdx.x;
    const int cpb = (a.j1 - a.j0 + gridDim.y - 1) / gridDim.y;
    const int jb = a.j0 + blockIdx.y * cpb;
    const int ncols = min(cpb, a.j1 - jb);
    if (threadIdx.x < ncols) {
        const int j = jb + threadIdx.x;
        s_hi[threadIdx.x] = trial.chi[j];
        s_lo[threadIdx.x] = trial.clo[j];
        s_p0[threadIdx.x] = trial.p0[j];
        s_nid[threadIdx.x] = trial.nid[j];
        s_nc[threadIdx.x] = trial.nc[j];
    }
    __syncthreads();
    if ((i & ~31) >= test.n) return;
    const bool row_ok = i < test.n;
    const int ii = row_ok ? i : test.n - 1;
    const float4 ih = test.chi[ii], il = test.clo[ii];
    const int4 inid = test.nid[ii];
    const int inc = test.nc[ii];
    const float area_i = test.p0[ii].x;  // w J of the one-point rule: the element's area
    R k, ki, are, aim, x0, x1, x2;
    if constexpr (sizeof(R) == 4) {
        k = a.k32;
        ki = a.k_im32;
        are = a.alpha_re32;
        aim = a.alpha_im32;
        x0 = ih.x + il.x;
        x1 = ih.y + il.y;
        x2 = ih.z + il.z;
    } else {
        k = a.k;
        ki = a.k_im;
        are = a.alpha_re;
        aim = a.alpha_im;
        x0 = test.center[3 * (int64_t)ii];
        x1 = test.center[3 * (int64_t)ii + 1];
        x2 = test.center[3 * (int64_t)ii + 2];
    }
    Out *out_s = reinterpret_cast<Out *>(a.out_s);
    Out *out_d = reinterpret_cast<Out *>(a.out_d);
    // this thread's entries of the current column, one column (ld entries) further per step
    const int64_t ldo = a.ld;
    Out *ps = DO_S ? out_s + (int64_t)(jb - a.j0) * ldo + i : nullptr;
    Out *pd = DO_D ? out_d + (int64_t)(jb - a.j0) * ldo + i : nullptr;
    for (int c = 0; c < ncols; ++c, ps += DO_S ? ldo : 0, pd += DO_D ? ldo : 0) {
        const int j = jb + c;
        int ind1, ind2;
        // elements can share a node only when their centres are closer than
        // the sum of their centre-to-corner distances (< 2 D each): compare
        // node ids only then
        const float4 hj = s_hi[c];
        const float ex0 = hj.x - ih.x, ex1 = hj.y - ih.y, ex2 = hj.z - ih.z;
        const float reach = 2.0f * (rsqrtf(ih.w) + rsqrtf(hj.w));
        const bool may_share = a.same_mesh && ex0 * ex0 + ex1 * ex1 + ex2 * ex2 <= 1.01f * reach * reach;
        const int shared = may_share ? common_nodes(inid, inc, s_nid[c], s_nc[c], ind1, ind2) : 0;
        R sr = 0, si = 0, dr = 0, di = 0;
        bool done = false;
        if constexpr (sizeof(R) == 4) {
            // far field: both one-point rules, the centroid kernel times both areas
            const float4 h = s_hi[c], l = s_lo[c];  // hi/lo centre difference (as k_regular)
            const float fx = (h.x - ih.x) + (l.x - il.x), fy = (h.y - ih.y) + (l.y - il.y),
                        fz = (h.z - ih.z) + (l.z - il.z);
            const float q = (fx * fx + fy * fy + fz * fz) * h.w;
            if (__all_sync(0xffffffffu, q > 249.64f * (1.0f + 1e-4f) && shared == 0)) {
                const float4 p = s_p0[c];
                if constexpr (CK)
                    eval_point_ck<float>(fx, fy, fz, p.x, p.y, p.z, p.w, k, ki, DO_S ? area_i : 0.0f,
                                         DO_D ? area_i : 0.0f, sr, si, dr, di);
                else
                    eval_point<FAM, float>(fx, fy, fz, p.x, p.y, p.z, p.w, k, DO_S ? area_i : 0.0f,
                                           DO_D ? area_i : 0.0f, sr, si, dr, di);
                done = true;
            }
        }
        if (!done) {
            int ls, ld;
            float dx, dy, dz;
            const int kind = classify_pair(ih, il, s_hi[c], s_lo[c], ii, j, test.center, trial.center, trial.size,
                                           a.same_mesh, ls, ld, dx, dy, dz);
            if (kind != KIND_REGULAR || !row_ok) continue;  // self and d/D < 1.5: the FP64 kernel
            if (shared > 0) {
                // a node shared beyond 1.5 D (strongly graded mesh): singular rule
                const unsigned slot = atomicAdd(a.n_extra, 1u);
                if (slot < (unsigned)a.extra_cap) a.extra[slot] = make_int2(i, j);
                else atomicCAS(a.err, 0, -1);
                continue;
            }
            if (!DO_S) ls = ld;
            if (!DO_D) ld = ls;
            // the rule of degree C + 2 l on both elements: C = max complexity
            const int cmax = (il.w != 0.0f || s_lo[c].w != 0.0f) ? 1 : 0;
            const int64_t bi = ((int64_t)ii * 2 + cmax) * SLOTS, bj = ((int64_t)j * 2 + cmax) * SLOTS;
            for (int pass = 0; pass < 2; ++pass) {
                const int L = pass == 0 ? ls : ld;
                if (pass == 1 && ld == ls) break;
                const R ws = (DO_S && ls == L) ? R(1) : R(0), wd = (DO_D && ld == L) ? R(1) : R(0);
                const int npi = level_npts(inc, cmax, L), npj = level_npts(s_nc[c], cmax, L);
                for (int p = 0; p < npi; ++p) {
                    const int sp = level_slot0(L) + p;
                    R xp0, xp1, xp2, wp;
                    if constexpr (sizeof(R) == 4) {
                        const float4 y = __ldg(test.pts32 + 2 * (bi + sp));
                        xp0 = y.x;
                        xp1 = y.y;
                        xp2 = y.z;
                        wp = y.w;
                    } else {
                        const double *y = test.pts64 + 8 * (bi + sp);
                        xp0 = y[0];
                        xp1 = y[1];
                        xp2 = y[2];
                        wp = y[3];
                    }
                    for (int q = 0; q < npj; ++q) {
                        const int sq = level_slot0(L) + q;
                        if constexpr (sizeof(R) == 4) {
                            const float4 y = __ldg(trial.pts32 + 2 * (bj + sq));
                            const float4 n = __ldg(trial.pts32 + 2 * (bj + sq) + 1);
                            // r = (c_j - c_i) + (y - c_j) - (x_p - c_i): the hi/lo centre
                            // difference and the points' offsets from their centres
                            if constexpr (CK)
                                eval_point_ck<float>(dx + (y.x - xp0), dy + (y.y - xp1), dz + (y.z - xp2), y.w, n.x,
                                                     n.y, n.z, k, ki, ws * wp, wd * wp, sr, si, dr, di);
                            else
                                eval_point<FAM, float>(dx + (y.x - xp0), dy + (y.y - xp1), dz + (y.z - xp2), y.w, n.x,
                                                       n.y, n.z, k, ws * wp, wd * wp, sr, si, dr, di);
                        } else {
                            const double *y = trial.pts64 + 8 * (bj + sq);
                            if constexpr (CK)
                                eval_point_ck<double>(y[0] - xp0, y[1] - xp1, y[2] - xp2, y[3], y[4], y[5], y[6], k, ki,
                                                      ws * wp, wd * wp, sr, si, dr, di);
                            else
                                eval_point<FAM, double>(y[0] - xp0, y[1] - xp1, y[2] - xp2, y[3], y[4], y[5], y[6], k,
                                                        ws * wp, wd * wp, sr, si, dr, di);
                        }
                    }
                }
            }
        }
        if (!row_ok) continue;
        auto store = [&](Out *p, R re, R im) {
            Out o;
            if constexpr (PLAIN) {
                o.x = re;
                o.y = im;
            } else {
                const R vr = are * re - aim * im, vi = are * im + aim * re;
                if (a.accumulate) {
                    o = *p;
                    o.x += vr;
                    o.y += vi;
                } else {
                    o.x = vr;
                    o.y = vi;
                }
            }
            *p = o;
        };
        if (DO_S) store(ps, sr, si);
        if (DO_D) store(pd, dr, di);
    }
}

// ------------------------------------------------- two rows per thread
// The FP32 kernel into complex64 matrices of a real wave number with unit
// scale and no accumulation, through the column loop of two_row.cuh: far pairs
// (both one-point rules) in the loop, the others listed by rule,
//   0  9.1 <= d/D < 15.8: the centroids for the SLP, the level-1 product for the DLP
//   1  2.8 <= d/D < 9.1: the level-1 product (9 points on triangles) for both
//   2  all others: k_galerkin_regular's dispatch
// A far pair also has to be out of its elements' reach (2 (D_i + D_j), within
// which they may share a node), tested against the largest of the warp's rows;
// lists 0 and 1 compare node ids within it.
//
// Bound by latency at 20 warps an SM (96 registers; 45% of the issue slots).  The
// one-row kernel ran every lane of a warp through the largest product of its 32
// pairs.  5120 triangles, k = 5, both operators: with the near pairs' kernel 1269
// us before, 903 us now; alone 635 us (spill-free only up to 20 warps per SM, which
// measured 30 us less than 28).
struct Gal2Val {
    f2 sr, si, dr, di;
};
// one point of two pairs; w4: the trial point's weight and Jacobian over 4 pi, wx: the
// test point's (a rounding of their product would be the same for all pairs of two shapes)
template <int FAM, bool S_, bool D_>
__device__ __forceinline__ void gal2_point(f2 rx, f2 ry, f2 rz, f2 w4, f2 wx, f2 nx, f2 ny, f2 nz, float k, Gal2Val &v)
{
    const f2 r2 = f2_fma(rz, rz, f2_fma(rx, rx, ry * ry));
    const f2 rinv = f2_rsqrt(r2);
    const f2 g = w4 * rinv * wx;
    f2 f{};  // g (r.n) / r^2: minus the DLP's factor
    if constexpr (D_) f = (g * (rinv * rinv)) * f2_fma(rz, nz, f2_fma(ry, ny, rx * nx));
    if constexpr (FAM == FAM_HELMHOLTZ) {
        const f2 r = r2 * rinv, kr = r * f2_dup(k), nkr = r * f2_dup(-k);
        f2 sn, cs;
        f2_sincos_reduced(nkr, sn, cs);  // e^{-ikr} = cs + i sn
        if constexpr (S_) {
            v.sr = f2_fma(g, cs, v.sr);
            v.si = f2_fma(g, sn, v.si);
        }
        if constexpr (D_) {
            const f2 nf = f * f2_dup(-1.0f);
            v.dr = f2_fma(nf, f2_fma(nkr, sn, cs), v.dr);
            v.di = f2_fma(nf, f2_fma(kr, cs, sn), v.di);
        }
    } else {
        if constexpr (S_) v.sr = v.sr + g;
        if constexpr (D_) v.dr = f2_fma(f, f2_dup(-1.0f), v.dr);
    }
}

constexpr int GAL2_LANES = 4;  // lanes per pair of list 2, whose products have up to 45 points
struct Gal2Sums {
    float sr = 0.0f, si = 0.0f, dr = 0.0f, di = 0.0f;
};

// one point of one pair, w the trial point's weight, wx the test point's; W4: w is over
// 4 pi already (else points of equal weights round that one by one, which their sum
// averages)
template <int FAM, bool S_, bool D_, bool W4>
__device__ __forceinline__ void gal2_point1(float rx, float ry, float rz, float w, float wx, float nx, float ny, float nz, float k,
                                            Gal2Sums &o)
{
    constexpr float INV4PI = 0.0795774715459476679f;
    const float r2 = rx * rx + ry * ry + rz * rz;
    const float rinv = rsqrtf(r2);
    const float g = (W4 ? w * rinv : w * rinv * INV4PI) * wx;
    float sn = 0.0f, cs = 1.0f, kr = 0.0f;
    if constexpr (FAM == FAM_HELMHOLTZ) {
        kr = k * (r2 * rinv);
        sincos_reduced(kr, sn, cs);
    }
    if constexpr (S_) {
        o.sr += g * cs;
        o.si -= g * sn;
    }
    if constexpr (D_) {
        const float f = -g * (rinv * rinv) * (rx * nx + ry * ny + rz * nz);
        o.dr += f * (cs + kr * sn);
        o.di += f * (kr * cs - sn);
    }
}

// k_galerkin_regular's general dispatch of one pair by GAL2_LANES lanes (each
// takes every GAL2_LANES-th test point; every lane gets the sums); false when
// it is left to the near kernel or listed as an extra pair
template <int FAM, int OPS>
__device__ __noinline__ bool gal2_general(const GalArgs &a, int i, int j, Gal2Sums &o)
{
    constexpr bool DO_S = (OPS & OP_SLP) != 0, DO_D = (OPS & OP_DLP) != 0;
    const Lanes<GAL2_LANES> lanes;
    const DevMesh &test = a.test, &trial = a.trial;
    const float4 ih = test.chi[i], il = test.clo[i], jh = trial.chi[j], jl = trial.clo[j];
    int ls, ld;
    float dx, dy, dz;
    if (classify_pair(ih, il, jh, jl, i, j, test.center, trial.center, trial.size, a.same_mesh, ls, ld, dx, dy, dz) !=
        KIND_REGULAR)
        return false;
    const int inc = test.nc[i], jnc = trial.nc[j];
    int ind1, ind2;
    if (a.same_mesh && common_nodes(test.nid[i], inc, trial.nid[j], jnc, ind1, ind2) > 0) {
        // a node shared beyond 1.5 D (strongly graded mesh): singular rule
        if (lanes.lane == 0) {
            const unsigned slot = atomicAdd(a.n_extra, 1u);
            if (slot < (unsigned)a.extra_cap) a.extra[slot] = make_int2(i, j);
            else atomicCAS(a.err, 0, -1);
        }
        return false;
    }
    if (!DO_S) ls = ld;
    if (!DO_D) ld = ls;
    const int cmax = (il.w != 0.0f || jl.w != 0.0f) ? 1 : 0;
    const int64_t bi = ((int64_t)i * 2 + cmax) * SLOTS, bj = ((int64_t)j * 2 + cmax) * SLOTS;
    for (int pass = 0; pass < (ls == ld ? 1 : 2); ++pass) {
        const int L = pass == 0 ? ls : ld;
        const float ws = (DO_S && ls == L) ? 1.0f : 0.0f, wd = (DO_D && ld == L) ? 1.0f : 0.0f;
        const int npi = level_npts(inc, cmax, L), npj = level_npts(jnc, cmax, L);
        for (int p = lanes.lane; p < npi; p += GAL2_LANES) {
            const float4 x = __ldg(test.pts32 + 2 * (bi + level_slot0(L) + p));
            for (int q = 0; q < npj; ++q) {
                const float4 y = __ldg(trial.pts32 + 2 * (bj + level_slot0(L) + q));
                const float4 n = __ldg(trial.pts32 + 2 * (bj + level_slot0(L) + q) + 1);
                eval_point<FAM, float>(dx + (y.x - x.x), dy + (y.y - x.y), dz + (y.z - x.z), y.w, n.x, n.y, n.z, a.k32,
                                       ws * x.w, wd * x.w, o.sr, o.si, o.dr, o.di);
            }
        }
    }
    o.sr = lanes.sum(o.sr);
    o.si = lanes.sum(o.si);
    o.dr = lanes.sum(o.dr);
    o.di = lanes.sum(o.di);
    return true;
}

template <int FAM, int OPS>
struct Gal2Op {
    static constexpr bool DO_S = (OPS & OP_SLP) != 0, DO_D = (OPS & OP_DLP) != 0;
    static constexpr float Q0 = DO_D ? 249.64f : 82.81f, Q1 = DO_D ? 7.84f : 3.24f;  // as Reg2Op
    static constexpr int GENERAL_LANES = GAL2_LANES;

    const GalArgs &a;
    const TwoRowShared &sh;
    int jb;
    float2 *out_s, *out_d;
    float k;

    struct Extra {
        f2 area;
        float size;  // the largest of the warp's rows
    };
    __device__ __forceinline__ Extra extra(int i0, int i1) const
    {
        float d = fmaxf(rsqrtf(a.test.chi[i0].w), rsqrtf(a.test.chi[i1].w));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) d = fmaxf(d, __shfl_xor_sync(0xffffffffu, d, o));
        return {f2_pack(a.test.p0[i0].x, a.test.p0[i1].x), d};
    }
    // beyond the distance at which elements of sizes 1/sqrt(iw) and d may share a node
    __device__ __forceinline__ bool apart(float iw, float d, float r2) const
    {
        const float reach = 2.0f * (rsqrtf(iw) + d);
        return !a.same_mesh || r2 > 1.01f * reach * reach;
    }
    __device__ __forceinline__ bool far(const Extra &e, int c, float q, float r2) const
    {
        return q > Q0 * (1.0f + 1e-4f) && apart(TwoRowCol::first(sh.col[c].iw), e.size, r2);
    }
    __device__ __forceinline__ int list(float q) const
    {
        const float lo = q * (1.0f - 1e-5f), hi = q * (1.0f + 1e-5f);  // classify_pair's guard band
        if (hi < 2.25f) return -1;
        if (DO_S && DO_D && lo >= 82.81f && hi < Q0) return 0;
        if (lo >= Q1 && hi < (DO_S ? 82.81f : Q0)) return 1;
        return 2;
    }
    __device__ __forceinline__ void put_one(int i, int c, float sr, float si, float dr, float di) const
    {
        const int64_t off = (int64_t)c * a.ld + i;
        if (DO_S) out_s[off] = make_float2(sr, si);
        if (DO_D) out_d[off] = make_float2(dr, di);
    }
    using Val = Gal2Val;
    template <int H>
    __device__ __forceinline__ void put(const Val &v, int c, int i) const
    {
        float x[4], y[4];
        f2_unpack(v.sr, x[0], y[0]);
        f2_unpack(v.si, x[1], y[1]);
        f2_unpack(v.dr, x[2], y[2]);
        f2_unpack(v.di, x[3], y[3]);
        if (H == 0) put_one(i, c, x[0], x[1], x[2], x[3]);
        else put_one(i, c, y[0], y[1], y[2], y[3]);
    }
    __device__ __forceinline__ static Val zero() { return {f2_dup(0.0f), f2_dup(0.0f), f2_dup(0.0f), f2_dup(0.0f)}; }
    __device__ __forceinline__ void far_eval(const Extra &e, int c, f2 dx, f2 dy, f2 dz, f2, Val &v) const
    {
        const TwoRowCol &t = sh.col[c];
        v = zero();
        gal2_point<FAM, DO_S, DO_D>(dx, dy, dz, t.w4, e.area, t.nx, t.ny, t.nz, k, v);
    }
    template <int LIST>
    __device__ __forceinline__ void pair(int i, int c) const
    {
        if constexpr (LIST == 1 || (DO_S && DO_D)) {
            constexpr bool PS = LIST == 1 && DO_S;  // the SLP at the level-1 points
            const TwoRowCol &t = sh.col[c];
            const int j = jb + c;
            const float3 d = t.diff(a.test, i);
            const float4 p = t.p0();
            Gal2Sums o;
            if (LIST == 0) gal2_point1<FAM, true, false, true>(d.x, d.y, d.z, p.x, a.test.p0[i].x, p.y, p.z, p.w, k, o);
            if (!a.test.has_quad && !a.trial.has_quad) {
                // 3 x 3 points, one normal
                const float4 *px = a.test.pts32 + 2 * ((int64_t)i * 2 * SLOTS + level_slot0(1));
                const float4 *py = a.trial.pts32 + 2 * ((int64_t)j * 2 * SLOTS + level_slot0(1));
                const float4 y0 = __ldg(py), y1 = __ldg(py + 2), y2 = __ldg(py + 4);
#pragma unroll
                for (int u = 0; u < 3; ++u) {
                    const float4 x = __ldg(px + 2 * u);
                    // the points' difference first: one rounding at the size of r
                    gal2_point1<FAM, PS, DO_D, false>(d.x + (y0.x - x.x), d.y + (y0.y - x.y), d.z + (y0.z - x.z), y0.w, x.w, p.y, p.z, p.w, k, o);
                    gal2_point1<FAM, PS, DO_D, false>(d.x + (y1.x - x.x), d.y + (y1.y - x.y), d.z + (y1.z - x.z), y1.w, x.w, p.y, p.z, p.w, k, o);
                    gal2_point1<FAM, PS, DO_D, false>(d.x + (y2.x - x.x), d.y + (y2.y - x.y), d.z + (y2.z - x.z), y2.w, x.w, p.y, p.z, p.w, k, o);
                }
            } else {
                const int inc = a.test.nc[i], jnc = a.trial.nc[j], cmax = inc == 4 || jnc == 4 ? 1 : 0;
                const float4 *px = a.test.pts32 + 2 * (((int64_t)i * 2 + cmax) * SLOTS + level_slot0(1));
                const float4 *py = a.trial.pts32 + 2 * (((int64_t)j * 2 + cmax) * SLOTS + level_slot0(1));
                const int npi = level_npts(inc, cmax, 1), npj = level_npts(jnc, cmax, 1);
                for (int u = 0; u < npi; ++u) {
                    const float4 x = __ldg(px + 2 * u);
                    for (int v = 0; v < npj; ++v) {
                        const float4 y = __ldg(py + 2 * v), n = __ldg(py + 2 * v + 1);
                        gal2_point1<FAM, PS, DO_D, false>(d.x + (y.x - x.x), d.y + (y.y - x.y), d.z + (y.z - x.z), y.w, x.w, n.x, n.y, n.z, k, o);
                    }
                }
            }
            // within reach the elements may share a node: the singular rule's pairs are listed
            if (clear(i, j, t, d)) put_one(i, c, o.sr, o.si, o.dr, o.di);
        }
    }
    // false: a pair that shares a node, which goes to the extra list
    __device__ __forceinline__ bool clear(int i, int j, const TwoRowCol &t, float3 d) const
    {
        if (apart(TwoRowCol::first(t.iw), rsqrtf(a.test.chi[i].w), d.x * d.x + d.y * d.y + d.z * d.z)) return true;
        int ind1, ind2;
        if (common_nodes(a.test.nid[i], a.test.nc[i], a.trial.nid[j], a.trial.nc[j], ind1, ind2) == 0) return true;
        const unsigned slot = atomicAdd(a.n_extra, 1u);
        if (slot < (unsigned)a.extra_cap) a.extra[slot] = make_int2(i, j);
        else atomicCAS(a.err, 0, -1);
        return false;
    }
    __device__ __forceinline__ void general(int i, int c) const
    {
        Gal2Sums o;
        if (gal2_general<FAM, OPS>(a, i, jb + c, o) && (threadIdx.x & (GAL2_LANES - 1)) == 0)
            put_one(i, c, o.sr, o.si, o.dr, o.di);
    }
};

template <int FAM, int OPS>
__global__ void __launch_bounds__(TWO_ROW_THREADS, 20 / TWO_ROW_WARPS) k_galerkin_regular2(const __grid_constant__ GalArgs a,
                                                                                          int cols_per_block)
{
    __shared__ TwoRowShared sh;
    const int jb = a.j0 + blockIdx.y * cols_per_block;
    const int ncols = min(cols_per_block, a.j1 - jb);
    if (threadIdx.x < ncols) sh.stage(threadIdx.x, a.trial, jb + threadIdx.x);
    __syncthreads();
    const int ib = blockIdx.x * TWO_ROW_ROWS;
    if (ib + 64 * (threadIdx.x >> 5) >= a.test.n) return;
    const int64_t off = (int64_t)(jb - a.j0) * a.ld;
    const Gal2Op<FAM, OPS> op{a, sh, jb, reinterpret_cast<float2 *>(a.out_s) + off,
                              reinterpret_cast<float2 *>(a.out_d) + off, a.k32};
    if (ib + TWO_ROW_ROWS <= a.test.n) two_row_columns<true>(op, sh, a.test, ib, ncols);
    else two_row_columns<false>(op, sh, a.test, ib, ncols);
}

template <int FAM>
static cudaError_t launch_galerkin_regular2(const GalArgs &a, cudaStream_t s)
{
    const auto kernel = a.ops == OP_SLP   ? k_galerkin_regular2<FAM, OP_SLP>
                        : a.ops == OP_DLP ? k_galerkin_regular2<FAM, OP_DLP>
                                          : k_galerkin_regular2<FAM, OP_SLP | OP_DLP>;
    return two_row_launches(a.test.n, a.j0, a.j1, [&](int j0, int j1, dim3 grid, int cols) {
        GalArgs b = a;
        b.j0 = j0;
        b.j1 = j1;
        b.out_s = reinterpret_cast<float2 *>(a.out_s) + (int64_t)(j0 - a.j0) * a.ld;
        b.out_d = reinterpret_cast<float2 *>(a.out_d) + (int64_t)(j0 - a.j0) * a.ld;
        kernel<<<grid, TWO_ROW_THREADS, 0, s>>>(b, cols);
    });
}

// ------------------------------------------------- near pairs, FP32 triangles

// sin and cos in FP32: the Taylor series to x^13 and x^12 for |x| <= pi/2
// (truncation below 7e-10 and 7e-9), when the caller's bound allows (warp-uniform), else
// the library's
__device__ __forceinline__ void sincos_short(float x, bool bounded, float &s, float &c)
{
    if (!bounded) {
        sincosf(x, &s, &c);
        return;
    }
    const float u = x * x;
    float p = fmaf(1.0f / 6227020800.0f, u, -1.0f / 39916800.0f), q = 1.0f / 479001600.0f;
    p = fmaf(p, u, 1.0f / 362880.0f);
    q = fmaf(q, u, -1.0f / 3628800.0f);
    p = fmaf(p, u, -1.0f / 5040.0f);
    q = fmaf(q, u, 1.0f / 40320.0f);
    p = fmaf(p, u, 1.0f / 120.0f);
    q = fmaf(q, u, -1.0f / 720.0f);
    p = fmaf(p, u, -1.0f / 6.0f);
    q = fmaf(q, u, 1.0f / 24.0f);
    q = fmaf(q, u, -0.5f);
    s = fmaf(p * u, x, x);
    c = fmaf(q, u, 1.0f);
}

// k_galerkin_near for triangles under FP32 quadrature and a real wave number:
// the same rules and points.  That kernel runs every warp through FP64 copies
// of the pair's corners on all lanes (46% of its time the FP64 pipe, two
// blocks per SM at 128 registers); here 21 lanes form one corner or centre
// difference each in FP64, rounded to FP32 and shared by shuffles.
// 5120 triangles (94 100 pairs), alone: 250 us.
template <typename Out, int FAM>
__global__ void __launch_bounds__(GAL_WARPS * 32) k_galerkin_near_tria(const __grid_constant__ GalArgs a, NearList near,
                                                                       int extra)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    int64_t n_near = 0, p_begin = 0, total = 0;
    if (extra) {
        total = min((int64_t)*a.n_extra, (int64_t)a.extra_cap);
    } else {
        p_begin = near.col_ptr ? near.col_ptr[a.j0] : 0;
        n_near = (near.col_ptr ? near.col_ptr[a.j1] : 0) - p_begin;
        total = n_near + (a.same_mesh ? (int64_t)(a.j1 - a.j0) : 0);
    }
    const bool do_s = (a.ops & OP_SLP) != 0, do_d = (a.ops & OP_DLP) != 0;
    Out *out_s = reinterpret_cast<Out *>(a.out_s);
    Out *out_d = reinterpret_cast<Out *>(a.out_d);
    const float kf = a.k32;
    for (int64_t item = warp; item < total; item += nwarps) {
        int i, j;
        if (extra) {
            const int2 e = a.extra[item];
            i = e.x;
            j = e.y;
        } else if (item < n_near) {
            const int64_t p = p_begin + item;
            i = near.rows[p];
            j = near_column(near.col_ptr, a.j0, a.j1, p);
        } else {
            j = a.j0 + (int)(item - n_near);
            i = j;
            if (i >= a.test.n) continue;
        }
        int match = -1, ind1 = 0, ind2 = 0;
        if (a.same_mesh) {
            if (i == j) {
                match = 2;
            } else {
                const int num = common_nodes(a.test.nid[i], 3, a.trial.nid[j], 3, ind1, ind2);
                match = num > 1 ? 1 : (num == 1 ? 0 : -1);
            }
        }
        // lane 3 q + d (9 + 3 q + d): coordinate d of corner q of the test (trial)
        // element, relative to test corner 0 (matched), or of its sides and of
        // corner 0 relative to its centre (unmatched); 18 + d: the centres' difference
        float mine = 0.0f;
        if (lane < 21) {
            const int d = lane % 3, q = (lane / 3) % 3;
            const bool on_trial = lane >= 9;
            const double *ci = a.test.corners + 12 * (int64_t)i, *cj = a.trial.corners + 12 * (int64_t)j;
            const double *xi = a.test.center + 3 * (int64_t)i, *xj = a.trial.center + 3 * (int64_t)j;
            double from, to;
            if (lane >= 18) {
                to = xj[d];
                from = xi[d];
            } else {
                to = (on_trial ? cj : ci)[3 * q + d];
                from = match >= 0 ? ci[d] : (q == 0 ? (on_trial ? xj : xi)[d] : (on_trial ? cj : ci)[d]);
            }
            mine = (float)(to - from);
        }
        float tc[3][3], rc[3][3];
#pragma unroll
        for (int q = 0; q < 3; ++q)
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                tc[q][d] = __shfl_sync(0xffffffffu, mine, 3 * q + d);
                rc[q][d] = __shfl_sync(0xffffffffu, mine, 9 + 3 * q + d);
            }
        // sides of both elements (in their own orientation), normals
        float e1[3], e2[3], f1[3], f2v[3], ntv[3], nrv[3], nrm[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            e1[d] = match >= 0 ? tc[1][d] - tc[0][d] : tc[1][d];
            e2[d] = match >= 0 ? tc[2][d] - tc[0][d] : tc[2][d];
            f1[d] = match >= 0 ? rc[1][d] - rc[0][d] : rc[1][d];
            f2v[d] = match >= 0 ? rc[2][d] - rc[0][d] : rc[2][d];
        }
        ntv[0] = e1[1] * e2[2] - e1[2] * e2[1];
        ntv[1] = e1[2] * e2[0] - e1[0] * e2[2];
        ntv[2] = e1[0] * e2[1] - e1[1] * e2[0];
        nrv[0] = f1[1] * f2v[2] - f1[2] * f2v[1];
        nrv[1] = f1[2] * f2v[0] - f1[0] * f2v[2];
        nrv[2] = f1[0] * f2v[1] - f1[1] * f2v[0];
        const float Jt = sqrtf(ntv[0] * ntv[0] + ntv[1] * ntv[1] + ntv[2] * ntv[2]);
        const float Jr = sqrtf(nrv[0] * nrv[0] + nrv[1] * nrv[1] + nrv[2] * nrv[2]);
#pragma unroll
        for (int d = 0; d < 3; ++d) nrm[d] = nrv[d] / Jr;
        const float wscale = Jt * Jr * (float)(1.0 / FOUR_PI);
        // a corner is at most D from its centre (the longest side is below 1.5 D), a
        // listed pair's centres at most 1.5 D_j apart: r <= D_i + 2.5 D_j
        const float r_max = rsqrtf(a.test.chi[i].w) + 2.5f * rsqrtf(a.trial.chi[j].w);
        const bool bounded = !extra && fabsf(kf) * r_max <= 1.57f;
        float fsr = 0, fsi = 0, fdr = 0, fdi = 0;
        auto point = [&](const float rv[3], float w, bool use_s, bool use_d) {
            const float r2 = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
            const float rinv = rsqrtf(r2);
            const float g = w * wscale * rinv;  // w Jt Jr / (4 pi r)
            float sn = 0.0f, cs = 1.0f, kr = 0.0f;
            if constexpr (FAM == FAM_HELMHOLTZ) {
                kr = kf * (r2 * rinv);
                sincos_short(kr, bounded, sn, cs);
            }
            if (use_s) {
                fsr += g * cs;
                fsi -= g * sn;
            }
            if (use_d) {
                const float f = -g * rinv * (rv[0] * nrm[0] + rv[1] * nrm[1] + rv[2] * nrm[2]) * rinv;
                fdr += f * (cs + kr * sn);
                fdi += f * (kr * cs - sn);
            }
        };
        if (match >= 0) {
            // both rotated triangles start at the common node: r_vec from their
            // sides there and the rule's FP64-formed coordinate differences
            int pt[3], pr[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                pt[q] = match == 2 ? q : (ind1 + q) % 3;
                pr[q] = match == 2 ? q : (match == 1 ? (ind2 + 1 + 3 - q) % 3 : (ind2 + q) % 3);
            }
            auto pick = [](const float (&c)[3][3], int idx, int d) {
                return idx == 0 ? c[0][d] : (idx == 1 ? c[1][d] : c[2][d]);
            };
            float at[3], bt[3], ar[3], br[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                at[d] = pick(tc, pt[1], d) - pick(tc, pt[0], d);
                bt[d] = pick(tc, pt[2], d) - pick(tc, pt[0], d);
                ar[d] = pick(rc, pr[1], d) - pick(rc, pr[0], d);
                br[d] = pick(rc, pr[2], d) - pick(rc, pr[0], d);
            }
            const float4 *rule = reinterpret_cast<const float4 *>(g_gal_rule32) + 2 * (size_t)gal_offset(match);
            const int np = gal_npts(match);
            // q0 = (xi1, xi2, eta1, eta2), q1 = (w, eta1 - xi1, eta2 - xi2, 0)
            auto sum = [&](auto form) {
#pragma unroll 2
                for (int p = lane; p < np; p += 32) {
                    const float4 q0 = __ldg(rule + 2 * p), q1 = __ldg(rule + 2 * p + 1);
                    float rv[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d) rv[d] = form(q0, q1, d);
                    point(rv, q1.x, do_s, do_d);
                }
            };
            if (match == 2) sum([&](float4, float4 q1, int d) { return q1.y * at[d] + q1.z * bt[d]; });
            else if (match == 1)
                sum([&](float4 q0, float4 q1, int d) { return q1.y * at[d] + q0.w * br[d] - q0.y * bt[d]; });
            else
                sum([&](float4 q0, float4, int d) {
                    return q0.z * ar[d] + q0.w * br[d] - q0.x * at[d] - q0.y * bt[d];
                });
        } else {
            // the product rules of the degrees of d/D, decided in FP32 with the
            // FP64 guard band of the classification
            float c0[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) c0[d] = __shfl_sync(0xffffffffu, mine, 18 + d);
            const float ratio = sqrtf(c0[0] * c0[0] + c0[1] * c0[1] + c0[2] * c0[2]) / (float)a.trial.size[j];
            double rx = (double)ratio;
            if (fabsf(ratio - 1.1f) < 1e-4f || fabsf(ratio - 1.5f) < 1e-4f || fabsf(ratio - 1.8f) < 1e-4f) {
                double dcd[3];
                for (int d = 0; d < 3; ++d)
                    dcd[d] = a.trial.center[3 * (int64_t)j + d] - a.test.center[3 * (int64_t)i + d];
                rx = norm3(dcd) / a.trial.size[j];
            }
            const int deg_s = rx < 11.0 / 10.0 ? 6 : (rx < T_S1 ? 4 : (rx < T_S0 ? 2 : 0));
            const int deg_d = rx < 11.0 / 10.0 ? 8 : (rx < T_NEAR ? 6 : (rx < T_D1 ? 4 : (rx < T_D0 ? 2 : 0)));
            const bool one_pass = !do_s || !do_d || deg_s == deg_d;
            for (int pass = 0; pass < (one_pass ? 1 : 2); ++pass) {
                const bool use_s = one_pass ? do_s : pass == 0;
                const bool use_d = one_pass ? do_d : pass == 1;
                const int deg = use_s ? deg_s : deg_d;
                const int npt = g_tri_npts[deg];
                const float *rule = TRI_F32.v + 3 * g_tri_off[deg];
                for (int p = lane; p < npt * npt; p += 32) {
                    const float *qa = rule + 3 * (p / npt), *qb = rule + 3 * (p % npt);
                    const float fxa = qa[0], fea = qa[1], wa = qa[2], fxb = qb[0], feb = qb[1], wb = qb[2];
                    float rv[3];
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        rv[d] = c0[d] + (rc[0][d] + fxb * f1[d] + feb * f2v[d]) - (tc[0][d] + fxa * e1[d] + fea * e2[d]);
                    point(rv, wa * wb, use_s, use_d);
                }
            }
        }
        // the four sums over the lanes in FP64, two, then one value per lane: after
        // two exchanges lanes 0-7 hold sr, 8-15 si, 16-23 dr, 24-31 di
        const bool up = lane & 16, odd = lane & 8;
        double va = (double)(up ? fdr : fsr), vb = (double)(up ? fdi : fsi);
        va += (double)__shfl_xor_sync(0xffffffffu, up ? fsr : fdr, 16);
        vb += (double)__shfl_xor_sync(0xffffffffu, up ? fsi : fdi, 16);
        double v = odd ? vb : va;
        v += __shfl_xor_sync(0xffffffffu, odd ? va : vb, 8);
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const double im = __shfl_down_sync(0xffffffffu, v, 8);
        if (lane == 0 || lane == 16) {
            const bool slp = lane == 0;
            if (slp ? do_s : do_d)
                store64((slp ? out_s : out_d) + (int64_t)(j - a.j0) * a.ld + i, v, im, a.alpha_re, a.alpha_im,
                        a.accumulate);
        }
    }
}

template <typename Out>
static cudaError_t launch_galerkin_near_tria(const GalArgs &a, const NearList &near, int extra, int64_t max_items, int sms,
                                             cudaStream_t s)
{
    const auto kernel = a.family == FAM_HELMHOLTZ ? k_galerkin_near_tria<Out, FAM_HELMHOLTZ>
                                                  : k_galerkin_near_tria<Out, FAM_LAPLACE>;
    const int64_t want = (max_items + GAL_WARPS - 1) / GAL_WARPS;
    // as many blocks as an SM holds at 72 registers: the regular kernel, launched
    // beside this one, follows into the SMs as they drain (5120 triangles, both
    // together: 4, 6, 7 blocks per SM 952, 900, 888 us; one after the other 950)
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(want, 7 * (int64_t)sms));
    kernel<<<blocks, GAL_WARPS * 32, 0, s>>>(a, near, extra);
    return cudaGetLastError();
}

// point p of the product rule of a given degree on an element: reference
// coordinates and weight (Dunavant on triangles, Gauss tensor on quads)
__device__ __forceinline__ void product_point(int nc, int degree, int p, double &xi, double &eta, double &w)
{
    if (nc == 3) {
        tri_pt(degree, p, xi, eta, w);
    } else {
        const int ng = degree / 2 + 1;
        double w0, w1;
        gauss_pt(ng, p / ng, xi, w0);
        gauss_pt(ng, p % ng, eta, w1);
        w = w0 * w1;
    }
}

__device__ __forceinline__ int product_npts(int nc, int degree)
{
    if (nc == 3) return g_tri_npts[degree];
    const int ng = degree / 2 + 1;
    return ng * ng;
}

// reference point under a corner rotation of the triangle: corner k of the
// rotated triangle is corner perm[k] of (0,0), (1,0), (0,1)
__device__ __forceinline__ void tri_rotate(const int perm[3], double xi, double eta, double &oxi, double &oeta)
{
    const double N[3] = {1.0 - xi - eta, xi, eta};
    oxi = 0.0;
    oeta = 0.0;
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        oxi += perm[q] == 1 ? N[q] : 0.0;
        oeta += perm[q] == 2 ? N[q] : 0.0;
    }
}

// reference point of the square under a corner rotation: corner k of the
// rotated square is corner perm[k] of (-1,-1), (1,-1), (1,1), (-1,1)
__device__ __forceinline__ void quad_rotate(const int perm[4], double u, double v, double &ou, double &ov)
{
    const double N[4] = {(1 - u) * (1 - v) / 4, (1 + u) * (1 - v) / 4, (1 + u) * (1 + v) / 4, (1 - u) * (1 + v) / 4};
    ou = 0.0;
    ov = 0.0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = perm[q];
        ou += (c == 1 || c == 2) ? N[q] : -N[q];
        ov += (c >= 2) ? N[q] : -N[q];
    }
}

// The self pairs, the nearly singular list of columns [j0, j1) (extra = 0)
// or the extra list (extra = 1): one warp per pair
// CK: a complex (lossy) wave number: the FP64 rules with the complex kernel in both modes
template <typename Out, bool CK>
__global__ void __launch_bounds__(GAL_WARPS * 32) k_galerkin_near(GalArgs a, NearList near, int extra)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    int64_t n_near = 0, p_begin = 0, total = 0;
    if (extra) {
        total = min((int64_t)*a.n_extra, (int64_t)a.extra_cap);
    } else {
        p_begin = near.col_ptr ? near.col_ptr[a.j0] : 0;
        n_near = (near.col_ptr ? near.col_ptr[a.j1] : 0) - p_begin;
        total = n_near + (a.same_mesh ? (int64_t)(a.j1 - a.j0) : 0);
    }
    const bool do_s = (a.ops & OP_SLP) != 0, do_d = (a.ops & OP_DLP) != 0;
    const int fam = a.family;
    const double k = a.k;
    const cd kc{a.k, a.k_im};
    // kernel values at one point pair: the real or the complex wave number
    auto kp = [&](const double *x, const double *y, const double *n, double J, bool s_, bool d_, cd &ks, cd &kd) {
        if constexpr (CK) kern_point(fam, kc, x, y, n, J, s_, d_, ks, kd);
        else kern_point(fam, k, x, y, n, J, s_, d_, ks, kd);
    };
    Out *out_s = reinterpret_cast<Out *>(a.out_s);
    Out *out_d = reinterpret_cast<Out *>(a.out_d);
    for (int64_t item = warp; item < total; item += nwarps) {
        int i, j;
        if (extra) {
            const int2 e = a.extra[item];
            i = e.x;
            j = e.y;
        } else if (item < n_near) {
            const int64_t p = p_begin + item;
            i = near.rows[p];
            j = near_column(near.col_ptr, a.j0, a.j1, p);
        } else {
            j = a.j0 + (int)(item - n_near);
            i = j;
            if (i >= a.test.n) continue;
        }
        Elem64 te, re;
        load_elem(a.test, i, te);
        load_elem(a.trial, j, re);
        int match = -1, ind1 = 0, ind2 = 0;
        if (a.same_mesh) {
            if (i == j) match = 2;
            else {
                const int num = common_nodes(a.test.nid[i], te.nc, a.trial.nid[j], re.nc, ind1, ind2);
                match = num > 1 ? 1 : (num == 1 ? 0 : -1);
            }
        }
        double sr = 0, si = 0, dr = 0, di = 0;
        if (match >= 0 && te.nc != re.nc) {
            // triangle-quad match, corner or edge (FP64 in both modes;
            // nihu/core/singular_galerkin_quadrature.hpp:624-790): the quad's
            // reference square split into the triangles (0, 1, 2) and (0, 2, 3)
            // of its rotated corners, the triangle-triangle corner rule on both
            // (corner match) or the edge rule on (0, 1, 2) and the corner rule on
            // (0, 2, 3) (edge match); the rule's first triangle on the quad half
            // by its linear map (Jacobian 4), its second on the triangle.  The
            // rotations are those of the other pairs.
            const int ntc = te.nc, nrc = re.nc;
            int pt[4], pr[4];
            for (int q = 0; q < ntc; ++q) pt[q] = (ind1 + q) % ntc;
            for (int q = 0; q < nrc; ++q) pr[q] = match == 1 ? (ind2 + 1 + nrc - q) % nrc : (ind2 + q) % nrc;
            const bool quad_test = ntc == 4;
            const int m_first = match == 1 ? 1 : 0;
            const int na = gal_npts(m_first), total_p = na + gal_npts(0);
            for (int p = lane; p < total_p; p += 32) {
                const int sub = p < na ? 0 : 1;
                const double *q = g_gal_rule + 5 * (size_t)(sub == 0 ? gal_offset(m_first) + p : gal_offset(0) + p - na);
                const double N0 = 1.0 - q[0] - q[1], N1 = q[0], N2 = q[1];
                // half (0, 1, 2): (-1,-1), (1,-1), (1,1); half (0, 2, 3): (-1,-1), (1,1), (-1,1)
                const double qu = sub == 0 ? -N0 + N1 + N2 : -N0 + N1 - N2;
                const double qv = sub == 0 ? -N0 - N1 + N2 : -N0 + N1 + N2;
                double tu, tv, ru, rv;
                if (quad_test) {
                    quad_rotate(pt, qu, qv, tu, tv);
                    tri_rotate(pr, q[2], q[3], ru, rv);
                } else {
                    tri_rotate(pt, q[2], q[3], tu, tv);
                    quad_rotate(pr, qu, qv, ru, rv);
                }
                double x[3], y[3], ntv[3], nrv[3];
                ex(te, tu, tv, x);
                enormal(te, tu, tv, ntv);
                ex(re, ru, rv, y);
                enormal(re, ru, rv, nrv);
                cd ks{0, 0}, kd{0, 0};
                kp(x, y, nrv, norm3(nrv), do_s, do_d, ks, kd);
                const double w = 4.0 * q[4] * norm3(ntv);
                sr += ks.re * w;
                si += ks.im * w;
                dr += kd.re * w;
                di += kd.im * w;
            }
        } else if (match >= 0 && te.nc == 4) {
            // matched quads (FP64, both precisions): points by the bilinear
            // maps, Jacobians and normals per point
            int pt[4], pr[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                pt[q] = match == 2 ? q : (ind1 + q) % 4;
                pr[q] = match == 2 ? q : (match == 1 ? (ind2 + 1 + 4 - q) % 4 : (ind2 + q) % 4);
            }
            const double *rule = g_galq_rule + 5 * (size_t)galq_offset(match);
            const int np = galq_npts(match);
            for (int p = lane; p < np; p += 32) {
                const double *q = rule + 5 * p;
                double u, v, x[3], y[3], nt3[3], nr3[3];
                quad_rotate(pt, q[0], q[1], u, v);
                ex(te, u, v, x);
                enormal(te, u, v, nt3);
                quad_rotate(pr, q[2], q[3], u, v);
                ex(re, u, v, y);
                enormal(re, u, v, nr3);
                cd ks{0, 0}, kd{0, 0};
                kp(x, y, nr3, norm3(nr3), do_s, do_d, ks, kd);
                const double w = q[4] * norm3(nt3);
                sr += ks.re * w;
                si += ks.im * w;
                dr += kd.re * w;
                di += kd.im * w;
            }
        } else if (match >= 0 && a.precision == 0 && !CK) {
            // FP32 regular quadrature: the matched pair's rule in FP32 too.  Both
            // rotated triangles start at the common node P, so r_vec = y - x is
            // formed from P-relative edge vectors and the rule's FP64-formed
            // coordinate differences, keeping FP32 relative accuracy as r -> 0
            int pt[3], pr[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                pt[q] = match == 2 ? q : (ind1 + q) % 3;
                pr[q] = match == 2 ? q : (match == 1 ? (ind2 + 1 + 3 - q) % 3 : (ind2 + q) % 3);
            }
            // corners relative to the test element's corner 0 in FP32 (the
            // differences in FP64); the rest of the set-up in FP32, so the
            // warp's lanes do not repeat FP64 work on the narrow FP64 pipe
            float tc[3][3], rc[3][3];
#pragma unroll
            for (int q = 0; q < 3; ++q)
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    tc[q][d] = (float)(te.c[q][d] - te.c[0][d]);
                    rc[q][d] = (float)(re.c[q][d] - te.c[0][d]);
                }
            auto pick = [](const float (&c)[3][3], int idx, int d) {
                return idx == 0 ? c[0][d] : (idx == 1 ? c[1][d] : c[2][d]);
            };
            float at[3], bt[3], ar[3], br[3], nrm[3], ntv[3], nrv[3], e1[3], e2[3], f1[3], f2[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                at[d] = pick(tc, pt[1], d) - pick(tc, pt[0], d);
                bt[d] = pick(tc, pt[2], d) - pick(tc, pt[0], d);
                ar[d] = pick(rc, pr[1], d) - pick(rc, pr[0], d);
                br[d] = pick(rc, pr[2], d) - pick(rc, pr[0], d);
                e1[d] = tc[1][d] - tc[0][d];
                e2[d] = tc[2][d] - tc[0][d];
                f1[d] = rc[1][d] - rc[0][d];  // the trial element's own orientation
                f2[d] = rc[2][d] - rc[0][d];
            }
            ntv[0] = e1[1] * e2[2] - e1[2] * e2[1];
            ntv[1] = e1[2] * e2[0] - e1[0] * e2[2];
            ntv[2] = e1[0] * e2[1] - e1[1] * e2[0];
            nrv[0] = f1[1] * f2[2] - f1[2] * f2[1];
            nrv[1] = f1[2] * f2[0] - f1[0] * f2[2];
            nrv[2] = f1[0] * f2[1] - f1[1] * f2[0];
            const float Jtf = sqrtf(ntv[0] * ntv[0] + ntv[1] * ntv[1] + ntv[2] * ntv[2]);
            const float Jrf = sqrtf(nrv[0] * nrv[0] + nrv[1] * nrv[1] + nrv[2] * nrv[2]);
#pragma unroll
            for (int d = 0; d < 3; ++d) nrm[d] = nrv[d] / Jrf;
            const float wscale = Jtf * Jrf * (float)(1.0 / FOUR_PI);
            const float kf = (float)k;
            const float *rule = g_gal_rule32 + 8 * (size_t)gal_offset(match);
            const int np = gal_npts(match);
            float fsr = 0, fsi = 0, fdr = 0, fdi = 0;
            for (int p = lane; p < np; p += 32) {
                const float4 q0 = *reinterpret_cast<const float4 *>(rule + 8 * p);
                const float4 q1 = *reinterpret_cast<const float4 *>(rule + 8 * p + 4);
                // q0 = (xi1, xi2, eta1, eta2), q1 = (w, eta1 - xi1, eta2 - xi2, 0)
                float rv[3];
                for (int d = 0; d < 3; ++d) {
                    if (match == 2) rv[d] = q1.y * at[d] + q1.z * bt[d];
                    else if (match == 1) rv[d] = q1.y * at[d] + q0.w * br[d] - q0.y * bt[d];
                    else rv[d] = q0.z * ar[d] + q0.w * br[d] - q0.x * at[d] - q0.y * bt[d];
                }
                const float r2 = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
                const float rinv = rsqrtf(r2);
                const float g = q1.x * wscale * rinv;  // w Jt Jr / (4 pi r)
                float sn = 0.0f, cs = 1.0f, kr = 0.0f;
                if (fam == FAM_HELMHOLTZ) {
                    kr = kf * (r2 * rinv);
                    sincosf(kr, &sn, &cs);
                }
                fsr += g * cs;
                fsi -= g * sn;
                const float f = -g * rinv * (rv[0] * nrm[0] + rv[1] * nrm[1] + rv[2] * nrm[2]) * rinv;
                fdr += f * (cs + kr * sn);
                fdi += f * (kr * cs - sn);
            }
            sr = fsr;
            si = fsi;
            dr = do_d ? fdr : 0.0f;
            di = do_d ? fdi : 0.0f;
        } else if (match >= 0) {
            // matched triangles: flat elements
            int pt[3], pr[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                pt[q] = match == 2 ? q : (ind1 + q) % 3;
                pr[q] = match == 2 ? q : (match == 1 ? (ind2 + 1 + 3 - q) % 3 : (ind2 + q) % 3);
            }
            double t1[3], t2[3], r1[3], r2[3], nt[3], nr[3];
            for (int d = 0; d < 3; ++d) {
                t1[d] = te.c[1][d] - te.c[0][d];
                t2[d] = te.c[2][d] - te.c[0][d];
                r1[d] = re.c[1][d] - re.c[0][d];
                r2[d] = re.c[2][d] - re.c[0][d];
            }
            cross3(t1, t2, nt);
            cross3(r1, r2, nr);
            const double Jt = norm3(nt), Jr = norm3(nr);
            const double *rule = g_gal_rule + 5 * (size_t)gal_offset(match);
            const int np = gal_npts(match);
            for (int p = lane; p < np; p += 32) {
                const double *q = rule + 5 * p;
                double u, v, x[3], y[3];
                tri_rotate(pt, q[0], q[1], u, v);
                for (int d = 0; d < 3; ++d) x[d] = te.c[0][d] + u * t1[d] + v * t2[d];
                tri_rotate(pr, q[2], q[3], u, v);
                for (int d = 0; d < 3; ++d) y[d] = re.c[0][d] + u * r1[d] + v * r2[d];
                cd ks{0, 0}, kd{0, 0};
                kp(x, y, nr, Jr, do_s, do_d, ks, kd);
                const double w = q[4] * Jt;
                sr += ks.re * w;
                si += ks.im * w;
                dr += kd.re * w;
                di += kd.im * w;
            }
        } else if (a.precision == 0 && te.nc == 3 && re.nc == 3 && !CK) {
            // unmatched close triangles under FP32 regular quadrature: the same
            // product rules in FP32, points relative to the element centres
            // (r_vec = (c_j - c_i) + (y - c_j) - (x - c_i), the first term
            // formed in FP64); the degree decision in FP32 with the FP64 guard
            // band of the classification
            double dcd[3];
            for (int d = 0; d < 3; ++d) dcd[d] = a.trial.center[3 * (int64_t)j + d] - a.test.center[3 * (int64_t)i + d];
            float c0[3];
            for (int d = 0; d < 3; ++d) c0[d] = (float)dcd[d];
            const float size_j = (float)a.trial.size[j];
            const float ratio = sqrtf(c0[0] * c0[0] + c0[1] * c0[1] + c0[2] * c0[2]) / size_j;
            int deg_s, deg_d;
            {
                const double rx = (fabsf(ratio - 1.1f) < 1e-4f || fabsf(ratio - 1.5f) < 1e-4f || fabsf(ratio - 1.8f) < 1e-4f)
                                      ? norm3(dcd) / a.trial.size[j]
                                      : (double)ratio;
                deg_s = rx < 11.0 / 10.0 ? 6 : (rx < T_S1 ? 4 : (rx < T_S0 ? 2 : 0));
                deg_d = rx < 11.0 / 10.0 ? 8 : (rx < T_NEAR ? 6 : (rx < T_D1 ? 4 : (rx < T_D0 ? 2 : 0)));
            }
            float ti0[3], ti1[3], ti2[3], tj0[3], tj1[3], tj2[3], nrm[3], nt[3], nr[3];
            for (int d = 0; d < 3; ++d) {
                ti0[d] = (float)(te.c[0][d] - a.test.center[3 * (int64_t)i + d]);
                ti1[d] = (float)(te.c[1][d] - te.c[0][d]);
                ti2[d] = (float)(te.c[2][d] - te.c[0][d]);
                tj0[d] = (float)(re.c[0][d] - a.trial.center[3 * (int64_t)j + d]);
                tj1[d] = (float)(re.c[1][d] - re.c[0][d]);
                tj2[d] = (float)(re.c[2][d] - re.c[0][d]);
            }
            nt[0] = ti1[1] * ti2[2] - ti1[2] * ti2[1];
            nt[1] = ti1[2] * ti2[0] - ti1[0] * ti2[2];
            nt[2] = ti1[0] * ti2[1] - ti1[1] * ti2[0];
            nr[0] = tj1[1] * tj2[2] - tj1[2] * tj2[1];
            nr[1] = tj1[2] * tj2[0] - tj1[0] * tj2[2];
            nr[2] = tj1[0] * tj2[1] - tj1[1] * tj2[0];
            const float Jt = sqrtf(nt[0] * nt[0] + nt[1] * nt[1] + nt[2] * nt[2]);
            const float Jr = sqrtf(nr[0] * nr[0] + nr[1] * nr[1] + nr[2] * nr[2]);
            for (int d = 0; d < 3; ++d) nrm[d] = nr[d] / Jr;
            const float kf = (float)k, wscale = Jt * Jr * (float)(1.0 / FOUR_PI);
            const bool one_pass = !do_s || !do_d || deg_s == deg_d;
            float fsr = 0, fsi = 0, fdr = 0, fdi = 0;
            for (int pass = 0; pass < (one_pass ? 1 : 2); ++pass) {
                const bool use_s = one_pass ? do_s : pass == 0;
                const bool use_d = one_pass ? do_d : pass == 1;
                const int deg = use_s ? deg_s : deg_d;
                const int npt = g_tri_npts[deg];
                const float *rule = TRI_F32.v + 3 * g_tri_off[deg];
                for (int p = lane; p < npt * npt; p += 32) {
                    const float *qa = rule + 3 * (p / npt), *qb = rule + 3 * (p % npt);
                    const float fxa = qa[0], fea = qa[1], wa = qa[2], fxb = qb[0], feb = qb[1], wb = qb[2];
                    float rv[3];
                    for (int d = 0; d < 3; ++d)
                        rv[d] = c0[d] + (tj0[d] + fxb * tj1[d] + feb * tj2[d]) - (ti0[d] + fxa * ti1[d] + fea * ti2[d]);
                    const float r2 = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
                    const float rinv = rsqrtf(r2);
                    const float g = wa * wb * wscale * rinv;
                    float sn = 0.0f, cs = 1.0f, kr = 0.0f;
                    if (fam == FAM_HELMHOLTZ) {
                        kr = kf * (r2 * rinv);
                        sincosf(kr, &sn, &cs);
                    }
                    if (use_s) {
                        fsr += g * cs;
                        fsi -= g * sn;
                    }
                    if (use_d) {
                        const float f = -g * rinv * (rv[0] * nrm[0] + rv[1] * nrm[1] + rv[2] * nrm[2]) * rinv;
                        fdr += f * (cs + kr * sn);
                        fdi += f * (kr * cs - sn);
                    }
                }
            }
            sr = fsr;
            si = fsi;
            dr = fdr;
            di = fdi;
        } else {
            // unmatched close pair: product of the degree C + interval(d/D)
            // rules (up to degree 8 + 1), the SLP and DLP degrees apart
            double dc[3];
            for (int d = 0; d < 3; ++d) dc[d] = a.trial.center[3 * (int64_t)j + d] - a.test.center[3 * (int64_t)i + d];
            const double ratio = norm3(dc) / a.trial.size[j];
            const int cmax = (te.nc == 4 || re.nc == 4) ? 1 : 0;
            const int deg_s = cmax + (ratio < 11.0 / 10.0 ? 6 : (ratio < T_S1 ? 4 : (ratio < T_S0 ? 2 : 0)));
            const int deg_d =
                cmax + (ratio < 11.0 / 10.0 ? 8 : (ratio < T_NEAR ? 6 : (ratio < T_D1 ? 4 : (ratio < T_D0 ? 2 : 0))));
            const bool shared_pass = !do_s || !do_d || deg_s == deg_d;
            for (int pass = 0; pass < (shared_pass ? 1 : 2); ++pass) {
                const bool use_s = shared_pass ? do_s : pass == 0;
                const bool use_d = shared_pass ? do_d : pass == 1;
                const int deg = use_s ? deg_s : deg_d;
                const int npt = product_npts(te.nc, deg), npr = product_npts(re.nc, deg);
                for (int p = lane; p < npt * npr; p += 32) {
                    double xi, eta, wt, xr, er, wr;
                    product_point(te.nc, deg, p / npr, xi, eta, wt);
                    product_point(re.nc, deg, p % npr, xr, er, wr);
                    double x[3], y[3], n[3], nx[3];
                    ex(te, xi, eta, x);
                    enormal(te, xi, eta, nx);
                    ex(re, xr, er, y);
                    enormal(re, xr, er, n);
                    cd ks{0, 0}, kd{0, 0};
                    kp(x, y, n, norm3(n), use_s, use_d, ks, kd);
                    const double w = wt * norm3(nx) * wr;
                    if (use_s) {
                        sr += ks.re * w;
                        si += ks.im * w;
                    }
                    if (use_d) {
                        dr += kd.re * w;
                        di += kd.im * w;
                    }
                }
            }
        }
        sr = warp_sum(sr);
        si = warp_sum(si);
        dr = warp_sum(dr);
        di = warp_sum(di);
        if (lane == 0) {
            const int64_t off = (int64_t)(j - a.j0) * a.ld + i;
            if (do_s) store64(out_s + off, sr, si, a.alpha_re, a.alpha_im, a.accumulate);
            if (do_d) store64(out_d + off, dr, di, a.alpha_re, a.alpha_im, a.accumulate);
        }
    }
}

template <typename R, typename Out, int FAM>
static void launch_gal_ops(const GalArgs &a, dim3 grid, cudaStream_t s)
{
    if constexpr (FAM == FAM_HELMHOLTZ) {
        if (a.k_im != 0.0) {  // complex (lossy) wave number: separate instantiations
            if (a.ops == OP_SLP) k_galerkin_regular<R, Out, FAM, OP_SLP, false, true><<<grid, GAL_THREADS, 0, s>>>(a);
            else if (a.ops == OP_DLP) k_galerkin_regular<R, Out, FAM, OP_DLP, false, true><<<grid, GAL_THREADS, 0, s>>>(a);
            else k_galerkin_regular<R, Out, FAM, OP_SLP | OP_DLP, false, true><<<grid, GAL_THREADS, 0, s>>>(a);
            return;
        }
    }
    if constexpr (sizeof(R) == 4 && sizeof(Out) == 16) {  // into complex64: k_galerkin_regular2
        if (a.alpha_re == 1.0 && a.alpha_im == 0.0 && !a.accumulate) {
            if (a.ops == OP_SLP) k_galerkin_regular<R, Out, FAM, OP_SLP, true><<<grid, GAL_THREADS, 0, s>>>(a);
            else if (a.ops == OP_DLP) k_galerkin_regular<R, Out, FAM, OP_DLP, true><<<grid, GAL_THREADS, 0, s>>>(a);
            else k_galerkin_regular<R, Out, FAM, OP_SLP | OP_DLP, true><<<grid, GAL_THREADS, 0, s>>>(a);
            return;
        }
    }
    if (a.ops == OP_SLP) k_galerkin_regular<R, Out, FAM, OP_SLP><<<grid, GAL_THREADS, 0, s>>>(a);
    else if (a.ops == OP_DLP) k_galerkin_regular<R, Out, FAM, OP_DLP><<<grid, GAL_THREADS, 0, s>>>(a);
    else k_galerkin_regular<R, Out, FAM, OP_SLP | OP_DLP><<<grid, GAL_THREADS, 0, s>>>(a);
}

template <typename R, typename Out>
static void launch_gal_fam(const GalArgs &a, dim3 grid, cudaStream_t s)
{
    if (a.family == FAM_HELMHOLTZ) launch_gal_ops<R, Out, FAM_HELMHOLTZ>(a, grid, s);
    else launch_gal_ops<R, Out, FAM_LAPLACE>(a, grid, s);
}

cudaError_t launch_galerkin_regular(const GalArgs &a, cudaStream_t s)
{
    const int ncols = a.j1 - a.j0;
    if (a.test.n == 0 || ncols <= 0) return cudaSuccess;
    if (a.precision == 0 && a.dtype == 0 && a.k_im == 0.0 && a.alpha_re == 1.0 && a.alpha_im == 0.0 && !a.accumulate)
        return a.family == FAM_HELMHOLTZ ? launch_galerkin_regular2<FAM_HELMHOLTZ>(a, s)
                                         : launch_galerkin_regular2<FAM_LAPLACE>(a, s);
    dim3 grid((a.test.n + GAL_THREADS - 1) / GAL_THREADS);
    grid.y = column_blocks(grid.x, ncols, GAL_COLS);
    if (a.precision == 0) {
        if (a.dtype == 0) launch_gal_fam<float, float2>(a, grid, s);
        else launch_gal_fam<float, double2>(a, grid, s);
    } else {
        if (a.dtype == 0) launch_gal_fam<double, float2>(a, grid, s);
        else launch_gal_fam<double, double2>(a, grid, s);
    }
    return cudaGetLastError();
}

cudaError_t launch_galerkin_near(const GalArgs &a, const NearList &near, int extra, int64_t max_items, cudaStream_t s)
{
    if (max_items <= 0) return cudaSuccess;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (a.precision == 0 && a.k_im == 0.0 && !a.test.has_quad && !a.trial.has_quad)
        return a.dtype == 0 ? launch_galerkin_near_tria<float2>(a, near, extra, max_items, sms, s)
                            : launch_galerkin_near_tria<double2>(a, near, extra, max_items, sms, s);
    // two 4-warp blocks per SM: the kernel runs beside the regular one and
    // must leave it most of the register file
    const int64_t want = (max_items + GAL_WARPS - 1) / GAL_WARPS;
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(want, 2 * (int64_t)sms));
    if (a.family == FAM_HELMHOLTZ && a.k_im != 0.0) {
        if (a.dtype == 0) k_galerkin_near<float2, true><<<blocks, GAL_WARPS * 32, 0, s>>>(a, near, extra);
        else k_galerkin_near<double2, true><<<blocks, GAL_WARPS * 32, 0, s>>>(a, near, extra);
    } else {
        if (a.dtype == 0) k_galerkin_near<float2, false><<<blocks, GAL_WARPS * 32, 0, s>>>(a, near, extra);
        else k_galerkin_near<double2, false><<<blocks, GAL_WARPS * 32, 0, s>>>(a, near, extra);
    }
    return cudaGetLastError();
}

template <typename Out>
__global__ void k_add_mass(int n, const double *pts64, double are, double aim, Out *out, int64_t ld)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // w J of the element's one-point rule (parity 0, level 0): its area,
    // exact for flat triangles and bilinear quads
    const double area = pts64[8 * ((int64_t)i * 2 * SLOTS) + 3];
    Out o = out[(int64_t)i * ld + i];
    o.x += are * area;
    o.y += aim * area;
    out[(int64_t)i * ld + i] = o;
}

cudaError_t launch_add_mass(int n, const double *pts64, double are, double aim, int dtype, void *out, int64_t ld,
                            cudaStream_t s)
{
    if (n == 0) return cudaSuccess;
    const int t = 256, b = (n + t - 1) / t;
    if (dtype == 0) k_add_mass<float2><<<b, t, 0, s>>>(n, pts64, are, aim, (float2 *)out, ld);
    else k_add_mass<double2><<<b, t, 0, s>>>(n, pts64, are, aim, (double2 *)out, ld);
    return cudaGetLastError();
}

}  // namespace nihu
