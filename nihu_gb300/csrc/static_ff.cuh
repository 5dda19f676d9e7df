// The nearly singular static (Laplace) parts of a flat triangle in float-float
// arithmetic, for all four operators.
#pragma once

#include "ffloat.cuh"
#include "planar.cuh"

namespace nihu {

// The four operators of one pair in FP64
struct Acc4 {
    double sr = 0, si = 0, dr = 0, di = 0, tr = 0, ti = 0, hr = 0, hi = 0;
};

// which operators a launch evaluates (uniform over the launch)
struct OpSet {
    bool s, d, t, h;
};

// near_static4 in float-float arithmetic, for results that are stored in FP32
// (ffloat.cuh): the same points and formulas, with the plane coordinates, the
// side lines and the products of the normals in FP64 (about 120 FP64
// instructions per pair), everything per angular point in float-float.
//
// Per side, with the foot point's distance s = |c1 x l| from the side's line
// and the corners at u1, u2 along it, psi = theta - t0 runs over
// [atan2(u1, s), atan2(u2, s)] (measured from the foot towards c2), and with
// t = s^2 + z^2 cos^2 psi, r = sqrt(t) / cos psi the integrands need neither a
// division nor an angle per point:
//   HSP   s^2/z (A cos psi + B sin psi) t^{-3/2},  A = s (n.f) - n_2 z, B = s (n.l)
//   DLPt  -(A cos psi + B sin psi) / sqrt(t) + (n.f cos psi + n.l sin psi)
//         log((s + sqrt t) / cos psi) - n_2 sgn(z)
// (f the foot direction, l the side's).  DLPt's last term and the 1 of DLP's
// 1 - |z|/r are constant: they take the angle that the sides make up, 2 pi or 0,
// exactly, so that a surface that is nearly flat keeps its small DLP and DLPt
// entries (a plate folded by 1e-7: error 3.5e-5 of the largest entry when they were
// summed, 1e-7 now).  The rule is symmetric about the
// side's middle angle, so one sin / cos of h x serves the two points +-x.
// cos psi never falls below s / max(rho_1, rho_2), which the clamp keeps
// against rounding when x0 lies on a side's line.  Lengths are scaled by a
// power of two near the element's size, so that no product leaves FP32 range.
//
// About 18 000 FP32 instructions per pair in place of 8 500 FP64 ones (GB300:
// 128 against 2 per SM and cycle).  Bound by the latency of one thread's chain: the
// kernels that call it issue in 46% of the cycles with twelve warps an SM (pair
// lists; their FP64 set-up and self terms keep that pipe active in 65%) and in
// 34% with eight (the Burton-Miller system).  On the sphere of
// 20480 triangles the singular kernel of the Burton-Miller system, beside the
// regular one, went from 4.04 to 0.84 ms and the near field list of 5.1 M
// pairs from 3.53 to 0.80 ms; the complex64 entries' error against 64 bits
// stays 2.6e-8 and 2.4e-8.  Returns false (nothing added) where the HSP's 1/z
// cancels between the sides by more than three digits: |z| small against the
// in-plane part of nx times the side, a folded pair whose collocation point
// nearly lies in the element's plane; those take FP64.
template <int G = 1, int SIDES = 3>
__device__ inline bool near_static4_ff(const double *__restrict__ frame, const double c0[3], const double x0[3],
                                       const double nxg[3], OpSet ops, Acc4 &a, const Lanes<G> &g = Lanes<G>())
{
    const double dv0 = c0[0] - x0[0], dv1 = c0[1] - x0[1], dv2 = c0[2] - x0[2];
    const double u0 = frame[0] * dv0 + frame[1] * dv1 + frame[2] * dv2;
    const double v0 = frame[3] * dv0 + frame[4] * dv1 + frame[5] * dv2;
    const double z = -(frame[6] * dv0 + frame[7] * dv1 + frame[8] * dv2);
    const double n0 = dot3(frame, nxg), n1 = dot3(frame + 3, nxg), n2 = dot3(frame + 6, nxg);
    const bool in_plane = !(fabs(z) > 1e-12);
    const float len0 = (float)frame[11];  // first side: along the first axis
    if (ops.h && !in_plane && 1e3f * (float)fabs(z) < (float)(fabs(n0) + fabs(n1)) * len0) return false;
    const int ex2 = ((__float_as_int(len0) >> 23) & 255) - 127;
    const float sc = __int_as_float((127 - ex2) << 23), isc = __int_as_float((127 + ex2) << 23);  // 2^-+ex2
    const ff zf = ff_scale(ff_from(fabs(z)), sc), z2 = ff_mul(zf, zf);
    const bool six = ops.s || ops.d || ops.t;
    double s_sum = 0.0, d_sum = 0.0, t_sum = 0.0, h_sum = 0.0, angle = 0.0;
#pragma unroll 1
    for (int sd = g.lane; sd < SIDES; sd += G) {
        const int e1 = sd, e2 = sd == SIDES - 1 ? 0 : sd + 1;
        const double a0 = frame[9 + 2 * e1], a1 = frame[10 + 2 * e1], b0 = frame[9 + 2 * e2], b1 = frame[10 + 2 * e2];
        const double d0 = b0 - a0, d1 = b1 - a1, il = rsqrt(d0 * d0 + d1 * d1);
        const double l0 = d0 * il, l1 = d1 * il;
        const double p0 = a0 + u0, p1 = a1 + v0;
        const double sv = p0 * l1 - p1 * l0;  // signed distance of the line
        const double u1 = p0 * l0 + p1 * l1, u2 = (b0 + u0) * l0 + (b1 + v0) * l1;
        const double sgn = sv < 0.0 ? -1.0 : 1.0, sa = fabs(sv);
        const double na = sgn * (n0 * l1 - n1 * l0), nb = n0 * l0 + n1 * l1;  // n.f and n.l
        const ff u1f = ff_scale(ff_from(u1), sc), u2f = ff_scale(ff_from(u2), sc);
        ff s = ff_scale(ff_from(sa), sc);
        s.h = fmaxf(s.h, 1e-14f);
        const ff A = ff_scale(ff_from(sa * na - n2 * z), sc), B = ff_scale(ff_from(sa * nb), sc);
        const ff s2 = ff_mul(s, s);
        const float cmin = s.h * rsqrtf(fmaxf(u1f.h * u1f.h, u2f.h * u2f.h) + s2.h);
        const ff q1 = ff_angle(u1f, s), q2 = ff_angle(u2f, s);
        const ff mid = ff_scale(ff_add(q1, q2), 0.5f), hw = ff_scale(ff_sub(q2, q1), 0.5f);
        ff sm, cm;
        ff_sincos(mid, sm, cm);
        // f(cos psi, sin psi) at the points +-x, weights w
        auto pair_points = [&](ff x, auto &&f) {
            ff sh, ch;
            ff_sincos(ff_mul(hw, x), sh, ch);
            const ff cc = ff_mul(cm, ch), ss = ff_mul(sm, sh), scp = ff_mul(sm, ch), csp = ff_mul(cm, sh);
            f(ff_sub(cc, ss), ff_add(scp, csp));
            f(ff_add(cc, ss), ff_sub(scp, csp));
        };
        auto clamp_cos = [&](ff c) { return c.h < cmin ? ff{cmin, 0.0f} : c; };
        const double wj = sgn * ff_double(hw);  // half the side's angle in theta
        if (six) {
            const ff naf = ff_from(na), nbf = ff_from(nb);
            ff sl{0.0f, 0.0f}, sdl{0.0f, 0.0f}, st{0.0f, 0.0f};
#pragma unroll 1
            for (int q = 0; q < 3; ++q) {
                const ff w{GAUSS6_FF.wh[q], GAUSS6_FF.wl[q]};
                pair_points(ff{GAUSS6_FF.xh[q], GAUSS6_FF.xl[q]}, [&](ff c, ff sn) {
                    c = clamp_cos(c);
                    const ff t = ff_add(s2, ff_mul(z2, ff_mul(c, c)));
                    const ff rs = ff_rsqrt(t), rt = ff_mul(t, rs);
                    const ff ic = ff_recip(c);
                    const ff zc = ff_mul(zf, c);
                    if (ops.s) sl = ff_add(sl, ff_mul(w, ff_mul(ff_sub(rt, zc), ic)));
                    if (ops.d) sdl = ff_add(sdl, ff_mul(w, ff_mul(zc, rs)));
                    if (ops.t) {
                        const ff g = ff_add(ff_mul(naf, c), ff_mul(nbf, sn));
                        const ff v = ff_mul(ff_add(ff_mul(A, c), ff_mul(B, sn)), rs);
                        const ff lg = ff_log(ff_mul(ff_add(s, rt), ic), ex2);
                        st = ff_add(st, ff_mul(w, ff_sub(ff_mul(g, lg), v)));
                    }
                });
            }
            angle += wj;
            s_sum += wj * ff_double(sl);
            d_sum -= wj * ff_double(sdl);
            t_sum += wj * ff_double(st);
        }
        if (ops.h) {
            ff sum{0.0f, 0.0f};
            auto point = [&](ff w, ff c, ff sn) {
                c = clamp_cos(c);
                if (in_plane) {
                    sum = ff_add(sum, ff_mul(w, c));
                } else {
                    const ff t = ff_add(s2, ff_mul(z2, ff_mul(c, c)));
                    const ff rs = ff_rsqrt(t);
                    // (r_vec.nx / r) (s / sqrt t)^2: both factors stay within 1
                    const ff v = ff_mul(ff_add(ff_mul(A, c), ff_mul(B, sn)), rs), sr = ff_mul(s, rs);
                    sum = ff_add(sum, ff_mul(ff_mul(w, v), ff_mul(sr, sr)));
                }
            };
#pragma unroll 1
            for (int q = 0; q < 10; ++q) {
                const ff w{GAUSS21_FF.wh[q], GAUSS21_FF.wl[q]};
                pair_points(ff{GAUSS21_FF.xh[q], GAUSS21_FF.xl[q]}, [&](ff c, ff sn) { point(w, c, sn); });
            }
            point(ff{GAUSS21_FF.wh[10], GAUSS21_FF.wl[10]}, cm, sm);
            // in the plane: -n_2 cos psi / s
            if (in_plane) h_sum -= wj * n2 * ff_double(sum) / ff_double(s);
            else h_sum += wj * ff_double(sum);
        }
    }
    if constexpr (G > 1) {
        s_sum = g.sum(s_sum);
        d_sum = g.sum(d_sum);
        t_sum = g.sum(t_sum);
        angle = g.sum(angle);
        h_sum = g.sum(h_sum);
    }
    // the constants of DLP and DLPt times the angle that the sides make up: a
    // multiple of 2 pi but for rounding, unless the foot is a corner
    const double turns = rint(angle * (1.0 / PI));
    const double full = fabs(angle - turns * PI) < 1e-9 ? turns * (2.0 * PI) : 2.0 * angle;
    const double sg = (0.0 < z) - (z < 0.0);
    if (ops.d) d_sum += full;
    if (ops.t) t_sum -= n2 * sg * full;
    a.sr += s_sum * (INV_FOUR_PI * isc);
    a.dr += sg * d_sum * INV_FOUR_PI;
    a.tr += t_sum * INV_FOUR_PI;
    if (ops.h) a.hr += (in_plane ? h_sum : h_sum / (z * (double)sc)) * (INV_FOUR_PI * sc);
    return true;
}

// near_static on a flat quadrilateral, for results that are stored in FP32: its
// plane frame in FP64 (DevMesh::frame's layout, four corners), the rest as above
template <int G = 1>
static __device__ __noinline__ void near_static_quad_ff(const Elem64 &e, const double x0[3], bool do_s, bool do_d, Acc &a,
                                                        const Lanes<G> &g = Lanes<G>())
{
    double loc[4][2], z, T[3][3], frame[17];
    plane_local_frame(e, x0, loc, z, T);
    for (int d = 0; d < 3; ++d) {
        frame[d] = T[0][d];
        frame[3 + d] = T[1][d];
        frame[6 + d] = T[2][d];
    }
    for (int c = 0; c < 4; ++c) {
        frame[9 + 2 * c] = loc[c][0] - loc[0][0];
        frame[10 + 2 * c] = loc[c][1] - loc[0][1];
    }
    Acc4 st;
    near_static4_ff<G, 4>(frame, e.c[0], x0, x0, OpSet{do_s, do_d, false, false}, st, g);
    if (do_s) a.sr += st.sr;
    if (do_d) a.dr += st.dr;
}

}  // namespace nihu
