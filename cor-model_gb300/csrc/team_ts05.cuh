// team_ts05.cuh -- the TS05 field (ts05.cuh) cut into tasks for a team block
// (team.cuh).
//
// The model's cost is in a few functions it evaluates several times at
// different arguments (cones, ring-current potentials, quadrupole radial and
// polar functions: 500 to 1,500 FP64 warp instructions each): every call is a
// task.
//   phase 1: the four 3 x 3 shields, the magnetopause field, the magnetopause
//            distance, and what the calls of phase 2 take;
//   phase 2: cones (4), partial-ring (4) and symmetric-ring (4) potentials,
//            quadrupole functions (3 + 3), tail disks (2), the sines and
//            cosines of the tail's shields (20);
//   phase 3: the tail shields' 50 exponential terms, and the fields made of
//            phase 2's values;
//   phase 4: the tail shields' sums, in order.
// The functions are ts05.cuh's own, called with the same arguments, and what
// is left between them keeps its expressions and roundings, so results do
// not move by a bit (tests/test_gpu_team.py).
#pragma once

#include "ts05.cuh"

namespace cor {

// The position-independent constants again, for per-lane indices.
static __device__ TS05Tables g_ts05;

struct TS05Slot {
    double x, y, z;               // GSM [R_E] x xappa
    double X, Y, Z;               // GSM [R_E]
    double sigma;
    double w[6];                  // warped: yy, zz, sf, cf, cphi, sphi
    double bk[2][10];             // birk_1n2: xs, ys, zs, cphics, sphics, dpsp, dpsr, rho, cphic, sphic
    double sy[2][16];             // symm: R, r2, sint, cost, x, y, z, stp, stm, and the calls' R and angles
    double qd[16];                // prc_quad
    double cone[4][3];
    double ap[2][4];
    double br[3], bt[3];
    double disk[2][3];
    double sc[20][2];
    double ex[50][3];
    double h5[2][3];
    double sh[4][3];              // shields R11, R21, symmetric and partial ring
    double cf[3];
    double f[2][3];               // birk_1n2 of R11 and R21
    double rc[2][3];              // symmetric, partial ring
    double quad[3];
    const TS05Cond* c;
};

// ---- before phase 1 (the quad) ---------------------------------------------
__device__ __forceinline__ void ts05_slot_start(TS05Slot& s, const TS05Cond& c, const Vec3 X) {
    s.X = X.x;
    s.Y = X.y;
    s.Z = X.z;
    s.x = X.x * c.xappa;
    s.y = X.y * c.xappa;
    s.z = X.z * c.xappa;
    s.c = &c;
}

// ---- phase 1 ---------------------------------------------------------------
static __device__ __noinline__ void ts05_task_main(TS05Slot& s) {
    const TS05Cond& c = *s.c;
    const double x = s.X, y = s.Y, z = s.Z;
    double xmxm = c.am + x - c.x0;
    if (xmxm < 0) xmxm = 0.;
    const double axx0 = xmxm * xmxm;
    const double rho2 = __dadd_rn(__dmul_rn(y, y), __dmul_rn(z, z));   // ts05_field's squares have other uses
    const double aro = (c.asq + rho2) + axx0;
    s.sigma = sqrt(div_r(aro + sqrt(aro * aro - c.four_asq * axx0), c.two_asq, c.r_two_asq));
}

// ts05_warped up to its disks and shields.
static __device__ __noinline__ void ts05_task_warp(TS05Slot& s) {
    const double y = s.y, z = s.z;
    const double rho2 = y * y + z * z;
    const double rho = sqrt(rho2);
    double phi = 0., cphi = 1., sphi = 0.;
    if (y != 0. || z != 0.) {
        phi = ol_atan2(z, y);
        const double rr = 1. / rho;
        cphi = div_r(y, rho, rr);
        sphi = div_r(z, rho, rr);
    }
    double sf, cf;
    ol_sincos(phi, &sf, &cf);
    s.w[0] = rho * cf;
    s.w[1] = rho * sf;
    s.w[2] = sf;
    s.w[3] = cf;
    s.w[4] = cphi;
    s.w[5] = sphi;
}

// ts05_birk_1n2 up to its cones, numb = k + 1.
static __device__ __noinline__ void ts05_task_birk(TS05Slot& s, const int k) {
    const double xkappa = k == 0 ? s.c->xk1 : s.c->xk2;
    const double dphi = k == 0 ? 0.055 : 0.030;
    const double xs_ = s.x * xkappa, ys = s.y * xkappa, zs_ = s.z * xkappa;
    const double xs2 = xs_ * xs_, zs2 = zs_ * zs_;
    const double rho = sqrt(xs2 + zs2);
    const double rho2 = rho * rho;
    double phi = 0.;
    if (xs_ != 0. || zs_ != 0.) phi = ol_atan2(-zs_, xs_);
    double sphic, cphic;
    ol_sincos(phi, &sphic, &cphic);
    const double r02 = 49. + rho2;
    const double brack = dphi + 0.5 * 49. / 50. * (rho2 - 1.) / r02;
    const double phis = phi - brack * sphic;
    const double dpsp = 1. - brack * cphic;
    const double dpsr = -2. * 0.5 * 49. * rho / (r02 * r02) * sphic;
    double sphics, cphics;
    ol_sincos(phis, &sphics, &cphics);
    double* o = s.bk[k];
    o[0] = rho * cphics;
    o[1] = ys;
    o[2] = -rho * sphics;
    o[3] = cphics;
    o[4] = sphics;
    o[5] = dpsp;
    o[6] = dpsr;
    o[7] = rho;
    o[8] = cphic;
    o[9] = sphic;
}

// ts05_symm up to its potentials: k = 0 symmetric, 1 partial ring.
static __device__ __noinline__ void ts05_task_symm(TS05Slot& s, const int k) {
    constexpr double D = 1.E-4;
    const double sc = k == 0 ? s.c->scsy : s.c->scpr, rs = 1. / sc;
    const double x = div_r(s.x, sc, rs), y = div_r(s.y, sc, rs), z = div_r(s.z, sc, rs);
    const double rho2 = __fma_rn(x, x, __dmul_rn(y, y));
    const double r2 = __fma_rn(z, z, rho2);
    const double R = sqrt(r2);
    const double rr = 1. / R;
    const double sint = div_r(sqrt(rho2), R, rr);
    const double cost = div_r(z, R, rr);
    double* o = s.sy[k];
    o[0] = R;
    o[1] = r2;
    o[2] = sint;
    o[3] = cost;
    o[4] = x;
    o[5] = y;
    o[6] = z;
    if (!(sint < 1.E-2)) {
        const double th = ol_atan2(sint, cost);
        double stp, ctp, stm, ctm;
        ol_sincos(th + D, &stp, &ctp);
        ol_sincos(th - D, &stm, &ctm);
        o[7] = stp;
        o[8] = ctp;
        o[9] = stm;
        o[10] = ctm;
    }
}

// ts05_prc_quad up to its functions.
static __device__ __noinline__ void ts05_task_quad(TS05Slot& s) {
    constexpr double D = 1.E-4, DS = 1.E-2, DC = 0.99994999875;
    const double rpr = 1. / s.c->scpr, scpr = s.c->scpr;
    const double xta = div_r(s.x, scpr, rpr), yta = div_r(s.y, scpr, rpr), zta = div_r(s.z, scpr, rpr);
    const double cp = g_ts05.cphi, sp = g_ts05.sphi;
    const double x = __fma_rn(xta, cp, -__dmul_rn(yta, sp)), y = __fma_rn(yta, cp, __dmul_rn(xta, sp)), z = zta;
    const double rho2 = __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y));   // the squares have other uses there
    const double R = sqrt(__fma_rn(z, z, rho2));
    const double rho = sqrt(rho2);
    const double rr = 1. / R;
    const double sint = div_r(rho, R, rr), cost = div_r(z, R, rr);
    const bool off = sint > DS;
    const double st = off ? sint : DS, ct = off ? cost : z < 0. ? -DC : DC;
    const double th = ol_atan2(st, ct);
    double stp, ctp, stm, ctm;
    ol_sincos(th + D, &stp, &ctp);
    ol_sincos(th - D, &stm, &ctm);
    double* o = s.qd;
    o[0] = x;
    o[1] = y;
    o[2] = z;
    o[3] = R;
    o[4] = rho;
    o[5] = sint;
    o[6] = cost;
    o[7] = st;
    o[8] = ct;
    o[9] = stp;
    o[10] = ctp;
    o[11] = stm;
    o[12] = ctm;
}

__device__ __forceinline__ void put3(double* o, const Vec3 v) {
    o[0] = v.x;
    o[1] = v.y;
    o[2] = v.z;
}

__device__ __forceinline__ void ts05_task_shield(TS05Slot& s, const int k) {
    const TS05Cond& c = *s.c;
    const bool rc = k >= 2;
    const double* P = rc ? g_ts05.rc_p[k - 2] : g_ts05.bs_p[k];
    const double* R = rc ? g_ts05.rc_r[k - 2] : g_ts05.bs_r[k];
    const double* Q = rc ? g_ts05.rc_sq[k - 2] : g_ts05.bs_sq[k];
    const double* amp = k == 0 ? c.amp11 : k == 1 ? c.amp21 : k == 2 ? c.amp_sy : c.amp_pr;
    put3(s.sh[k], ts05_shield3(P, R, Q, amp, k == 2 ? c.fac_sy : k == 3 ? c.fac_pr : 1., rc, s.x, s.y, s.z));
}

// ---- phase 2 ---------------------------------------------------------------
// Cone k: R11 north, south, R21 north, south.
__device__ __forceinline__ void ts05_task_cone(TS05Slot& s, const int k) {
    const int numb = k >> 1;
    const double* b = s.bk[numb];
    const double sg = (k & 1) ? -1. : 1.;
    put3(s.cone[k], ts05_one_cone(numb == 0 ? c_ts05_a11 : c_ts05_a21, g_ts05.rs_sq[numb], b[0], sg * b[1], sg * b[2],
                                  numb == 0 ? 0.06 : 0.09));
}

// Potential j of ts05_symm's four (three on the axis).
__device__ __forceinline__ void ts05_task_ap(TS05Slot& s, const int k, const int j) {
    constexpr double DS = 1.E-2, DC = 0.99994999875, D = 1.E-4;
    const double* o = s.sy[k];
    const double R = o[0], rp = R + D, rm = R - D;
    const bool axis = o[2] < DS;
    if (axis && j == 3) return;
    const double r = axis ? (j == 0 ? R : j == 1 ? rp : rm) : (j < 2 ? R : j == 2 ? rm : rp);
    const double st = axis ? DS : j == 0 ? o[7] : j == 1 ? o[9] : o[2];
    const double ct = axis ? DC : j == 0 ? o[8] : j == 1 ? o[10] : o[3];
    s.ap[k][j] = k == 0 ? ts05_ap(r, st, ct) : ts05_apprc(r, st, ct);
}

__device__ __forceinline__ void ts05_task_br(TS05Slot& s, const int j) {
    constexpr double D = 1.E-4;
    const double R = s.qd[3];
    s.br[j] = ts05_br_prc_q(j == 0 ? R : j == 1 ? R + D : R - D, s.qd[7], s.qd[8]);
}

__device__ __forceinline__ void ts05_task_bt(TS05Slot& s, const int j) {
    s.bt[j] = ts05_bt_prc_q(s.qd[3], s.qd[j == 0 ? 7 : j == 1 ? 9 : 11], s.qd[j == 0 ? 8 : j == 1 ? 10 : 12]);
}

__device__ __forceinline__ void ts05_task_disk(TS05Slot& s, const int k) {
    const TS05Cond& c = *s.c;
    const double f = k == 0 ? 1.1 : 0.25;
    const double x = k == 0 ? __fma_rn(s.x - 6. - c.dx1, 1.1, 1.2) : __fma_rn(s.x - 4. - c.dx2, 0.25, -9.);
    put3(s.disk[k], ts05_taildisk(c.d * f, k == 0 ? 1. : 0., x, s.w[0] * f, s.w[1] * f));
}

// Sines and cosines of the tail shields: table t, 0-4 z, 5-9 y.
__device__ __forceinline__ void ts05_task_sc(TS05Slot& s, const int i) {
    const int t = i / 10, k = i % 10;
    const SinCos r = ol_sincos_v(k < 5 ? s.w[1] * g_ts05.s5_rr[t][k] : s.w[0] * g_ts05.s5_rp[t][k - 5]);
    s.sc[i][0] = r.s;
    s.sc[i][1] = r.c;
}

// ---- phase 3 ---------------------------------------------------------------
__device__ __forceinline__ void ts05_task_exp(TS05Slot& s, const int j) {
    const int t = j / 25, l = j % 25, i = l / 5, k = l % 5;
    const double* zs = s.sc[10 * t + k];
    const double* ys = s.sc[10 * t + 5 + i];
    const double sq = g_ts05.s5_sq[t][l];
    const double e = ol_exp(s.x * sq);
    s.ex[j][0] = -sq * e * ys[1] * zs[0];
    s.ex[j][1] = g_ts05.s5_rp[t][i] * e * ys[0] * zs[0];
    s.ex[j][2] = -g_ts05.s5_rr[t][k] * e * ys[1] * zs[1];
}

// ts05_birk_1n2's end.
static __device__ __noinline__ void ts05_end_birk(TS05Slot& s, const int k) {
    const double xkappa = k == 0 ? s.c->xk1 : s.c->xk2;
    const double* b = s.bk[k];
    const double cphics = b[3], sphics = b[4], dpsp = b[5], dpsr = b[6], rho = b[7], cphic = b[8], sphic = b[9];
    const double *bn = s.cone[2 * k], *bs = s.cone[2 * k + 1];
    const double bxs = bn[0] - bs[0], byas = bn[1] + bs[1], bzs = bn[2] + bs[2];
    const double brhoas = bxs * cphics - bzs * sphics;
    const double bphias = -bxs * sphics - bzs * cphics;
    const double brho_s = brhoas * dpsp * xkappa;
    const double bphi_s = (bphias - rho * (brhoas * dpsr)) * xkappa;
    const double by_s = byas * dpsp * xkappa;
    put3(s.f[k], {brho_s * cphic - bphi_s * sphic, by_s, -brho_s * sphic - bphi_s * cphic});
}

// ts05_symm's end.
static __device__ __noinline__ void ts05_end_symm(TS05Slot& s, const int k) {
    constexpr double DS = 1.E-2, D = 1.E-4, DRD = 5E3;
    const double* o = s.sy[k];
    const double R = o[0], r2 = o[1], sint = o[2], cost = o[3], x = o[4], y = o[5], z = o[6];
    const double *a = s.ap[k];
    const double rp = R + D, rm = R - D;
    const double rr = 1. / R;
    double fxy, bz;
    if (sint < DS) {
        const double A = a[0] / DS;
        const double dardr = __dmul_rn(__fma_rn(-rm, a[2], __dmul_rn(rp, a[1])), DRD);
        fxy = z * __dadd_rn(2. * A, -dardr) / (R * r2);
        bz = div_r(__fma_rn(2. * A, cost * cost, __dmul_rn(dardr, sint * sint)), R, rr);
    } else {
        const double stp = o[7], stm = o[9];
        const double br = __dmul_rn(__fma_rn(-stm, a[1], __dmul_rn(stp, a[0])) / (R * sint), DRD);
        const double bt = __dmul_rn(div_r(__fma_rn(-rp, a[3], __dmul_rn(rm, a[2])), R, rr), DRD);
        fxy = div_r(__dadd_rn(br, __dmul_rn(bt, cost) / sint), R, rr);
        bz = __fma_rn(br, cost, -__dmul_rn(bt, sint));
    }
    put3(s.rc[k], {fxy * x, fxy * y, bz});
}

// ts05_prc_quad's end.
static __device__ __noinline__ void ts05_end_quad(TS05Slot& s) {
    constexpr double DD = 2.E-4, DS = 1.E-2;
    const double* o = s.qd;
    const double x = o[0], y = o[1], R = o[3], rho = o[4], sint = o[5], cost = o[6];
    const double br = s.br[0], bt = s.bt[0];
    const double dbrr = div_c(s.br[1] - s.br[2], DD, 1. / DD);
    const double dbtt = div_c(s.bt[1] - s.bt[2], DD, 1. / DD);
    Vec3 b;
    if (sint > DS) {
        const double rrho = 1. / rho;
        const double cphi = div_r(x, rho, rrho), sphi = div_r(y, rho, rrho);
        const double w = __fma_rn(R, dbrr, br) + dbtt;
        b = {__fma_rn(cost, bt, __dmul_rn(sint, __fma_rn(w, __dmul_rn(sphi, sphi), br))), -sint * sphi * cphi * w,
             __fma_rn(br, cost, -__dmul_rn(bt, sint)) * cphi};
    } else {
        const double st = DS;
        const double rr = 1. / R;
        const double fcxy = __fma_rn(R, dbrr, dbtt);
        const double rst = R * st;
        const double rst2 = rst * rst;
        const double y2 = y * y;
        const double rr2 = 1. / rst2;
        const double w = __fma_rn(br, __fma_rn(x, x, 2. * y2), __dmul_rn(fcxy, y2));
        b = {__fma_rn(bt, cost, div_r(w, rst2, rr2)), div_r(-(br + fcxy) * x * y, rst2, rr2),
             div_r(__dadd_rn(__dmul_rn(br, cost) / st, -bt) * x, R, rr)};
    }
    put3(s.quad, b);
}

// ---- phase 4 ---------------------------------------------------------------
__device__ __forceinline__ void ts05_sum5(TS05Slot& s, const int t, const int c) {
    const double* coef = t == 0 ? s.c->coef1 : s.c->coef2;
    double h = 0.;
    for (int l = 0; l < 25; l++) h = h + coef[l] * s.ex[25 * t + l][c];
    s.h5[t][c] = h;
}

// ts05_warped's end, table t.
static __device__ __noinline__ Vec3 ts05_end_warp(const TS05Slot& s, const int t) {
    const double sf = s.w[2], cf = s.w[3], cphi = s.w[4], sphi = s.w[5];
    const double *f = s.disk[t], *h = s.h5[t];
    const Vec3 u = {f[0] + h[0], f[1] + h[1], f[2] + h[2]};
    const double br = u.y * cf + u.z * sf;
    const double bp = -u.y * sf + u.z * cf;
    return {u.x, br * cphi - bp * sphi, br * sphi + bp * cphi};
}

// ts05_field's sum inside the magnetopause.
static __device__ __noinline__ Vec3 ts05_slot_inside(const TS05Slot& s) {
    const TS05Cond& c = *s.c;
    const Vec3 t1 = ts05_end_warp(s, 0), t2 = ts05_end_warp(s, 1);
    const Vec3 cf = {s.cf[0], s.cf[1], s.cf[2]};
    const Vec3 r11 = {s.f[0][0] + s.sh[0][0], s.f[0][1] + s.sh[0][1], s.f[0][2] + s.sh[0][2]};
    const Vec3 r21 = {s.f[1][0] + s.sh[1][0], s.f[1][1] + s.sh[1][1], s.f[1][2] + s.sh[1][2]};
    const double cp = g_ts05.cphi, sp = g_ts05.sphi;
    const Vec3 bq = {s.quad[0], s.quad[1], s.quad[2]};
    const double bxq = bq.x * cp + bq.y * sp;
    const double byq = -bq.x * sp + bq.y * cp;
    const Vec3 src = {s.rc[0][0] + s.sh[2][0], s.rc[0][1] + s.sh[2][1], s.rc[0][2] + s.sh[2][2]};
    const Vec3 prc = {(s.rc[1][0] + bxq) + s.sh[3][0], (s.rc[1][1] + byq) + s.sh[3][1],
                      (s.rc[1][2] + bq.z) + s.sh[3][2]};
    constexpr double A19 = 0.452536;
    const double bbx = 1.00000 * (cf.x * c.xappa3) + c.tamp1 * t1.x + c.tamp2 * t2.x + c.a_src * src.x +
                       c.a_prc * prc.x + c.a_r11 * r11.x + c.a_r21 * r21.x + A19 * 0.;
    const double bby = 1.00000 * (cf.y * c.xappa3) + c.tamp1 * t1.y + c.tamp2 * t2.y + c.a_src * src.y +
                       c.a_prc * prc.y + c.a_r11 * r11.y + c.a_r21 * r21.y + A19 * c.byimf;
    const double bbz = 1.00000 * (cf.z * c.xappa3) + c.tamp1 * t1.z + c.tamp2 * t2.z + c.a_src * src.z +
                       c.a_prc * prc.z + c.a_r11 * r11.z + c.a_r21 * r21.z + A19 * c.bzimf;
    return {bbx, bby, bbz};
}

// ts05_field's end (the quad), rounded as the compiler rounds it there.
static __device__ __noinline__ Vec3 ts05_slot_end(const TS05Slot& s) {
    const TS05Cond& c = *s.c;
    const double x = s.X, y = s.Y, z = s.Z, sigma = s.sigma;
    if (sigma < 1.1960 - 0.005) return ts05_slot_inside(s);
    const double oimfy = c.oimfy_k, oimfz = c.oimfz_k;
    const double u = __dmul_rn(z, z);
    const double pt = __fma_rn(x, x, __dmul_rn(y, y));
    const double sq = sqrt(__dadd_rn(pt, u));
    const double q = 30115. / (sq * sq * sq * sq * sq);
    const double qx = q * 3. * z * x, qya = q * -3. * z, qzb = __dadd_rn(pt, -2. * u);   // q.y = qya y, q.z = q qzb
    if (!(sigma < 1.1960 + 0.005)) return {-qx, __fma_rn(-qya, y, oimfy), __fma_rn(-q, qzb, oimfz)};
    const Vec3 f = ts05_slot_inside(s);
    const double fint = 0.5 * (1. - div_c(sigma - 1.1960, 0.005, 1. / 0.005));
    const double fext = 0.5 * (1. + div_c(sigma - 1.1960, 0.005, 1. / 0.005));
    const double my = __fma_rn(oimfy, fext, __dmul_rn(__fma_rn(qya, y, f.y), fint));
    const double mz = __fma_rn(oimfz, fext, __dmul_rn(__fma_rn(q, qzb, f.z), fint));
    return {__fma_rn(__dadd_rn(f.x, qx), fint, -qx), __fma_rn(-qya, y, my), __fma_rn(-q, qzb, mz)};
}

}  // namespace cor
