// team_t96.cuh -- the T96 field (t96.cuh) cut into tasks for a team block
// (team.cuh).
//
// One lane's T96 evaluation is about 8,000 FP64 warp instructions.  Its parts
// are sums of independent terms of a few forms; each form is a kind of task
// here, taken by any lane of the block:
//   phase 1: the Region-1 band, xksi, the magnetopause distance, Bessel terms
//            (6), ring and tail loop terms (6), tail line currents (3), the
//            sines and cosines of the shields (36);
//   phase 2: exponential terms of the shields (56), dipoles of the conical
//            basis (46) and of the loops basis (21), current circles (up to
//            14), the conical harmonics by order (5 each), the Region-2 sheet
//            by component;
//   phase 3: every sum in its order, one lane per sum and component.
// The expressions, and what is rounded before it is added, are t96.cuh's: a
// term whose last product the one-lane code adds with one rounding is kept as
// two factors, so results do not move by a bit (tests/test_gpu_team.py).
// Tables that tasks index per lane sit in global memory (L1): constant memory
// serves one address at a time.
#pragma once

#include "t96.cuh"

namespace cor {

// The position-independent constants again, for per-lane indices.
static __device__ T96Tables g_t96;

constexpr int kT96Exp = 56, kT96Sc = 36, kT96Dip = 46, kT96Lop = 21;

// Shield terms: tables ARC, ATAIL2, ATAIL3 (9 each, 3 i + k), birk1shld (16,
// 4 i + k), birk2shl (4, 2 i + k), intercon (9, 3 i + k).  amp multiplies the
// term; the y and z factors divide by yc, zc (or, where that is 0, multiply by
// yr, zr); ys, zs are the sine/cosine tasks of their arguments.
static __device__ const double g_e_amp[56] = {
    -3.087699646 + 3.516259114, 18.81380577 + -13.95772338, -5.497076303 + 0.1712890838,
    2.392629189 + -2.728020808, -14.79349936 + 11.08738083, 4.388174084 + 0.2492163197E-01,
    0.7030375685 + -.7966023165, -3.835041334 + 2.642228681, -0.2405352424 + -0.7297705678,
    0.8747515218 + -0.9116821411, 2.209365387 + -2.159059518, -7.059828867 + 5.924671028,
    -1.916935691 + 1.996707344, -3.877101873 + 3.947666061, 11.38715899 + -8.343210833,
    1.194109867 + -1.244316975, 3.73895491 + -4.406522465, -20.66884863 + 3.020952989,
    -19091.95061 + -3011.613928, 20582.16203 + 4242.918430, -2377.091102 + -1504.820043,
    19884.04650 + 2725.150544, -21389.04845 + -3990.475093, 2401.610097 + 1548.171792,
    -946.5493963 + 490.1528941, 986.9156625 + -489.3265930, -67.99278499 + 8.711175710,
    1.174198045 + -1.463820502, 4.840161537 + -3.674506864, 82.18368896 + -94.94071588,
    -4122.331796 + 4670.278676, -21.54975037 + 26.72661293, -72.81365728 + 44.09887902,
    40.08073706 + -51.23563510, 1955.348537 + -1940.971550, 794.0496433 + -982.2441344,
    1889.837171 + -558.9779727, -1260.543238 + 1260.063802, -293.5942373 + 344.7250789,
    -773.7002492 + 957.0094135, -1824.143669 + 520.7994379, 1192.484774 + -1192.184565,
    89.15537624 + -98.52042999, -111.6371348 + 124.5402702, 110.3735178 + -122.0095905,
    111.9448247 + -129.1957743, -110.7586562 + 126.5649012, -8.411078731, 5932254.951, -9073284.93,
    -11.68794634, 6027598.824, -9218378.368, -6.508798398, -11824.42793, 18015.66212};
static __device__ const double g_e_yc[56] = {
    12.75434981, 12.75434981, 12.75434981, 11.37659788, 11.37659788, 11.37659788, 636.4346279, 636.4346279,
    636.4346279, 5.187666221, 5.187666221, 5.187666221, 6.802472048, 6.802472048, 6.802472048, 39.13543412,
    39.13543412, 39.13543412, 19.69877970, 19.69877970, 19.69877970, 20.30095680, 20.30095680, 20.30095680,
    86.45407420, 86.45407420, 86.45407420, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0, 0.0, 13.85650567, 13.85650567, 14.90554500, 14.90554500, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0};
static __device__ const double g_e_yr[56] = {
    1.0 / 12.75434981, 1.0 / 12.75434981, 1.0 / 12.75434981, 1.0 / 11.37659788, 1.0 / 11.37659788,
    1.0 / 11.37659788, 1.0 / 636.4346279, 1.0 / 636.4346279, 1.0 / 636.4346279, 1.0 / 5.187666221,
    1.0 / 5.187666221, 1.0 / 5.187666221, 1.0 / 6.802472048, 1.0 / 6.802472048, 1.0 / 6.802472048,
    1.0 / 39.13543412, 1.0 / 39.13543412, 1.0 / 39.13543412, 1.0 / 19.69877970, 1.0 / 19.69877970,
    1.0 / 19.69877970, 1.0 / 20.30095680, 1.0 / 20.30095680, 1.0 / 20.30095680, 1.0 / 86.45407420,
    1.0 / 86.45407420, 1.0 / 86.45407420, 1.0 / 5.303648988, 1.0 / 5.303648988, 1.0 / 5.303648988,
    1.0 / 5.303648988, 1.0 / 10.40368955, 1.0 / 10.40368955, 1.0 / 10.40368955, 1.0 / 10.40368955,
    1.0 / 69.65230348, 1.0 / 69.65230348, 1.0 / 69.65230348, 1.0 / 69.65230348, 1.0 / 466.5099509,
    1.0 / 466.5099509, 1.0 / 466.5099509, 1.0 / 466.5099509, 1.0 / 13.85650567, 1.0 / 13.85650567,
    1.0 / 14.90554500, 1.0 / 14.90554500, 0.12503844191332988, 0.12503844191332988, 0.12503844191332988,
    0.071597395204476152, 0.071597395204476152, 0.071597395204476152, 0.011080976889832743,
    0.011080976889832743, 0.011080976889832743};
static __device__ const double g_e_zc[56] = {
    1.752483754, 3.604231143, 12.83078674, 1.752483754, 3.604231143, 12.83078674, 1.752483754, 3.604231143,
    12.83078674, 2.784722096, 6.979576616, 25.71716760, 2.784722096, 6.979576616, 25.71716760, 2.784722096,
    6.979576616, 25.71716760, 22.50403727, 23.41617329, 48.48140573, 22.50403727, 23.41617329, 48.48140573,
    22.50403727, 23.41617329, 48.48140573, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0, 0.0, 10.21914434, 10.09021632, 10.21914434, 10.09021632, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0};
static __device__ const double g_e_zr[56] = {
    1.0 / 1.752483754, 1.0 / 3.604231143, 1.0 / 12.83078674, 1.0 / 1.752483754, 1.0 / 3.604231143,
    1.0 / 12.83078674, 1.0 / 1.752483754, 1.0 / 3.604231143, 1.0 / 12.83078674, 1.0 / 2.784722096,
    1.0 / 6.979576616, 1.0 / 25.71716760, 1.0 / 2.784722096, 1.0 / 6.979576616, 1.0 / 25.71716760,
    1.0 / 2.784722096, 1.0 / 6.979576616, 1.0 / 25.71716760, 1.0 / 22.50403727, 1.0 / 23.41617329,
    1.0 / 48.48140573, 1.0 / 22.50403727, 1.0 / 23.41617329, 1.0 / 48.48140573, 1.0 / 22.50403727,
    1.0 / 23.41617329, 1.0 / 48.48140573, 1.0 / 1.645049286, 1.0 / 3.825838190, 1.0 / 11.66675599,
    1.0 / 558.9781177, 1.0 / 1.645049286, 1.0 / 3.825838190, 1.0 / 11.66675599, 1.0 / 558.9781177,
    1.0 / 1.645049286, 1.0 / 3.825838190, 1.0 / 11.66675599, 1.0 / 558.9781177, 1.0 / 1.645049286,
    1.0 / 3.825838190, 1.0 / 11.66675599, 1.0 / 558.9781177, 1.0 / 10.21914434, 1.0 / 10.09021632,
    1.0 / 10.21914434, 1.0 / 10.09021632, 0.059675527522452816, 0.00098459526668325296,
    0.00064371058922777988, 0.059675527522452816, 0.00098459526668325296, 0.00064371058922777988,
    0.059675527522452816, 0.00098459526668325296, 0.00064371058922777988};
static __device__ const unsigned char g_e_ys[56] = {
    3, 3, 3, 4, 4, 4, 5, 5, 5, 9, 9, 9, 10, 10, 10, 11, 11, 11, 15, 15, 15, 16, 16, 16, 17, 17, 17, 22, 22,
    22, 22, 23, 23, 23, 23, 24, 24, 24, 24, 25, 25, 25, 25, 28, 28, 29, 29, 33, 33, 33, 34, 34, 34, 35, 35,
    35};
static __device__ const unsigned char g_e_zs[56] = {
    0, 1, 2, 0, 1, 2, 0, 1, 2, 6, 7, 8, 6, 7, 8, 6, 7, 8, 12, 13, 14, 12, 13, 14, 12, 13, 14, 18, 19, 20,
    21, 18, 19, 20, 21, 18, 19, 20, 21, 18, 19, 20, 21, 26, 27, 26, 27, 30, 31, 32, 30, 31, 32, 30, 31, 32};
// The sine/cosine tasks: argument v / c (c = 0: v r) with v = yy, zz, or the y
// or z of intercon's frame.
static __device__ const double g_s_c[36] = {
    1.752483754, 3.604231143, 12.83078674, 12.75434981, 11.37659788, 636.4346279, 2.784722096, 6.979576616,
    25.71716760, 5.187666221, 6.802472048, 39.13543412, 22.50403727, 23.41617329, 48.48140573, 19.69877970,
    20.30095680, 86.45407420, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 10.21914434, 10.09021632,
    13.85650567, 14.90554500, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
static __device__ const double g_s_r[36] = {
    1.0 / 1.752483754, 1.0 / 3.604231143, 1.0 / 12.83078674, 1.0 / 12.75434981, 1.0 / 11.37659788,
    1.0 / 636.4346279, 1.0 / 2.784722096, 1.0 / 6.979576616, 1.0 / 25.71716760, 1.0 / 5.187666221,
    1.0 / 6.802472048, 1.0 / 39.13543412, 1.0 / 22.50403727, 1.0 / 23.41617329, 1.0 / 48.48140573,
    1.0 / 19.69877970, 1.0 / 20.30095680, 1.0 / 86.45407420, 1.0 / 1.645049286, 1.0 / 3.825838190,
    1.0 / 11.66675599, 1.0 / 558.9781177, 1.0 / 5.303648988, 1.0 / 10.40368955, 1.0 / 69.65230348,
    1.0 / 466.5099509, 1.0 / 10.21914434, 1.0 / 10.09021632, 1.0 / 13.85650567, 1.0 / 14.90554500,
    0.059675527522452816, 0.00098459526668325296, 0.00064371058922777988, 0.12503844191332988,
    0.071597395204476152, 0.011080976889832743};
static __device__ const unsigned char g_s_v[36] = {
    1, 1, 1, 0, 0, 0, 1, 1, 1, 0, 0, 0, 1, 1, 1, 0, 0, 0, 1, 1, 1, 1, 0, 0, 0, 0, 1, 1, 0, 0, 3, 3, 3, 2,
    2, 2};
// Dipoles of condip1 (nine quadruples, then five pairs on the axis) and of
// diploop1 (pairs, or one where y = 0).
static __device__ const double g_dip_dx[46] = {
    -(-10.0 * 0.4), -(-10.0 * 0.4), -(-10.0 * 0.4), -(-10.0 * 0.4), -(-7.0 * 0.4), -(-7.0 * 0.4),
    -(-7.0 * 0.4), -(-7.0 * 0.4), -(-4.0 * 0.08), -(-4.0 * 0.08), -(-4.0 * 0.08), -(-4.0 * 0.08),
    -(-4.0 * 0.4), -(-4.0 * 0.4), -(-4.0 * 0.4), -(-4.0 * 0.4), -(0.0 * 0.08), -(0.0 * 0.08),
    -(0.0 * 0.08), -(0.0 * 0.08), -(4.0 * 0.08), -(4.0 * 0.08), -(4.0 * 0.08), -(4.0 * 0.08), -(4.0 * 0.4),
    -(4.0 * 0.4), -(4.0 * 0.4), -(4.0 * 0.4), -(7.0 * 0.4), -(7.0 * 0.4), -(7.0 * 0.4), -(7.0 * 0.4),
    -(10.0 * 0.4), -(10.0 * 0.4), -(10.0 * 0.4), -(10.0 * 0.4), 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0, 0.0};
static __device__ const double g_dip_dy[46] = {
    -(3.0 * 0.4), (3.0 * 0.4), -(3.0 * 0.4), (3.0 * 0.4), -(6.0 * 0.4), (6.0 * 0.4), -(6.0 * 0.4),
    (6.0 * 0.4), -(3.0 * 0.08), (3.0 * 0.08), -(3.0 * 0.08), (3.0 * 0.08), -(9.0 * 0.4), (9.0 * 0.4),
    -(9.0 * 0.4), (9.0 * 0.4), -(6.0 * 0.08), (6.0 * 0.08), -(6.0 * 0.08), (6.0 * 0.08), -(3.0 * 0.08),
    (3.0 * 0.08), -(3.0 * 0.08), (3.0 * 0.08), -(9.0 * 0.4), (9.0 * 0.4), -(9.0 * 0.4), (9.0 * 0.4),
    -(6.0 * 0.4), (6.0 * 0.4), -(6.0 * 0.4), (6.0 * 0.4), -(3.0 * 0.4), (3.0 * 0.4), -(3.0 * 0.4),
    (3.0 * 0.4), 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
static __device__ const double g_dip_dz[46] = {
    -20.0, -20.0, 20.0, 20.0, -20.0, -20.0, 20.0, 20.0, -4.0, -4.0, 4.0, 4.0, -20.0, -20.0, 20.0, 20.0,
    -4.0, -4.0, 4.0, 4.0, -4.0, -4.0, 4.0, 4.0, -20.0, -20.0, 20.0, 20.0, -20.0, -20.0, 20.0, 20.0, -20.0,
    -20.0, 20.0, 20.0, -2.0, 2.0, -3.0, 3.0, -4.5, 4.5, -7.0, 7.0, -10.0, 10.0};
static __device__ const double g_lop_dx[21] = {
    -11.0 * 1.12541, -11.0 * 1.12541, -7.0 * 1.12541, -7.0 * 1.12541, -7.0 * 1.12541, -3.0 * 1.12541,
    -3.0 * 1.12541, -3.0 * 1.12541, -3.0 * 1.12541, 1.0 * 1.12541, 1.0 * 1.12541, 1.0 * 1.12541,
    1.0 * 1.12541, 1.0 * 1.12541, 5.0 * 1.12541, 5.0 * 1.12541, 5.0 * 1.12541, 5.0 * 1.12541,
    9.0 * 1.12541, 9.0 * 1.12541, 9.0 * 1.12541};
static __device__ const double g_lop_dy[21] = {
    -(2.0 * 0.945719), 2.0 * 0.945719, -(0.0 * 0.945719), -(4.0 * 0.945719), 4.0 * 0.945719,
    -(2.0 * 0.945719), 2.0 * 0.945719, -(6.0 * 0.945719), 6.0 * 0.945719, -(0.0 * 0.945719),
    -(4.0 * 0.945719), 4.0 * 0.945719, -(8.0 * 0.945719), 8.0 * 0.945719, -(2.0 * 0.945719),
    2.0 * 0.945719, -(6.0 * 0.945719), 6.0 * 0.945719, -(0.0 * 0.945719), -(4.0 * 0.945719), 4.0 * 0.945719};
static __device__ const unsigned char g_lop_first[13] = {0, 2, 3, 5, 7, 9, 10, 12, 14, 16, 18, 19, 21};

// Per shield: first term, rows, columns.
static __device__ const unsigned char g_sh_first[7] = {0, 9, 18, 27, 43, 47, 56};

struct T96Slot {
    double x, y, z;               // GSM [R_E] x xappa
    double yi, zi;                // intercon's rotated y, z
    double X, Y, Z;               // GSM [R_E]
    double sigma, oimfy, oimfz;
    double xks;
    double pl[3], pc[3];          // where the loops and the conical basis are taken
    double e1[3], e2[3];          // blend band: the two edge points
    double sc[kT96Sc][2];
    double ex[kT96Exp][3];
    double bes[6][3][2];
    double rt[6][3][2];
    double t87[3][7];
    double dip[kT96Dip][6];
    double lop[kT96Lop][4];
    double cir[18][3];            // 0-2 loops basis, 3-13 r2outer, 3-6 r2inner
    double con[5][3], inn[7][3], sheet[3];   // harmonics by order; inn: 5, 6 the distributed dipoles
    double shield[6][3];
    double tl[3], tc[3], cyl[3], ring[3], tail[3], tail87[2], ri[3], ro[3];
    const T96Cond* c;
    unsigned flags;               // kT96* below, after phase 1
    int band;                     // r2_birk's band of xksi
};

constexpr unsigned kT96In = 1u, kT96Loops = 2u, kT96Con = 4u, kT96Blend = 8u, kT96South = 16u;

// ---- before phase 1 (the quad) -------------------------------------------
__device__ __forceinline__ void t96_slot_start(T96Slot& s, const T96Cond& c, const Vec3 X) {
    const double x = X.x, y = X.y, z = X.z;
    const double ys = y * c.ct - z * c.st, zs = z * c.ct + y * c.st;
    s.X = x;
    s.Y = y;
    s.Z = z;
    s.x = x * c.xappa;
    s.y = y * c.xappa;
    s.z = z * c.xappa;
    s.yi = ys * c.xappa;
    s.zi = zs * c.xappa;
    s.c = &c;
    s.flags = kT96In;
    s.band = 2;
}

// ---- phase 1 ---------------------------------------------------------------
// IMF field outside and the magnetopause distance (t96_field's start).
static __device__ __noinline__ void t96_task_main(T96Slot& s) {
    const T96Cond& c = *s.c;
    const double x = s.X, y = s.Y, z = s.Z;
    const double ys = y * c.ct - z * c.st;
    const double ysd = div_c(ys, 10.0, 1.0 / 10.0);
    const double factimf = ol_exp(div_c(x, 20.0, 1.0 / 20.0) - ysd * ysd);
    s.oimfy = c.kimfy * factimf;
    s.oimfz = c.kimfz * factimf;
    const double rho2 = __dadd_rn(__dmul_rn(y, y), __dmul_rn(z, z));   // t96_field's squares have other uses
    double xmxm = c.am + x - c.c548;
    if (xmxm < 0.0) xmxm = 0.0;
    const double axx0 = xmxm * xmxm;
    const double aro = c.asq + rho2;
    const double aa = aro + axx0;
    s.sigma = sqrt(div_r(aro + axx0 + sqrt(aa * aa - c.four_asq * axx0), c.two_asq, c.r_two_asq));
}

// t96_birk1tot up to the points where its bases are taken, by two neighbouring
// lanes that take one of the two arc tangents and of their sines each (the
// whole warp calls; live: the lane's slot is evaluated).
static __device__ __noinline__ void t96_task_b1(T96Slot& s, const bool live) {
    const double x = s.x, y = s.y, z = s.z;
    const bool odd = threadIdx.x & 1;
    const double an = ol_atan2(odd ? sqrt(x * x + y * y) : y, odd ? z : x);
    const double ap = !odd && x == 0.0 && y == 0.0 ? 0.0 : an;
    const double sn = ol_sin(odd ? ap : ap * 0.5);
    const double pas = __shfl_sync(0xffffffffu, ap, threadIdx.x & 30);
    const double tas = __shfl_sync(0xffffffffu, ap, threadIdx.x | 1);
    const double sh = __shfl_sync(0xffffffffu, sn, threadIdx.x & 30);
    const double stas = __shfl_sync(0xffffffffu, sn, threadIdx.x | 1);
    if (!live || odd) return;
    const double tnoonn = 12.0 * 0.01745329;
    const double tnoons = 3.141592654 - tnoonn;
    const double r2 = x * x + y * y + z * z;
    const double r = sqrt(r2);
    const double r3 = r * r2;
    double tet0 = ol_asin(stas / ol_pow((stas * stas * stas * stas * stas * stas) * (1.0 - r3) + r3, 0.1666666667));
    if (tas > 1.5707963) tet0 = 3.141592654 - tet0;
    const double dtet = (8.0 * 0.01745329) * (sh * sh);
    const double tr1n = tnoonn + dtet, tr1s = tnoons - dtet;
    const double t01n = tr1n - 0.034906, t01s = tr1s - 0.034906;
    const double t02s = tr1s + 0.034906, t02n = tr1n + 0.034906;
    const bool loops_here = tet0 < t01n || tet0 > t02s;
    const bool condip_here = tet0 > t02n && tet0 < t01s;
    const bool band = (tet0 >= t01n && tet0 <= t02n) || (tet0 >= t01s && tet0 <= t02s);
    const bool south = tet0 >= t01s;
    double pl[3] = {x, y, z}, pc[3] = {x, y, z};
    if (band) {
        double spas, cpas;
        ol_sincos(pas, &spas, &cpas);
        const B1Edges e = t96_birk1_edges(r, r3, cpas, spas, south ? t01s : t01n, south ? t02s : t02n, south);
        pl[0] = south ? e.x2 : e.x1;
        pl[1] = south ? e.y2 : e.y1;
        pl[2] = south ? e.z2 : e.z1;
        pc[0] = south ? e.x1 : e.x2;
        pc[1] = south ? e.y1 : e.y2;
        pc[2] = south ? e.z1 : e.z2;
        s.e1[0] = e.x1;
        s.e1[1] = e.y1;
        s.e1[2] = e.z1;
        s.e2[0] = e.x2;
        s.e2[1] = e.y2;
        s.e2[2] = e.z2;
    }
#pragma unroll
    for (int i = 0; i < 3; i++) {
        s.pl[i] = pl[i];
        s.pc[i] = pc[i];
    }
    s.flags = kT96In | (loops_here || band ? kT96Loops : 0u) | (condip_here || band ? kT96Con : 0u) |
              (band ? kT96Blend : 0u) | (south ? kT96South : 0u);
}

static __device__ __noinline__ void t96_task_xksi(T96Slot& s) {
    const double dl = 0.03, dl1 = 0.015;
    const double xks = t96_xksi(s.x, s.y, s.z);
    s.xks = xks;
    s.band = xks < -(dl + dl1) ? 0 : xks < -dl + dl1 ? 1 : xks < dl - dl1 ? 2 : xks < dl + dl1 ? 3 : 4;
}

// Term i of cylharm: factor pairs of the three components.
static __device__ __noinline__ void t96_task_bes(T96Slot& s, const int i) {
    constexpr double AC[12] = {0.24777, -27.003, -0.46815, 7.0637, -1.5918, -0.90317E-01,
                               57.522, 13.757, 2.0100, 10.458, 4.5798, 2.1695};
    double A = AC[0], c = AC[6], rc = 1.0 / AC[6];
#pragma unroll
    for (int k = 1; k < 6; k++)
        if (i == k) {
            A = AC[k];
            c = AC[6 + k];
            rc = 1.0 / AC[6 + k];
        }
    const double x = s.x, y = s.y, z = s.z;
    double rho = sqrt(y * y + z * z), sf, cf;
    if (rho < 1.0e-8) {
        sf = 1.0;
        cf = 0.0;
        rho = 1.0e-8;
    } else {
        const double rr = 1.0 / rho;
        sf = div_r(z, rho, rr);
        cf = div_r(y, rho, rr);
    }
    const double sf2 = sf * sf;
    const double s2c2 = sf2 - cf * cf;
    const double dz = div_c(rho, c, rc);
    const double xk = div_c(x, c, rc);
    double j0, j1;
    t96_bes01(dz, j0, j1);
    const double e = ol_exp(xk);
    double(*o)[2] = s.bes[i];
    if (i < 3) {
        const double j1dz = j1 / dz;
        o[0][0] = -(A * j1 * e);
        o[0][1] = sf;
        o[1][0] = A * (2.0 * j1 / dz - j0) * e * sf;
        o[1][1] = cf;
        o[2][0] = A * (j1dz * s2c2 - j0 * sf2);
        o[2][1] = e;
    } else {
        const double brho = (xk * j0 - (dz * dz + xk - 1.0) * j1 / dz) * e * sf;
        const double bphi = (j0 + j1 / dz * (xk - 1.0)) * e * cf;
        o[0][0] = A * (dz * j0 + xk * j1) * e;
        o[0][1] = sf;
        o[1][0] = A;
        o[1][1] = __fma_rn(brho, cf, -__dmul_rn(bphi, sf));
        o[2][0] = A;
        o[2][1] = __fma_rn(bphi, cf, __dmul_rn(brho, sf));
    }
}

// Loop term i of ringcurr_96 (0, 1) or taildisk_t96 (2 .. 5): the ring current
// is the disk's form with half thickness 2, no shift and no warp.
static __device__ __noinline__ void t96_task_rt(T96Slot& s, const int i) {
    constexpr double FC[6] = {569.895366, -1603.386993, -745796.7338, 1176470.141, -444610.529, -57508.01028};
    constexpr double BC[6] = {2.722188, 3.766875, 7.9250000, 8.0850000, 8.4712500, 27.89500};
    double F = FC[0], bi = BC[0], bb = (2.0 * BC[0]) * (2.0 * BC[0]);
#pragma unroll
    for (int k = 1; k < 6; k++)
        if (i == k) {
            F = FC[k];
            bi = BC[k];
            bb = (2.0 * BC[k]) * (2.0 * BC[k]);
        }
    const bool ring = i < 2;
    const double x = s.x, y = s.y, z = s.z;
    const double y20 = div_c(y, 20.0, 1.0 / 20.0);
    const double dt = __fma_rn(10.0, __dmul_rn(y20, y20), 2.0);
    const double d = ring ? 2.0 : dt;
    const double dzs = sqrt(__fma_rn(z, z, __dmul_rn(d, d)));
    const double rdz = 1.0 / dzs;
    const double ddy = ring ? 0.0 : div_r(d * 10.0 * y * 0.005, dzs, rdz);
    const double ddz = div_r(z, dzs, rdz);
    const double xs = ring ? x : x - 4.5;
    const double rhos = sqrt(__fma_rn(xs, xs, __dmul_rn(y, y)));
    double drx = 0.0, dry = (y >= 0) ? 1.0 : -1.0;
    if (rhos >= 1.0e-5) {
        const double rr = 1.0 / rhos;
        drx = div_r(xs, rhos, rr);
        dry = div_r(y, rhos, rr);
    }
    const double dzb = dzs + bi, rp = rhos + bi, rm = rhos - bi;
    const double s1 = sqrt(__fma_rn(dzb, dzb, __dmul_rn(rp, rp))), s2 = sqrt(__fma_rn(dzb, dzb, __dmul_rn(rm, rm)));
    const double r1 = 1.0 / s1, r2 = 1.0 / s2;
    const double ds1dz = div_r(dzb, s1, r1), ds2dz = div_r(dzb, s2, r2);
    const double ds1dr = div_r(rp, s1, r1), ds2dr = div_r(rm, s2, r2);
    const double s12 = s1 * s2, sp = s1 + s2, sp2 = __dmul_rn(sp, sp);
    const double fac1 = sqrt(__dadd_rn(sp2, -bb));
    const double as = fac1 / (s12 * sp2);
    const double term1 = 1.0 / (s12 * sp * fac1);
    const double fac2 = as / sp2;
    const double q1 = __fma_rn(3.0, s1, __dmul_rn(4.0, s2)), q2 = __fma_rn(3.0, s2, __dmul_rn(4.0, s1));
    const double w1 = __fma_rn(s2, s2, __dmul_rn(s1, q1)), w2 = __fma_rn(s1, s1, __dmul_rn(s2, q2));
    const double das1 = __fma_rn(-div_r(fac2, s1, r1), w1, term1);
    const double das2 = __fma_rn(-div_r(fac2, s2, r2), w2, term1);
    const double dasdx = __fma_rn(das1, __dmul_rn(ds1dr, drx), __dmul_rn(das2, __dmul_rn(ds2dr, drx)));
    const double e1 = __fma_rn(ds1dz, ddy, __dmul_rn(ds1dr, dry)), e2 = __fma_rn(ds2dz, ddy, __dmul_rn(ds2dr, dry));
    const double dasdy = __fma_rn(das1, e1, __dmul_rn(das2, e2));
    const double dasdz = __fma_rn(das1, __dmul_rn(ds1dz, ddz), __dmul_rn(das2, __dmul_rn(ds2dz, ddz)));
    double(*o)[2] = s.rt[i];
    o[0][0] = ring ? -F * x : F;
    o[0][1] = ring ? dasdz : (4.5 - x) * dasdz;
    o[1][0] = -(F * y);
    o[1][1] = dasdz;
    o[2][0] = F;
    o[2][1] = __fma_rn(xs, dasdx, __fma_rn(2.0, as, __dmul_rn(y, dasdy)));
}

// Line current i of tail87: z, z - 40, z + 40.
static __device__ __noinline__ void t96_task_t87(T96Slot& s, const int i) {
    const double x = s.x, z = s.z;
    const double zp = z - 40.0, zm = z + 40.0;
    const double zl = i == 0 ? z : i == 1 ? zp : zm;
    const double xnx = -10.0 - x;
    const double xnx2 = xnx * xnx;
    const double xc1 = x + 1.261, xc2 = x + 0.663;
    const double xc22 = xc2 * xc2;
    const double xr2 = xc2 * -0.1071;
    const double xc12 = xc1 * xc1;
    const double d2 = 3.0 * 3.0;
    const double b2 = __fma_rn(zl, zl, d2);
    const T87Line l = t96_tail87_line(b2, xnx, xnx2, xc1, xc12, xc2, xc22, xr2);
    s.t87[i][0] = l.s0;
    s.t87[i][1] = l.s1;
    s.t87[i][2] = l.s2;
    s.t87[i][3] = l.g1;
    s.t87[i][4] = l.xln1;
    // g2's last product as factors: t96_tail87 adds one of them unrounded
    const double f = __dadd_rn(b2, -__dmul_rn(xc2, xc2));
    const double w = __fma_rn(0.5 * f, l.xln1 + 0.13238005, __dmul_rn(2. * l.s0 * b2, xc2));
    s.t87[i][5] = __fma_rn(xc2, -0.1071, __dmul_rn(w, l.xa2));
    s.t87[i][6] = l.xa2;
}

__device__ __forceinline__ double div_or_mul(const double v, const double c, const double r) {
    const double q = div_c(v, c, r);
    return c != 0.0 ? q : v * r;
}

__device__ __forceinline__ void t96_task_sc(T96Slot& s, const int i) {
    const int v = g_s_v[i];
    const double a = v == 0 ? s.y : v == 1 ? s.z : v == 2 ? s.yi : s.zi;
    const SinCos r = ol_sincos_v(div_or_mul(a, g_s_c[i], g_s_r[i]));
    s.sc[i][0] = r.s;
    s.sc[i][1] = r.c;
}

// ---- phase 2 ---------------------------------------------------------------
__device__ __forceinline__ void t96_task_exp(T96Slot& s, const int i) {
    const double sq = i < 27   ? g_t96.shl_sq[i / 9][i % 9]
                      : i < 43 ? g_t96.b1s_sq[i - 27]
                      : i < 47 ? g_t96.b2s_sq[i - 43]
                               : g_t96.ic_sq[i - 47];
    const double* ys = s.sc[g_e_ys[i]];
    const double* zs = s.sc[g_e_zs[i]];
    const double sy = ys[0], cy = ys[1], sz = zs[0], cz = zs[1];
    const double e = ol_exp(s.x * sq);
    s.ex[i][0] = -sq * e * cy * sz;
    s.ex[i][1] = div_or_mul(e, g_e_yc[i], g_e_yr[i]) * sy * sz;
    s.ex[i][2] = -div_or_mul(e, g_e_zc[i], g_e_zr[i]) * cy * cz;
}

__device__ __forceinline__ void t96_task_dip(T96Slot& s, const int i) {
    const Dip3 d = t96_dipxyz(s.pc[0] + g_dip_dx[i], s.pc[1] + g_dip_dy[i], s.pc[2] + g_dip_dz[i]);
    double* o = s.dip[i];
    o[0] = d.dx.x;
    o[1] = d.dx.y;
    o[2] = d.dx.z;
    o[3] = d.dy.y;
    o[4] = d.dy.z;
    o[5] = d.dz.z;
}

static __device__ __noinline__ void t96_task_lop(T96Slot& s, const int i) {
    const double x = s.pl[0], y = s.pl[1], z = s.pl[2];
    const double z2 = z * z;
    const double xd = x - g_lop_dx[i];
    const double yd = y + g_lop_dy[i];
    const double r2 = __dadd_rn(__fma_rn(yd, yd, __dmul_rn(xd, xd)), z2);
    const double xmr5 = 30574.0 / (r2 * r2 * sqrt(r2));
    const double xmr53 = 3.0 * xmr5;
    s.lop[i][0] = xmr53 * xd;
    s.lop[i][1] = xmr53 * yd;
    s.lop[i][2] = xmr5;
    s.lop[i][3] = __fma_rn(3.0, z2, -r2);
}

// Current circles: 0, 1 the crossed loops and 2 the circle of the loops basis;
// r2outer's three crossed loops (3 .. 8), circle (9) and four tilted loops
// (10 .. 13); r2inner's four tilted loops (3 .. 6).
static __device__ __noinline__ void t96_task_circle(T96Slot& s, const int k, const bool inner) {
    double x = s.x, y = s.y, z = s.z, rl;
    if (k < 3) {
        x = s.pl[0];
        y = s.pl[1];
        z = s.pl[2];
    }
    if (k < 2 || (k < 9 && !inner && k >= 3)) {
        // crosslp
        const int it = k < 2 ? 0 : (k - 1) >> 1;
        const bool second = k < 2 ? k == 1 : ((k - 3) & 1) != 0;
        const double xc = it == 0 ? 2.28397 : it == 1 ? 0.55 : it == 2 ? 1.55 : -0.7;
        rl = it == 0 ? 1.86106 : it == 1 ? 0.694 : it == 2 ? 2.8 : 0.2;
        const double cal = g_t96.cross_cs[it][0], sal = g_t96.cross_cs[it][1];
        const double sg = second ? -sal : sal;
        const double yc = __fma_rn(y, cal, -__dmul_rn(z, sg));
        z = __fma_rn(z, cal, __dmul_rn(y, sg));
        y = yc;
        x = x - xc;
    } else if (k == 2 || (k == 9 && !inner)) {
        x = x + (k == 2 ? 5.60831 : 2.994);
        rl = k == 2 ? 7.83281 : 2.925;
    } else {
        // loops4
        const int il = inner ? 0 : 1, v = inner ? k - 3 : k - 10;
        const double xc = inner ? -8.1902 : -1.775, yc = inner ? 6.5239 : 4.3, zc = inner ? 5.504 : -0.275;
        rl = inner ? 7.7815 : 2.7;
        const double st = g_t96.loop_cs[il][0], ct = g_t96.loop_cs[il][1];
        const double sp = g_t96.loop_cs[il][2], cp = g_t96.loop_cs[il][3];
        // (both products of a sum that is not fused here have two uses there)
        const double dx = x - xc, dm = y - yc, dq = y + yc;
        const double xs0 = __dadd_rn(__dmul_rn(dx, cp), __dmul_rn(dm, sp));
        const double ys0 = __dadd_rn(__dmul_rn(dm, cp), -__dmul_rn(dx, sp));
        const double xs1 = __dadd_rn(__dmul_rn(dx, cp), -__dmul_rn(dq, sp));
        const double ys1 = __fma_rn(dq, cp, __dmul_rn(dx, sp));
        const double xs2 = -xs1;
        const double ys2 = -ys1;
        const double xs3 = __fma_rn(-dx, cp, -__dmul_rn(dm, sp));
        const double ys3 = -ys0;
        const double xs = v == 0 ? xs0 : v == 1 ? xs1 : v == 2 ? xs2 : xs3;
        const double yss = v == 0 ? ys0 : v == 1 ? ys1 : v == 2 ? ys2 : ys3;
        const double zs = v < 2 ? z - zc : z + zc;
        x = __fma_rn(xs, ct, -__dmul_rn(zs, st));
        z = __fma_rn(zs, ct, __dmul_rn(xs, st));
        y = yss;
    }
    const Vec3 b = t96_circle(x, y, z, rl);
    s.cir[k][0] = b.x;
    s.cir[k][1] = b.y;
    s.cir[k][2] = b.z;
}

// (tan t/2)^m + (cot t/2)^m of a conical harmonic and the powers below, m =
// k + 1: the last order's powers are only added there, in one rounding.
__device__ __forceinline__ double t96_cone_powers(const double tnh, const double cnh, const int k, double& tp,
                                                  double& cp) {
    tp = cp = 1.0;
    double t1 = tnh, c1 = cnh;
#pragma unroll
    for (int i = 1; i < 5; i++) {
        if (i <= k) {
            tp = t1;
            cp = c1;
            t1 = __dmul_rn(tp, tnh);
            c1 = __dmul_rn(cp, cnh);
        }
    }
    return k == 4 ? __fma_rn(tp, tnh, c1) : __dadd_rn(t1, c1);
}

// Conical harmonic k + 1 of condip1 (t96_r1_condip's first sum).  The angles
// are every order's; three quotients and the powers are its own.  All five by
// one lane took 22,500 cycles (r2inner's, with the dipoles, 30,400) and were
// their phase's longest tasks; by order a lone T96 trajectory's step went
// from 62.4 us to 56.8 (with the arc tangents of t96_task_b1 by two lanes,
// 23,200 cycles by one), 8,000 trajectories of 250 steps from 114 ms to 110.
static __device__ __noinline__ void t96_task_con(T96Slot& sl, const int k) {
    const double x = sl.pc[0], y = sl.pc[1], z = sl.pc[2];
    const double xsm = x + 0.16;
    const double ro2 = xsm * xsm + y * y;
    const double ro = sqrt(ro2);
    const double rro = 1.0 / ro;
    const double cf0 = div_r(xsm, ro, rro), sf0 = div_r(y, ro, rro);
    double cf = cf0, sf = sf0;
    if (k > 0) {
        cf = cf0 * cf0 - sf0 * sf0;
        sf = 2.0 * sf0 * cf0;
    }
#pragma unroll
    for (int m = 2; m < 5; m++) {
        const double c1 = __fma_rn(cf, cf0, -__dmul_rn(sf, sf0));
        const double s1 = __fma_rn(sf, cf0, __dmul_rn(cf, sf0));
        if (m <= k) {
            cf = c1;
            sf = s1;
        }
    }
    const double r2 = ro2 + z * z;
    const double r = sqrt(r2);
    const double rr = 1.0 / r;
    const double c = div_r(z, r, rr), s = div_r(ro, r, rr);
    const double ch = sqrt(0.5 * (1.0 + c)), sh = sqrt(0.5 * (1.0 - c));
    const double tnh = sh / ch, cnh = 1.0 / tnh;
    const double ch2 = ch * ch, sh2 = sh * sh;
    const double rs = r * s;
    const double mn = k + 1;
    double tp, cp;
    const double sum = t96_cone_powers(tnh, cnh, k, tp, cp);
    const double bt = mn * cf / rs * sum;
    const double bf = div_r(-0.5 * mn * sf, r, rr) * (tp / ch2 - cp / sh2);
    sl.con[k][0] = __fma_rn(bt * c, cf0, -__dmul_rn(bf, sf0));
    sl.con[k][1] = __fma_rn(bt * c, sf0, __dmul_rn(bf, cf0));
    sl.con[k][2] = -bt * s;
}

// Conical harmonic k + 1 of r2inner (k < 5), or its distributed dipoles (5, 6).
static __device__ __noinline__ void t96_task_inner(T96Slot& sl, const int k) {
    const double x = sl.x, y = sl.y, z = sl.z;
    double* o = sl.inn[k];
    // a square that t96_r2inner uses in several sums, and so does not fuse
    const double yy = __dmul_rn(y, y);
    if (k >= 5) {
        const double xx = k == 5 ? x - .0774 : x + .038;
        const double x2 = __dmul_rn(xx, xx);
        const double rho2 = __dadd_rn(x2, yy);
        const double rho4 = rho2 * rho2;
        if (k == 5) {
            const double q2 = __fma_rn(z, z, rho2);
            const double r3 = q2 * sqrt(q2);
            o[0] = z / rho4 * __fma_rn(q2, __dadd_rn(yy, -x2), -__dmul_rn(rho2, x2)) / r3;
            o[1] = -xx * y * z / rho4 * (2.0 * q2 + rho2) / r3;
            o[2] = xx / r3;
        } else {
            o[0] = z / rho4 * __dadd_rn(yy, -x2);
            o[1] = -2.0 * xx * y * z / rho4;
            o[2] = xx / rho2;
        }
        return;
    }
    const double ro2 = __fma_rn(x, x, yy);
    const double ro = sqrt(ro2);
    const double rro = 1.0 / ro;
    const double cf = div_r(x, ro, rro), sf = div_r(y, ro, rro);
    const double r2 = __fma_rn(z, z, ro2);
    const double r = sqrt(r2);
    const double rr = 1.0 / r;
    const double c = div_r(z, r, rr), s = div_r(ro, r, rr);
    const double ch = sqrt(0.5 * (1.0 + c)), sh = sqrt(0.5 * (1.0 - c));
    const double tnh = sh / ch, cnh = 1.0 / tnh;
    const double ch2 = ch * ch, sh2 = sh * sh;
    const double rs = r * s;
    double cfm = cf, sfm = sf;
#pragma unroll
    for (int m = 1; m < 5; m++) {
        const double c1 = __fma_rn(cfm, cf, -__dmul_rn(sfm, sf));
        const double s1 = __fma_rn(cfm, sf, __dmul_rn(sfm, cf));
        if (m <= k) {
            cfm = c1;
            sfm = s1;
        }
    }
    double tp, cp;
    const double sum = t96_cone_powers(tnh, cnh, k, tp, cp);
    const double mn = k + 1;
    const double bt = mn * cfm / rs * sum;
    const double bf = div_r(-0.5 * mn * sfm, r, rr) * (tp / ch2 - cp / sh2);
    o[0] = __fma_rn(bt * c, cf, -__dmul_rn(bf, sf));
    o[1] = __fma_rn(bt * c, sf, __dmul_rn(bf, cf));
    o[2] = -bt * s;
}

// Component C of t96_r2sheet.
template <int C>
static __device__ __noinline__ void t96_task_sheet(T96Slot& sl) {
    constexpr double CX[5][4][4] = T96_SHEET_X;
    constexpr double CY[5][4][4] = T96_SHEET_Y;
    constexpr double CZ[5][4][4] = T96_SHEET_Z;
    const double x = sl.x, y = sl.y, z = sl.z, xks = sl.xks;
    const double xks2 = xks * xks;
    const double rho2 = x * x + y * y;
    const double r = sqrt(rho2 + z * z);
    const double rho = sqrt(rho2);
    const double rrho = 1.0 / rho;
    const double c1p = div_r(x, rho, rrho), s1p = div_r(y, rho, rrho);
    const double s2p = 2.0 * s1p * c1p;
    const double c2p = c1p * c1p - s1p * s1p;
    const double s3p = s2p * c1p + c2p * s1p;
    const double c3p = c2p * c1p - s2p * s1p;
    const double s4p = s3p * c1p + c3p * s1p;
    const double ct = z / r;
    const double ct2 = ct * ct;
    const double ct2m1 = ct2 - 1.0;
    double s[5], acc;
    if constexpr (C == 0) {
        const double t1x = xks / sqrt(__dadd_rn(xks2, 0.483750e-01 * 0.483750e-01));
        const double px72 = 0.396953e-01 * 0.396953e-01;
        const double qx = sqrt(__dadd_rn(xks2, px72));
        const double t2x = (px72 * 0.396953e-01) / (qx * qx * qx);
        const double ux = sqrt(__dadd_rn(xks2, 0.579023e-01 * 0.579023e-01));
        const double t3x = xks / T96_POW5(ux) * 3.493856 * c_t96.r2s_k[5];
        s[0] = c_t96.r2s_k[0] * ct * ol_exp(-19.0969 * ct2);
        s[1] = c_t96.r2s_k[1] * ct * ol_exp(-9.28828 * ct2);
        s[2] = c_t96.r2s_k[2] * ct * ol_exp(-0.129687 * ct2);
        s[3] = ct * ol_exp(5.58594 * ct2m1);
        s[4] = ct * ol_exp(22.5055 * ct2m1);
        acc = 0.0;
    #pragma unroll
        for (int l = 0; l < 5; l++) {
            const double term = (CX[l][0][0] + CX[l][0][1] * t1x + CX[l][0][2] * t2x + CX[l][0][3] * t3x) +
                                c1p * (CX[l][1][0] + CX[l][1][1] * t1x + CX[l][1][2] * t2x + CX[l][1][3] * t3x) +
                                c2p * (CX[l][2][0] + CX[l][2][1] * t1x + CX[l][2][2] * t2x + CX[l][2][3] * t3x) +
                                c3p * (CX[l][3][0] + CX[l][3][1] * t1x + CX[l][3][2] * t2x + CX[l][3][3] * t3x);
            acc = (l == 0) ? s[l] * term : acc + s[l] * term;
        }
    } else if constexpr (C == 1) {
        const double t1y = xks / sqrt(__dadd_rn(xks2, 0.478750e-01 * 0.478750e-01));
        const double py72 = 0.363750e-01 * 0.363750e-01;
        const double qy = sqrt(__dadd_rn(xks2, py72));
        const double t2y = (py72 * 0.363750e-01) / (qy * qy * qy);
        const double uy = sqrt(__dadd_rn(xks2, 0.567500e-01 * 0.567500e-01));
        const double t3y = xks / T96_POW5(uy) * 3.493856 * c_t96.r2s_k[6];
        s[0] = c_t96.r2s_k[3] * ct * ol_exp(-13.6750 * ct2);
        s[1] = c_t96.r2s_k[4] * ct * ol_exp(-6.70625 * ct2);
        s[2] = ct * ol_exp(2.31875 * ct2m1);
        s[3] = ct * ol_exp(11.4062 * ct2m1);
        s[4] = ct * ol_exp(20.4562 * ct2m1);
        acc = 0.0;
    #pragma unroll
        for (int l = 0; l < 5; l++) {
            const double term = s1p * (CY[l][0][0] + CY[l][0][1] * t1y + CY[l][0][2] * t2y + CY[l][0][3] * t3y) +
                                s2p * (CY[l][1][0] + CY[l][1][1] * t1y + CY[l][1][2] * t2y + CY[l][1][3] * t3y) +
                                s3p * (CY[l][2][0] + CY[l][2][1] * t1y + CY[l][2][2] * t2y + CY[l][2][3] * t3y) +
                                s4p * (CY[l][3][0] + CY[l][3][1] * t1y + CY[l][3][2] * t2y + CY[l][3][3] * t3y);
            acc = (l == 0) ? s[l] * term : acc + s[l] * term;
        }
    } else {
        const double t1z = xks / sqrt(__dadd_rn(xks2, 0.355625e-01 * 0.355625e-01));
        const double pz72 = 0.318750e-01 * 0.318750e-01;
        const double qz = sqrt(__dadd_rn(xks2, pz72));
        const double t2z = (pz72 * 0.318750e-01) / (qz * qz * qz);
        const double uz = sqrt(__dadd_rn(xks2, 0.538750e-01 * 0.538750e-01));
        const double t3z = xks / T96_POW5(uz) * 3.493856 * c_t96.r2s_k[7];
        s[0] = ol_exp(-16.7125 * ct2);
        s[1] = ol_exp(-16.4625 * ct2);
        s[2] = ol_exp(-0.1625 * ct2);
        s[3] = ol_exp(5.1 * (ct2 - 1.0));
        s[4] = ol_exp(23.7125 * (ct2 - 1.0));
        acc = 0.0;
    #pragma unroll
        for (int l = 0; l < 5; l++) {
            const double term = (CZ[l][0][0] + CZ[l][0][1] * t1z + CZ[l][0][2] * t2z + CZ[l][0][3] * t3z) +
                                c1p * (CZ[l][1][0] + CZ[l][1][1] * t1z + CZ[l][1][2] * t2z + CZ[l][1][3] * t3z) +
                                c2p * (CZ[l][2][0] + CZ[l][2][1] * t1z + CZ[l][2][2] * t2z + CZ[l][2][3] * t3z) +
                                c3p * (CZ[l][3][0] + CZ[l][3][1] * t1z + CZ[l][3][2] * t2z + CZ[l][3][3] * t3z);
            acc = (l == 0) ? s[l] * term : acc + s[l] * term;
        }
    }
    sl.sheet[C] = acc;
}

// ---- phase 3 ---------------------------------------------------------------
__device__ __forceinline__ void t96_sum_shield(T96Slot& s, const int t, const int c) {
    double h = 0.0;
    for (int i = g_sh_first[t]; i < g_sh_first[t + 1]; i++) h += s.ex[i][c] * g_e_amp[i];
    s.shield[t][c] = h;
}

// Component c of the conical basis: dipole o's three fields are stored as the
// six different components.
static __device__ const unsigned char g_dip_at[3][3] = {{0, 1, 2}, {1, 3, 4}, {2, 4, 5}};
static __device__ const double g_con_c2[37] = {
    1.41714, -27.2586, -4.28833, -1.30675, 35.5607, 8.95792, 0.961617E-03, -0.801477E-03, -0.782795E-03,
    -1.65242, -16.5242, -5.33798, 0.424878E-03, 0.331787E-03, -0.704305E-03, 0.844342E-03, 0.953682E-04,
    0.886271E-03, 25.1120, 20.9299, 5.14569, -44.1670, -51.0672, -1.87725, 20.2998, 48.7505, -2.97415,
    0.174615E-03, -0.789777E-06, 0.686047E-03, 0.460104E-04, -0.345216E-02, 0.221871E-02, 0.110078E-01,
    -0.661373E-02, 0.249201E-02, 0.343978E-01};

__device__ __forceinline__ void t96_sum_con(T96Slot& s, const int c) {
    constexpr double C2[5] = {6.04133, 0.305415, 0.606066E-02, 0.128379E-03, -0.179406E-04};
    double b = 0.0;
#pragma unroll
    for (int m = 0; m < 5; m++) b += C2[m] * s.con[m][c];
    const int ax = g_dip_at[0][c], ay = g_dip_at[1][c], az = g_dip_at[2][c];
    for (int i = 0; i < 9; i++) {
        const double(*d)[6] = &s.dip[4 * i];
        b += g_con_c2[3 * i] * (d[0][ax] + d[1][ax] - d[2][ax] - d[3][ax]);
        b += g_con_c2[3 * i + 1] * (d[0][ay] - d[1][ay] - d[2][ay] + d[3][ay]);
        b += g_con_c2[3 * i + 2] * (d[0][az] + d[1][az] + d[2][az] + d[3][az]);
    }
    for (int i = 0; i < 5; i++) {
        const double(*d)[6] = &s.dip[36 + 2 * i];
        b += g_con_c2[27 + 2 * i] * (d[0][ax] - d[1][ax]);
        b += g_con_c2[28 + 2 * i] * (d[0][az] + d[1][az]);
    }
    s.tc[c] = b;
}

// t96_crosslp's combination of its two circles; loops4's of its four.
static __device__ __noinline__ Vec3 t96_cross_of(const double (*q)[3], const int it) {
    const double cal = g_t96.cross_cs[it][0], sal = g_t96.cross_cs[it][1];
    const Vec3 b1 = {q[0][0], q[0][1], q[0][2]}, b2 = {q[1][0], q[1][1], q[1][2]};
    return {b1.x + b2.x, (b1.y + b2.y) * cal + (b1.z - b2.z) * sal, -(b1.y - b2.y) * sal + (b1.z + b2.z) * cal};
}

static __device__ __noinline__ Vec3 t96_loops_of(const double (*p)[3], const int il) {
    const double st = g_t96.loop_cs[il][0], ct = g_t96.loop_cs[il][1];
    const double sp = g_t96.loop_cs[il][2], cp = g_t96.loop_cs[il][3];
    double bxs;
    Vec3 q = {p[0][0], p[0][1], p[0][2]};
    bxs = q.x * ct + q.z * st;
    const double bz1 = q.z * ct - q.x * st;
    const double bx1 = bxs * cp - q.y * sp;
    const double by1 = bxs * sp + q.y * cp;
    q = {p[1][0], p[1][1], p[1][2]};
    bxs = q.x * ct + q.z * st;
    const double bz2 = q.z * ct - q.x * st;
    const double bx2 = bxs * cp + q.y * sp;
    const double by2 = -bxs * sp + q.y * cp;
    q = {p[2][0], p[2][1], p[2][2]};
    bxs = q.x * ct + q.z * st;
    const double bz3 = q.z * ct - q.x * st;
    const double bx3 = -bxs * cp - q.y * sp;
    const double by3 = bxs * sp - q.y * cp;
    q = {p[3][0], p[3][1], p[3][2]};
    bxs = q.x * ct + q.z * st;
    return {bx1 + bx2 + bx3 + (-bxs * cp + q.y * sp), by1 + by2 + by3 + (-bxs * sp - q.y * cp),
            bz1 + bz2 + bz3 + (q.z * ct - q.x * st)};
}

__device__ __forceinline__ void t96_sum_loops(T96Slot& s, const int c) {
    constexpr double C1[14] = {-0.911582E-03, -0.376654E-02, -0.727423E-02, -0.270084E-02, -0.123899E-02,
                               -0.154387E-02, -0.340040E-02, -0.191858E-01, -0.518979E-01, 0.635061E-01,
                               0.440680, -0.396570, -89.5587, 23.2806};
    const double z = s.pl[2];
    double b = 0.0;
#pragma unroll
    for (int i = 0; i < 12; i++) {
        const int f = g_lop_first[i], two = g_lop_first[i + 1] - f;
        const double* p = s.lop[f];
        const double u = p[c], w = c == 2 ? p[3] : z;
        double b2 = 0.0;
        if (two == 2) {
            const double* r = s.lop[f + 1];
            b2 = r[c] * (c == 2 ? r[3] : z);
        }
        b += C1[i] * __fma_rn(u, w, b2);
    }
    const Vec3 o = t96_cross_of(&s.cir[0], 0);
    b += C1[12] * comp(o, c);
    b += C1[13] * s.cir[2][c];
    s.tl[c] = b;
}

__device__ __forceinline__ void t96_sum_cyl(T96Slot& s, const int c) {
    double b = 0.0;
    for (int i = 0; i < 6; i++) b = b + s.bes[i][c][0] * s.bes[i][c][1];
    s.cyl[c] = b;
}

__device__ __forceinline__ void t96_sum_rt(T96Slot& s, const bool tail, const int c) {
    double b = 0.0;
    const int i0 = tail ? 2 : 0, i1 = tail ? 6 : 2;
    for (int i = i0; i < i1; i++) b = b + s.rt[i][c][0] * s.rt[i][c][1];
    if (tail) s.tail[c] = b;
    else s.ring[c] = b;
}

__device__ __forceinline__ void t96_sum_t87(T96Slot& sl) {
    const double z = sl.z;
    const double zp = z - 40.0, zm = z + 40.0;
    const double *c = sl.t87[0], *p = sl.t87[1], *m = sl.t87[2];
    const double aln = 0.25 * (p[4] + m[4] - 2. * c[4]);
    sl.tail87[0] = 0.391734 * (z * c[0] - 0.5 * (zp * p[0] + zm * m[0])) + 5.89715 * (z * c[1] - 0.5 * (zp * p[1] + zm * m[1])) +
                   24.6833 * (z * c[2] - 0.5 * (zp * p[2] + zm * m[2]));
    const double g1 = c[3] - 0.5 * (p[3] + m[3]);
    const double g2 = __dadd_rn(__dmul_rn(c[5], c[6]), -0.5 * __fma_rn(p[5], p[6], __dmul_rn(m[5], m[6])));
    sl.tail87[1] = __fma_rn(24.6833, g2, __fma_rn(0.391734, aln, __dmul_rn(5.89715, g1)));
}

static __device__ __noinline__ void t96_sum_outer(T96Slot& s) {
    const Vec3 d1 = t96_cross_of(&s.cir[3], 1);
    const Vec3 d2 = t96_cross_of(&s.cir[5], 2);
    const Vec3 d3 = t96_cross_of(&s.cir[7], 3);
    const Vec3 d4 = {s.cir[9][0], s.cir[9][1], s.cir[9][2]};
    const Vec3 d5 = t96_loops_of(&s.cir[10], 1);
    s.ro[0] = -34.105 * d1.x + -2.00019 * d2.x + 628.639 * d3.x + 73.4847 * d4.x + 12.5162 * d5.x;
    s.ro[1] = -34.105 * d1.y + -2.00019 * d2.y + 628.639 * d3.y + 73.4847 * d4.y + 12.5162 * d5.y;
    s.ro[2] = -34.105 * d1.z + -2.00019 * d2.z + 628.639 * d3.z + 73.4847 * d4.z + 12.5162 * d5.z;
}

static __device__ __noinline__ void t96_sum_inner(T96Slot& s) {
    const Vec3 d8 = t96_loops_of(&s.cir[3], 0);
    constexpr double CB[5] = {154.185, -2.12446, 0.601735E-01, -.153954E-02, .355077E-04};
    const double(*h)[3] = s.inn;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        double b = __fma_rn(CB[0], h[0][c], __dmul_rn(CB[1], h[1][c]));
#pragma unroll
        for (int m = 2; m < 5; m++) b = b + CB[m] * h[m][c];
        s.ri[c] = b + 29.9996 * h[5][c] + 262.886 * h[6][c] + 99.9132 * comp(d8, c);
    }
}

// r2_birk's mix of the sub-fields of its band.
static __device__ __noinline__ Vec3 t96_r2mix(const T96Slot& s) {
    const double dl = 0.03, dl1 = 0.015;
    const double xks = s.xks;
    const int band = s.band;
    const Vec3 qo = {s.ro[0], s.ro[1], s.ro[2]}, qs = {s.sheet[0], s.sheet[1], s.sheet[2]},
               qi = {s.ri[0], s.ri[1], s.ri[2]};
    if (band == 0) return {qo.x * -0.02, qo.y * -0.02, qo.z * -0.02};
    if (band == 1) {
        const double f2 = -0.02 * t96_tksi(xks, -dl, dl1);
        const double f1 = -0.02 - f2;
        return {qo.x * f1 + qs.x * f2, qo.y * f1 + qs.y * f2, qo.z * f1 + qs.z * f2};
    }
    if (band == 2) return {qs.x * -0.02, qs.y * -0.02, qs.z * -0.02};
    if (band == 3) {
        const double f1 = -0.02 * t96_tksi(xks, dl, dl1);
        const double f2 = -0.02 - f1;
        return {qi.x * f1 + qs.x * f2, qi.y * f1 + qs.y * f2, qi.z * f1 + qs.z * f2};
    }
    return {-qi.x * 0.02, -qi.y * 0.02, -qi.z * 0.02};
}

// t96_birk1_mix at the slot's edge points.
static __device__ __noinline__ Vec3 t96_slot_blend(const T96Slot& s) {
    const bool south = (s.flags & kT96South) != 0;
    const double* b1 = south ? s.tc : s.tl;
    const double* b2 = south ? s.tl : s.tc;
    const double dx2 = s.e2[0] - s.e1[0], dy2 = s.e2[1] - s.e1[1], dz2 = s.e2[2] - s.e1[2];
    const double ss = sqrt(__fma_rn(dz2, dz2, __fma_rn(dx2, dx2, __dmul_rn(dy2, dy2))));
    const double dx = s.x - s.e1[0], dy = s.y - s.e1[1], dz = s.z - s.e1[2];
    const double ds = sqrt(__fma_rn(dz, dz, __fma_rn(dx, dx, __dmul_rn(dy, dy))));
    const double frac = ds / ss, f1 = 1.0 - frac;
    return {__fma_rn(b1[0], f1, __dmul_rn(b2[0], frac)), __fma_rn(b1[1], f1, __dmul_rn(b2[1], frac)),
            __fma_rn(b1[2], f1, __dmul_rn(b2[2], frac))};
}

// t96_field's sum inside the magnetopause.
static __device__ __noinline__ Vec3 t96_slot_inside(const T96Slot& s) {
    const T96Cond& c = *s.c;
    const Vec3 cf = {s.cyl[0], s.cyl[1], s.cyl[2]};
    const Vec3 rc = {s.shield[0][0] + s.ring[0], s.shield[0][1] + s.ring[1], s.shield[0][2] + s.ring[2]};
    const Vec3 t2 = {s.shield[1][0] + s.tail[0], s.shield[1][1] + s.tail[1], s.shield[1][2] + s.tail[2]};
    const Vec3 t3 = {s.shield[2][0] + s.tail87[0], s.shield[2][1], s.shield[2][2] + s.tail87[1]};
    Vec3 b = {0.0, 0.0, 0.0};
    if (s.flags & kT96Blend) b = t96_slot_blend(s);
    else if (s.flags & kT96Loops) b = {s.tl[0], s.tl[1], s.tl[2]};
    else if (s.flags & kT96Con) b = {s.tc[0], s.tc[1], s.tc[2]};
    const Vec3 r1 = {b.x + s.shield[3][0], b.y + s.shield[3][1], b.z + s.shield[3][2]};
    Vec3 r2 = {s.shield[4][0], s.shield[4][1], s.shield[4][2]};
    const Vec3 r2h = t96_r2mix(s);
    r2.x += r2h.x;
    r2.y += r2h.y;
    r2.z += r2h.z;
    const Vec3 im = {s.shield[5][0], s.shield[5][1], s.shield[5][2]};
    const double rimfy = im.y * c.ct + im.z * c.st;
    const double rimfz = im.z * c.ct - im.y * c.st;
    const double fx = cf.x * c.xappa3 + c.rcampl * rc.x + c.tampl2 * t2.x + c.tampl3 * t3.x + c.b1ampl * r1.x +
                      c.b2ampl * r2.x + c.rimfampl * im.x;
    const double fy = cf.y * c.xappa3 + c.rcampl * rc.y + c.tampl2 * t2.y + c.tampl3 * t3.y + c.b1ampl * r1.y +
                      c.b2ampl * r2.y + c.rimfampl * rimfy;
    const double fz = cf.z * c.xappa3 + c.rcampl * rc.z + c.tampl2 * t2.z + c.tampl3 * t3.z + c.b1ampl * r1.z +
                      c.b2ampl * r2.z + c.rimfampl * rimfz;
    return {fx, fy, fz};
}

// t96_field's end (the quad).  The dipole's sums are rounded as the compiler
// rounds them in its two places there.
static __device__ __noinline__ Vec3 t96_slot_end(const T96Slot& s) {
    const double x = s.X, y = s.Y, z = s.Z, sigma = s.sigma, oimfy = s.oimfy, oimfz = s.oimfz;
    if (sigma < 1.08 - 0.005) return t96_slot_inside(s);
    const bool outside = sigma >= 1.08 + 0.005;
    const double p = __dmul_rn(x, x), t = __dmul_rn(y, y), u = __dmul_rn(z, z);
    const double tu = __dadd_rn(t, u), pt = __dadd_rn(p, t);
    const double ptu = sqrt(__dadd_rn(pt, u));
    const double q = 30574.0 / (ptu * ptu * ptu * ptu * ptu);
    const double z3 = 3.0 * z, e = __dadd_rn(tu, -2.0 * p);
    const double qx = q * (outside ? __dadd_rn(e, -__dmul_rn(z3, x)) : __fma_rn(-z3, x, e));
    const double qya = -3.0 * y * q, qzb = __dadd_rn(pt, -2.0 * u);   // q.y = qya z, q.z = q qzb
    if (outside) return {-qx, __fma_rn(-qya, z, oimfy), __fma_rn(-q, qzb, oimfz)};
    const Vec3 f = t96_slot_inside(s);
    const double fint = 0.5 * (1.0 - div_c(sigma - 1.08, 0.005, 1.0 / 0.005));
    const double fext = 0.5 * (1.0 + div_c(sigma - 1.08, 0.005, 1.0 / 0.005));
    const double my = __fma_rn(oimfy, fext, __dmul_rn(__fma_rn(qya, z, f.y), fint));
    const double mz = __fma_rn(oimfz, fext, __dmul_rn(__fma_rn(q, qzb, f.z), fint));
    return {__fma_rn(__dadd_rn(f.x, qx), fint, -qx), __fma_rn(-qya, z, my), __fma_rn(-q, qzb, mz)};
}

}  // namespace cor
