// team.cuh -- block-cooperative trajectory steps: a block of eight warps holds
// up to 32 trajectories ("slots") and spreads every field evaluation over all
// of its threads.
//
// An FP64 warp instruction holds its sub-partition for 64 cycles however many
// lanes are active, four sub-partitions together retire one per 19 cycles, and
// instruction-level parallelism gains nothing (measured; the pipe is the
// bound).  So a scan with fewer trajectories than the GPU has lanes is bound
// by the number of warp instructions of one trajectory's step, 31 of 32 lanes
// idle in the limit.  Here
//   * four neighbouring lanes (a quad) hold one slot's state, replicated; the
//     three components of the RK step and independent quotients go to
//     different lanes of the quad;
//   * the field evaluation is cut into tasks -- independent terms of the same
//     form (columns and terms of the spherical harmonics, ...) -- that
//     warps take 32 at a time, tasks of all slots together, so that lanes are
//     full whatever branches the slots' positions take;
//   * sums are then taken in the reference's order by one lane per sum.
// Every operation is the one-lane code's on the same operands, so results do
// not move by a bit.
//
// Measured (IGRF-14): a lone trajectory's accepted step 126 us by one lane,
// 39.6 us by a team; one site of 400 rigidities, limit 2,500 steps, 331-507 ms
// and 100 ms; 8,000 trajectories, limit 1,000 steps, 243 ms and 79 ms.  A lone
// step is bound by the quad's trials (about 110 FP64 instructions each, 3.9
// per step) and the 105-term sums, a full block by the FP64 pipe.
#pragma once

#include <type_traits>

#include "trace.cuh"

namespace cor {
// One component of a vector by number.
__device__ __forceinline__ double comp(const Vec3 v, const int c) { return c == 0 ? v.x : c == 1 ? v.y : v.z; }
}  // namespace cor

#include "team_t96.cuh"
#include "team_ts05.cuh"

namespace cor {

constexpr int kTeamThreads = 256;
constexpr int kTeamWarps = kTeamThreads / 32;
constexpr int kTeamSlots = 32;                 // one bit each in a warp's masks
constexpr int kTeamSharedBytes = 224 * 1024;   // of 227 KB, TeamShared besides

// Threads of a block of n slots: eight warps, or six for a few slots, whose
// warps mostly find the chunk counters run out (1,000 T96 steps of one
// trajectory 58.4 ms with eight, 56.4 with six; 400 trajectories at three
// slots each 60.6 and 58.6; at 13 slots and more six are 3-5 % slower).
constexpr int team_threads(const int n_slots) { return n_slots <= 4 ? 192 : kTeamThreads; }
static_assert(6 * kTeamSlots <= kTeamThreads && 6 * 4 <= team_threads(4), "team_field's last phase is one pass");
constexpr unsigned kFull = 0xffffffffu;

// ---- quad helpers ---------------------------------------------------------
__device__ __forceinline__ double quad_get(const double v, const int q) {
    return __shfl_sync(kFull, v, (threadIdx.x & 28) | q);
}

__device__ __forceinline__ Vec3 quad_gather(const double v) {
    return {quad_get(v, 0), quad_get(v, 1), quad_get(v, 2)};
}

// rk_velocity with one component per lane: stage k's cross product needs the
// two other components of the stage velocity, which the quad exchanges.
template <bool PLAIN>
__device__ __forceinline__ Vec3 quad_rk_velocity(const double h, const double d, const Vec3 f, const Vec3 v,
                                                 const int c) {
    const int c1 = c == 2 ? 0 : c + 1, c2 = c == 0 ? 2 : c - 1;
    const double f1 = comp(f, c1), f2 = comp(f, c2);
    const double vc = comp(v, c);
#define CROSS(S1, S2) (h * (d * ((S1)*f2 - (S2)*f1)))
#define OTHERS(S) const double S##p = quad_get(S, c1), S##q = quad_get(S, c2)
    const double a1 = CROSS(comp(v, c1), comp(v, c2));
    const double s2 = vc + DIV3(a1);
    OTHERS(s2);
    const double a2 = CROSS(s2p, s2q);
    const double s3 = rk_3<PLAIN>(vc, a1, a2);
    OTHERS(s3);
    const double a3 = CROSS(s3p, s3q);
    const double s4 = rk_4<PLAIN>(vc, a1, a2, a3);
    OTHERS(s4);
    const double a4 = CROSS(s4p, s4q);
    const double s5 = rk_5<PLAIN>(vc, a1, a2, a3, a4);
    OTHERS(s5);
    const double a5 = CROSS(s5p, s5q);
    const double s6 = rk_6<PLAIN>(vc, a1, a2, a3, a4);
    OTHERS(s6);
    const double a6 = CROSS(s6p, s6q);
#undef CROSS
#undef OTHERS
    return quad_gather(vc + DIV192(23. * a1 + 125. * a3 - 81. * a5 + 125. * a6));
}

template <bool PLAIN>
__device__ __forceinline__ Vec3 quad_rk_position(const double h, const Vec3 v, const Vec3 x, const int c) {
    return quad_gather(rk_position_1<PLAIN>(h, comp(v, c), comp(x, c)));
}

// One component of geo_to_gsm and gsm_to_geo: the quad's lanes take one each
// and gather.  With the end of the internal field and the turn's two scalar
// products split the same way, a lone trajectory's step went from 41.5 us to
// 39.6 (IGRF-14) and from 57.2 to 52.9 (T96).
__device__ __forceinline__ double gsm_comp(const Vec3 g, const cor_model_params* __restrict__ p, const int c) {
    const double* a = c == 0 ? p->a1 : c == 1 ? p->a2 : p->a3;
    return __ldg(&a[0]) * g.x + __ldg(&a[1]) * g.y + __ldg(&a[2]) * g.z;
}

__device__ __forceinline__ double geo_comp(const Vec3 s, const cor_model_params* __restrict__ p, const int c) {
    return __ldg(&p->a1[c]) * s.x + __ldg(&p->a2[c]) * s.y + __ldg(&p->a3[c]) * s.z;
}

// t / nk0 for nk0 = nk1 2^k, given r1 = RN(1 / nk1): the quotient by nk1 in
// three operations, then an exact shift of its exponent, where both are
// normal numbers (else the division itself).
__device__ __forceinline__ double gyro_step(const double t, const int nk1, const double r1, const int nk0) {
    const double h1 = div_r(t, (double)nk1, r1);
    const int k = __clz(nk1) - __clz(nk0);
    const int ex = (int)((to_bits(h1) >> 52) & 0x7ff);
    if ((nk1 << k) == nk0 && ex > k && ex < 0x7ff) return from_bits(to_bits(h1) - ((long long)k << 52));
    return t / nk0;
}

// lane_advance for the slots of a warp, one quad each: every lane of the warp
// calls it, `run` says whether the lane's quad holds a trajectory.  The trial
// loop runs while any quad of the warp has a trial to make, with the others'
// lanes computing on without effect.  Returns the class of run lanes' quads.
template <bool PLAIN>
__device__ __forceinline__ int quad_advance(Lane& L, const TraceArgs& a, bool run) {
    const int q = threadIdx.x & 3, c = q == 3 ? 2 : q;
    const double zn = run ? L.job->zn : 1.;
    const int nk1 = run ? L.job->nk1 : 1;
    const cor_model_params* __restrict__ p = run ? &L.par->p : &a.params->p;
    // per trajectory and per step what the trials share; h = t / (nk1 2^k) is
    // the correctly rounded t / nk1 scaled by a power of two
    const double dq = 1.E-09 * zn * kQ, tb = fabs(zn) * kQ * L.b, r1 = 1. / nk1;
    int st = 0;
    while (__any_sync(kFull, run)) {
        bool trial = run;
        double h = 0.;
        Vec3 nv = {0., 0., 0.};
        while (__any_sync(kFull, trial)) {
            const double vc = DIVC(L.v);
            const double hm = a.mass / sqrt(1. - vc * vc);
            // t and d in one division: lanes 0, 1 and lanes 2, 3
            const double td = (q < 2 ? 2. * kPi * hm : dq) / (q < 2 ? tb : hm);
            const double t = quad_get(td, 0), d = quad_get(td, 2);
            const double hh = gyro_step(t, nk1, r1, L.nk0);
            const Vec3 n = quad_rk_velocity<PLAIN>(hh, d, L.field, L.vel, c);
            // |n|^2 by lanes 0, 1 and the cosine's numerator by lanes 2, 3
            const Vec3 w = q < 2 ? n : L.vel;
            const double nw = n.x * w.x + n.y * w.y + n.z * w.z;
            const double n2 = quad_get(nw, 0), nv0 = quad_get(nw, 2);
            if (trial) {
                L.step++;
                if (vc > 1.) {
                    st = COR_TRAJ_SUPERLUM;
                    trial = run = false;
                } else {
                    const double vprev = L.v;
                    L.trials++;
                    L.v = sqrt(n2);
                    const bool reject = turn_rejects(a, nv0, L.v * vprev);
                    if (reject && L.nk0 <= 50000) {
                        L.nk0 *= 2;
                        L.step--;
                    } else {
                        h = hh;
                        nv = n;
                        trial = false;
                    }
                }
            }
            __syncwarp();
        }
        const Vec3 np = quad_rk_position<PLAIN>(h, L.vel, L.pos, c);
        const Vec3 gsm = quad_gather(gsm_comp(np, p, c));
        if (run) {
            const double rr = sqrt(np.x * np.x + np.y * np.y + np.z * np.z);
            const double pax = div_c(DIVRE(gsm.x) + 25.3, 36.08, 1. / 36.08);
            const double paz = DIVRE2(gsm.y * gsm.y + gsm.z * gsm.z);
            const double r = DIVRE(rr);
            const double paus = pax * pax + div_c(paz, 459.6736, 1. / 459.6736);
            if (r >= 25. || paus > 1.) {
                if ((r >= 25. && fabs(r - 25.) < 0.002) || (r <= 25. && paus > 1. && fabs(paus - 1.) < 0.002)) {
                    L.pos = np;
                    L.vel = nv;
                    st = COR_TRAJ_ALLOWED;
                    run = false;
                } else if (L.nk0 >= kNk0Cap) {
                    st = COR_TRAJ_WATCHDOG;
                    run = false;
                } else {
                    L.nk0 *= 2;
                    L.step--;
                }
            } else {
                const Vec3 prev = L.pos;
                L.pos = np;
                L.vel = nv;
                run = false;
                if (r < 1.) {
                    st = COR_TRAJ_REENTRY;
                } else if ((uint64_t)L.step > a.step_limit) {
                    st = COR_TRAJ_STEP_LIMIT;
                } else {
                    L.gsm = gsm;
                    L.time = L.time + h;
                    L.alength += sqrt((np.x - prev.x) * (np.x - prev.x) + (np.y - prev.y) * (np.y - prev.y) +
                                      (np.z - prev.z) * (np.z - prev.z));
                    L.nk0 = nk1;
                }
            }
        }
        __syncwarp();
    }
    return st;
}

// ---- the internal field in tasks ---------------------------------------------
constexpr int kShTerms = 105;   // (m, n), 1 <= m <= n <= 14, at n(n-1)/2 + m - 1 in the tables
constexpr int kShCols = 14;

// Where a slot keeps term (m, m) if it goes up to n = K: column by column, as
// the sums take the terms, without gaps.
__device__ __forceinline__ int sh_at(const int m, const int K) { return (m - 1) * (K + 1) - m * (m - 1) / 2; }

// What internal_geo keeps in registers, for one slot.
struct ShSlot {
    double x, y, z;                      // GEO position [R_E]
    double R, rho;
    double C, S, cf, sf, pp;
    double pw[kShCols], pwn[kShCols];    // R^-(n+1), n R^-(n+1)
    double cm[kShCols], sm[kShCols];     // cos/sin of (m-1) phi
    double pmm[kShCols], dmm[kShCols];   // the diagonal
    double q[kShTerms], z_[kShTerms];    // P(n,m), dP(n,m)
    double a1[kShTerms], a2[kShTerms], a3[kShTerms];
    double sum[2 + kShCols];             // br, bt, and each order's share of bf
    const cor_model_params* p;
    int K;
    int pole;
};

static __device__ const unsigned char c_sh_n[kShTerms] = {
    1,  2,  2,  3,  3,  3,  4,  4,  4,  4,  5,  5,  5,  5,  5,  6,  6,  6,  6,  6,  6,  7,  7,  7,  7,  7,  7,
    7,  8,  8,  8,  8,  8,  8,  8,  8,  9,  9,  9,  9,  9,  9,  9,  9,  9,  10, 10, 10, 10, 10, 10, 10, 10, 10,
    10, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 11, 12, 12, 12, 12, 12, 12, 12, 12, 12, 12, 12, 12, 13, 13, 13,
    13, 13, 13, 13, 13, 13, 13, 13, 13, 13, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14, 14};

// The geometry of a slot, by its quad (all lanes of the warp call; want: the
// quad's slot is evaluated): the two square roots and the five quotients on
// different lanes.  A quotient's correctly rounded value does not depend on
// how it is computed (div_r in internal_geo, a division here).
__device__ __forceinline__ void quad_sh_geometry(ShSlot& s, const Vec3 x, const cor_model_params* p, const bool want) {
    const int q = threadIdx.x & 3;
    const double rho2 = x.x * x.x + x.y * x.y;
    const double r2 = rho2 + x.z * x.z;
    const double root = sqrt(q & 1 ? rho2 : r2);
    const double R = quad_get(root, 0), rho = quad_get(root, 1);
    const double quo = (q == 0 ? x.z : q == 1 ? rho : q == 2 ? x.x : x.y) / (q < 2 ? R : rho);
    const double C = quad_get(quo, 0), S = quad_get(quo, 1), cx = quad_get(quo, 2), sx = quad_get(quo, 3);
    const double pp = 1. / R;
    if (want && q == 0) {
        const bool pole = S < 1.E-5;
        s.x = x.x;
        s.y = x.y;
        s.z = x.z;
        s.R = R;
        s.rho = rho;
        s.C = C;
        s.S = S;
        s.cf = pole ? 1. : cx;
        s.sf = pole ? 0. : sx;
        s.pp = pp;
        int nm = 3 + 30 / ((int)R + 2);
        if (nm > 13) nm = 13;
        s.K = nm + 1;
        s.pole = pole;
        s.p = p;
    }
}

// a b + c, with one rounding where internal_geo's is contracted.
template <bool FMA>
__device__ __forceinline__ double sh_mad(const double a, const double b, const double c) {
    return FMA ? __fma_rn(a, b, c) : __dadd_rn(__dmul_rn(a, b), c);
}

// Chains that every column starts from, one lane per slot and chain (three
// kinds of task, taken by different warps).
__device__ __forceinline__ void sh_powers(ShSlot& s) {
    const double pp = s.pp;
    double pr = pp;
    for (int n = 1; n <= s.K; n++) {
        pr = pr * pp;
        s.pw[n - 1] = pr;
        s.pwn[n - 1] = pr * n;
    }
}

template <bool FMA>
__device__ __forceinline__ void sh_rotations(ShSlot& s) {
    const double cf = s.cf, sf = s.sf;
    double cm = 0., sm = 1.;
    for (int m = 1; m <= s.K; m++) {
        if (m != 1) {
            const double w = cm;
            cm = sh_mad<FMA>(w, cf, __dmul_rn(sm, sf));
            sm = sh_mad<FMA>(sm, cf, -__dmul_rn(w, sf));
        }
        s.cm[m - 1] = cm;
        s.sm[m - 1] = sm;
    }
}

template <bool FMA>
__device__ __forceinline__ void sh_diagonal(ShSlot& s) {
    const double C = s.C, S = s.S;
    double pmm = 1., dmm = 0.;
    for (int m = 1; m <= s.K; m++) {
        s.pmm[m - 1] = pmm;
        s.dmm[m - 1] = dmm;
        dmm = sh_mad<FMA>(C, pmm, __dmul_rn(S, dmm));
        pmm = S * pmm;
    }
}

// One column (order m - 1) of the Legendre recursion.
template <bool FMA>
__device__ __forceinline__ void sh_column(ShSlot& s, const int m) {
    const double C = s.C, S = s.S;
    const int K = s.K;
    const double* __restrict__ REC = s.p->rec;
    double q = s.pmm[m - 1], zz = s.dmm[m - 1], p2 = 0., d2 = 0.;
    int i = m * (m - 1) / 2 + m - 1, j = sh_at(m, K);
    double next = __ldg(&REC[i]);
    for (int n = m; n <= K; n++) {
        s.q[j] = q;
        s.z_[j++] = zz;
        if (n < K) {
            const double xk = next;
            if (n + 1 < K) next = __ldg(&REC[i + n]);
            const double dp = sh_mad<FMA>(-xk, d2, sh_mad<FMA>(C, zz, -__dmul_rn(S, q)));
            const double pm = sh_mad<FMA>(C, q, -__dmul_rn(xk, p2));
            d2 = zz;
            p2 = q;
            zz = dp;
            q = pm;
        }
        i += n;
    }
}

// The factors of term i that multiply P and dP in the three sums.
template <bool FMA>
__device__ __forceinline__ void sh_term(ShSlot& s, const int i) {
    const int n = c_sh_n[i], m = i - n * (n - 1) / 2 + 1, j = sh_at(m, s.K) + n - m;
    const double an = s.pw[n - 1];
    const double sm = s.sm[m - 1], cm = s.cm[m - 1];
    const double e = __ldg(&s.p->g[i]);
    const double hh = __ldg(&s.p->h[i]);
    const double w = sh_mad<FMA>(e, sm, __dmul_rn(hh, cm));
    s.a1[j] = s.pwn[n - 1] * w;
    s.a2[j] = -(an * w);
    s.a3[j] = an * sh_mad<FMA>(e, cm, -__dmul_rn(hh, sm));
}

// Without contraction the sums add rounded products, which are then taken
// term by term beforehand.
__device__ __forceinline__ void sh_product(ShSlot& s, const int i) {
    const double q = s.q[i], z = s.z_[i];
    s.a1[i] = s.a1[i] * q;
    s.a2[i] = s.a2[i] * z;
    s.a3[i] = s.a3[i] * (s.pole ? z : q);
}

constexpr int kShBatch = 7;

// One of the sums of internal_geo in its order: br (0), bt (1), or the share
// of order m - 1 in bf (m = 2 .. K).  The two long ones bound their phase:
// 10,700 cycles for 105 terms when each addition waited for its own loads,
// with the terms in the sums' order and loads ahead of them a lone IGRF
// trajectory's step went from 42.8 us to 41.5.
template <bool FMA>
__device__ __forceinline__ void sh_sum(ShSlot& s, const int which) {
    const int K = s.K;
    const double* A = which == 0 ? s.a1 : which == 1 ? s.a2 : s.a3;
    const double* B = which == 1 || (which >= 2 && s.pole) ? s.z_ : s.q;
    const int end = which < 2 ? K * (K + 1) / 2 : which <= K ? sh_at(which + 1, K) : 0;
    int j = which < 2 ? 0 : which <= K ? sh_at(which, K) : 0;
    double acc = 0.;
    // loads in batches: one at a time, each waits for the addition before it
    for (; j + kShBatch <= end; j += kShBatch) {
        double a[kShBatch], b[kShBatch];
#pragma unroll
        for (int k = 0; k < kShBatch; k++) {
            a[k] = A[j + k];
            if (FMA) b[k] = B[j + k];
        }
#pragma unroll
        for (int k = 0; k < kShBatch; k++) acc = FMA ? __fma_rn(a[k], b[k], acc) : __dadd_rn(acc, a[k]);
    }
    for (; j < end; j++) acc = FMA ? __fma_rn(A[j], B[j], acc) : __dadd_rn(acc, A[j]);
    if (which >= 2) acc = __dmul_rn(acc, which - 1);   // rounded before it is added, in both kinds of unit
    s.sum[which] = acc;
}

// The end of internal_geo, by the quad: component c.
template <bool FMA>
__device__ __forceinline__ double sh_finish(const ShSlot& s, const int c) {
    const double br = s.sum[0], bt = s.sum[1], C = s.C, S = s.S, cf = s.cf, sf = s.sf;
    double bf = 0., bphi;
#pragma unroll
    for (int m = 2; m <= kShCols; m++) {
        if (m > s.K) break;
        bf = bf + s.sum[m];
    }
    if (s.pole) {
        if (C < 0.) bf = -bf;
        bphi = bf;
    } else {
        bphi = bf / S;
    }
    const double he = sh_mad<FMA>(br, S, __dmul_rn(bt, C));
    return sh_mad<FMA>(c < 2 ? he : br, c == 0 ? cf : c == 1 ? sf : C,
                       __dmul_rn(c < 2 ? bphi : bt, c == 0 ? -sf : c == 1 ? cf : -S));
}

// ---- the block's task loop ----------------------------------------------------
// Shared state of a team block besides the slots.
struct TeamShared {
    unsigned next[4];                       // chunk counters of the phases
    unsigned char need[32];                 // slots whose field is evaluated in this pass
    unsigned char list[kTeamWarps][6][32];  // slots by kind of task, one copy per warp
};

// The slots set in `mask` as this warp's list k.
__device__ __forceinline__ const unsigned char* team_list(TeamShared& ts, const int k, const unsigned mask) {
    const int lane = threadIdx.x & 31;
    unsigned char* l = ts.list[threadIdx.x >> 5][k];
    if ((mask >> lane) & 1u) l[__popc(mask & ((1u << lane) - 1u))] = (unsigned char)lane;
    return l;
}

// The next chunk of the phase, for the whole warp.
__device__ __forceinline__ unsigned next_chunk(unsigned* ctr) {
    unsigned c = 0;
    if ((threadIdx.x & 31) == 0) c = atomicAdd(ctr, 1u);
    return __shfl_sync(kFull, c, 0);
}

// Whether the phase's chunk ch is one of the next n; if not, ch counts on
// from there.
__device__ __forceinline__ bool takes(unsigned& ch, const unsigned n) {
    if (ch < n) return true;
    ch -= n;
    return false;
}

__device__ __forceinline__ unsigned chunks(const int tasks) { return (unsigned)(tasks + 31) >> 5; }

// The units of sets with an external model are compiled with FMA contraction.
template <class MS>
constexpr bool kFma = MS::external != 0;

struct NoSlot {};
template <class MS>
struct TeamSlotBody {
    std::conditional_t<MS::internal != 0, ShSlot, NoSlot> sh;
    std::conditional_t<MS::external == COR_EXTERNAL_T96, T96Slot, NoSlot> t96;
    std::conditional_t<MS::external == COR_EXTERNAL_TS05, TS05Slot, NoSlot> ts05;
};
// An odd number of 8-byte words, so that slots start in different banks.
template <class MS>
struct TeamSlot : TeamSlotBody<MS> {
    double pad[1 + (sizeof(TeamSlotBody<MS>) / 8) % 2];
};

// Slots per block, at most.  With an external model as many as shared memory
// holds (19 with T96, 29 with TS05): most kinds of task are a few per slot, a
// chunk of them costs its 32 lanes whether they are filled or not, and blocks
// of 128 threads and 8 slots, two to an SM, filled 8 to 24 (3,573 TS05
// trajectories of 400 steps 173 ms with those, 135 with one block of 16
// slots, 96 with 24; 8,000 T96 trajectories of 250 steps 110, 94 and, with 18
// slots, 81).  The internal field alone has enough terms to fill its chunks,
// and two blocks of 16 slots overlap one's steps with the other's fields
// (8,000 trajectories of 1,000 steps: 81 ms; one block of 32 slots 96, two of
// 12 106).
template <class MS>
constexpr int kTeamSlotsOf = MS::external == 0 ? 16
                             : kTeamSharedBytes / (int)sizeof(TeamSlot<MS>) < kTeamSlots
                                 ? kTeamSharedBytes / (int)sizeof(TeamSlot<MS>)
                                 : kTeamSlots;

// The field of the slots in `mask` (not 0), from what the quads wrote.  All
// threads of the block; the phases are separated by block barriers, and
// within one the warps take chunks of 32 tasks, the longest kinds first.
template <class MS>
__device__ __forceinline__ void team_field(TeamShared& ts, TeamSlot<MS>* slots, const unsigned mask) {
    constexpr bool kSh = MS::internal != 0, kT96 = MS::external == COR_EXTERNAL_T96,
                   kTS05 = MS::external == COR_EXTERNAL_TS05;
    const int lane = threadIdx.x & 31;
    const int n = __popc(mask);
    const unsigned char* list = team_list(ts, 0, mask);
    __syncwarp();
    // phase 1
    for (;;) {
        unsigned ch = next_chunk(&ts.next[0]);
        bool any = false;
        if constexpr (kT96) {
            any = true;
            if (takes(ch, chunks(2 * n))) {
                const int t = (int)ch * 32 + lane;
                t96_task_b1(slots[list[t < 2 * n ? t >> 1 : 0]].t96, t < 2 * n);
            } else if (takes(ch, chunks(6 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 6 * n) t96_task_rt(slots[list[t % n]].t96, t / n);
            } else if (takes(ch, chunks(6 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 6 * n) t96_task_bes(slots[list[t % n]].t96, t / n);
            } else if (takes(ch, chunks(3 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 3 * n) t96_task_t87(slots[list[t % n]].t96, t / n);
            } else if (takes(ch, 1)) {
                if (lane < n) t96_task_xksi(slots[list[lane]].t96);
            } else if (takes(ch, 1)) {
                if (lane < n) t96_task_main(slots[list[lane]].t96);
            } else if (takes(ch, chunks(kT96Sc * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < kT96Sc * n) t96_task_sc(slots[list[t % n]].t96, t / n);
            } else {
                any = false;
            }
        }
        if constexpr (kTS05) {
            any = true;
            if (takes(ch, chunks(4 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 4 * n) ts05_task_shield(slots[list[t % n]].ts05, t / n);
            } else if (takes(ch, 1)) {
                if (lane < n) {
                    TS05Slot& s = slots[list[lane]].ts05;
                    put3(s.cf, ts05_shlcar3x3(s.x, s.y, s.z));
                }
            } else if (takes(ch, chunks(2 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 2 * n) ts05_task_birk(slots[list[t >> 1]].ts05, t & 1);
            } else if (takes(ch, chunks(2 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 2 * n) ts05_task_symm(slots[list[t >> 1]].ts05, t & 1);
            } else if (takes(ch, 1)) {
                if (lane < n) ts05_task_quad(slots[list[lane]].ts05);
            } else if (takes(ch, 1)) {
                if (lane < n) ts05_task_warp(slots[list[lane]].ts05);
            } else if (takes(ch, 1)) {
                if (lane < n) ts05_task_main(slots[list[lane]].ts05);
            } else {
                any = false;
            }
        }
        if constexpr (kSh) {
            if (!any) {
                any = true;
                if (ch < 3) {
                    if (lane < n) {
                        ShSlot& s = slots[list[lane]].sh;
                        if (ch == 0) sh_rotations<kFma<MS>>(s);
                        else if (ch == 1) sh_diagonal<kFma<MS>>(s);
                        else sh_powers(s);
                    }
                } else {
                    any = false;
                }
            }
        }
        __syncwarp();
        if (!any) break;
    }
    __syncthreads();
    // phase 2
    int nl = 0, nc = 0, no = 0, ni = 0, ns = 0;
    const unsigned char *ll = list, *lc = list, *lo = list, *li = list, *ls = list;
    if constexpr (kT96) {
        unsigned fl = 0;
        int band = 2;
        bool in = false;
        if ((mask >> lane) & 1u) {
            const T96Slot& s = slots[lane].t96;
            fl = s.flags;
            band = s.band;
            in = !(s.sigma >= 1.08 + 0.005);
        }
        const unsigned ml = __ballot_sync(kFull, in && (fl & kT96Loops)), mc = __ballot_sync(kFull, in && (fl & kT96Con));
        const unsigned mo = __ballot_sync(kFull, in && band <= 1), mi = __ballot_sync(kFull, in && band >= 3);
        const unsigned ms = __ballot_sync(kFull, in && band >= 1 && band <= 3);
        ll = team_list(ts, 1, ml);
        lc = team_list(ts, 2, mc);
        lo = team_list(ts, 3, mo);
        li = team_list(ts, 4, mi);
        ls = team_list(ts, 5, ms);
        nl = __popc(ml);
        nc = __popc(mc);
        no = __popc(mo);
        ni = __popc(mi);
        ns = __popc(ms);
        __syncwarp();
    }
    if constexpr (kTS05) {
        const unsigned mc = __ballot_sync(kFull, ((mask >> lane) & 1u) && slots[lane].ts05.sigma < 1.1960 + 0.005);
        lc = team_list(ts, 2, mc);
        nc = __popc(mc);
        __syncwarp();
    }
    // the columns in pairs of complementary length where the slots fill the
    // warps that way
    const bool pairs = n > 2;
    const int cols = pairs ? kShCols / 2 : kShCols;
    for (;;) {
        unsigned ch = next_chunk(&ts.next[1]);
        bool any = false;
        if constexpr (kT96) {
            any = true;
            const int ncir = 3 * nl + 11 * no + 4 * ni;
            if (takes(ch, ns ? 3 : 0)) {
                if (lane < ns) {
                    T96Slot& s = slots[ls[lane]].t96;
                    if (ch == 0) t96_task_sheet<0>(s);
                    else if (ch == 1) t96_task_sheet<1>(s);
                    else t96_task_sheet<2>(s);
                }
            } else if (takes(ch, chunks(5 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 5 * nc) t96_task_con(slots[lc[t % nc]].t96, t / nc);
            } else if (takes(ch, chunks(7 * ni))) {
                const int t = (int)ch * 32 + lane;
                if (t < 7 * ni) t96_task_inner(slots[li[t % ni]].t96, t / ni);
            } else if (takes(ch, chunks(ncir))) {
                const int t = (int)ch * 32 + lane;
                if (t < 3 * nl) t96_task_circle(slots[ll[t % nl]].t96, t / nl, false);
                else if (t - 3 * nl < 11 * no) t96_task_circle(slots[lo[(t - 3 * nl) % no]].t96, 3 + (t - 3 * nl) / no, false);
                else if (t < ncir)
                    t96_task_circle(slots[li[(t - 3 * nl - 11 * no) % ni]].t96, 3 + (t - 3 * nl - 11 * no) / ni, true);
            } else if (takes(ch, chunks(kT96Dip * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < kT96Dip * nc) t96_task_dip(slots[lc[t % nc]].t96, t / nc);
            } else if (takes(ch, chunks(kT96Exp * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < kT96Exp * n) t96_task_exp(slots[list[t % n]].t96, t / n);
            } else if (takes(ch, chunks(kT96Lop * nl))) {
                const int t = (int)ch * 32 + lane;
                if (t < kT96Lop * nl) t96_task_lop(slots[ll[t % nl]].t96, t / nl);
            } else {
                any = false;
            }
        }
        if constexpr (kTS05) {
            any = true;
            if (takes(ch, chunks(4 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 4 * nc) ts05_task_cone(slots[lc[t % nc]].ts05, t / nc);
            } else if (takes(ch, chunks(4 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 4 * nc) ts05_task_ap(slots[lc[t % nc]].ts05, 1, t / nc);
            } else if (takes(ch, chunks(3 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 3 * nc) ts05_task_br(slots[lc[t % nc]].ts05, t / nc);
            } else if (takes(ch, chunks(3 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 3 * nc) ts05_task_bt(slots[lc[t % nc]].ts05, t / nc);
            } else if (takes(ch, chunks(2 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 2 * nc) ts05_task_disk(slots[lc[t >> 1]].ts05, t & 1);
            } else if (takes(ch, chunks(4 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 4 * nc) ts05_task_ap(slots[lc[t % nc]].ts05, 0, t / nc);
            } else if (takes(ch, chunks(20 * nc))) {
                const int t = (int)ch * 32 + lane;
                if (t < 20 * nc) ts05_task_sc(slots[lc[t % nc]].ts05, t / nc);
            } else {
                any = false;
            }
        }
        if constexpr (kSh) {
            if (!any) {
                any = true;
                if (takes(ch, chunks(n * cols))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < n * cols) {
                        ShSlot& s = slots[list[t % n]].sh;
                        const int c = t / n, K = s.K;
                        if (pairs) {
                            if (2 * c < K) {
                                sh_column<kFma<MS>>(s, c + 1);
                                if (K - 1 - c > c) sh_column<kFma<MS>>(s, K - c);
                            }
                        } else if (c < K) {
                            sh_column<kFma<MS>>(s, c + 1);
                        }
                    }
                } else if (takes(ch, chunks(n * kShTerms))) {
                    // the terms' factors need only the chains
                    const int t = (int)ch * 32 + lane;
                    if (t < n * kShTerms) {
                        ShSlot& s = slots[list[t % n]].sh;
                        const int i = t / n;
                        if (i < s.K * (s.K + 1) / 2) sh_term<kFma<MS>>(s, i);
                    }
                } else {
                    any = false;
                }
            }
        }
        __syncwarp();
        if (!any) break;
    }
    __syncthreads();
    if (threadIdx.x == 0) ts.next[0] = 0;
    if constexpr (kSh && !kFma<MS>) {
        for (;;) {
            const unsigned ch = next_chunk(&ts.next[2]);
            if (ch >= chunks(n * kShTerms)) break;
            const int t = (int)ch * 32 + lane;
            if (t < n * kShTerms) {
                ShSlot& s = slots[list[t % n]].sh;
                const int i = t / n;
                if (i < s.K * (s.K + 1) / 2) sh_product(s, i);
            }
            __syncwarp();
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) ts.next[1] = 0;
    // phase 3: the sums, the two long ones of the internal field first
    for (;;) {
        unsigned ch = next_chunk(&ts.next[3]);
        bool any = false;
        if constexpr (kSh) {
            any = true;
            if (takes(ch, chunks(2 * n))) {
                const int t = (int)ch * 32 + lane;
                if (t < 2 * n) sh_sum<kFma<MS>>(slots[list[t >> 1]].sh, t & 1);
            } else if (takes(ch, chunks(n * (kShCols - 1)))) {
                const int t = (int)ch * 32 + lane;
                if (t < n * (kShCols - 1)) sh_sum<kFma<MS>>(slots[list[t % n]].sh, 2 + t / n);
            } else {
                any = false;
            }
        }
        if constexpr (kTS05) {
            if (!any) {
                any = true;
                if (takes(ch, chunks(50 * nc))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 50 * nc) ts05_task_exp(slots[lc[t % nc]].ts05, t / nc);
                } else if (takes(ch, chunks(2 * nc))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 2 * nc) ts05_end_birk(slots[lc[t >> 1]].ts05, t & 1);
                } else if (takes(ch, chunks(2 * nc))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 2 * nc) ts05_end_symm(slots[lc[t >> 1]].ts05, t & 1);
                } else if (takes(ch, nc ? 1 : 0)) {
                    if (lane < nc) ts05_end_quad(slots[lc[lane]].ts05);
                } else {
                    any = false;
                }
            }
        }
        if constexpr (kT96) {
            if (!any) {
                any = true;
                if (takes(ch, chunks(3 * nc))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 3 * nc) t96_sum_con(slots[lc[t % nc]].t96, t / nc);
                } else if (takes(ch, chunks(3 * nl))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 3 * nl) t96_sum_loops(slots[ll[t % nl]].t96, t / nl);
                } else if (takes(ch, no ? 1 : 0)) {
                    if (lane < no) t96_sum_outer(slots[lo[lane]].t96);
                } else if (takes(ch, ni ? 1 : 0)) {
                    if (lane < ni) t96_sum_inner(slots[li[lane]].t96);
                } else if (takes(ch, chunks(18 * n))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 18 * n) {
                        const int k = t / n;
                        t96_sum_shield(slots[list[t % n]].t96, k / 3, k % 3);
                    }
                } else if (takes(ch, 1)) {
                    if (lane < n) t96_sum_t87(slots[list[lane]].t96);
                } else if (takes(ch, chunks(3 * n))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 3 * n) t96_sum_cyl(slots[list[t % n]].t96, t / n);
                } else if (takes(ch, chunks(6 * n))) {
                    const int t = (int)ch * 32 + lane;
                    if (t < 6 * n) {
                        const int k = t / n;
                        t96_sum_rt(slots[list[t % n]].t96, k >= 3, k % 3);
                    }
                } else {
                    any = false;
                }
            }
        }
        __syncwarp();
        if (!any) break;
    }
    __syncthreads();
    if constexpr (kTS05) {
        const int t = (int)threadIdx.x;   // one pass: at most 6 tasks per slot
        if (t < 6 * nc) {
            const int k = t / nc;
            ts05_sum5(slots[lc[t % nc]].ts05, k / 3, k % 3);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) ts.next[2] = ts.next[3] = 0;
}

// What a quad writes for its slot before team_field and reads after it (all
// lanes of the warp call, with any par; need: the quad's slot is evaluated).
template <class MS>
__device__ __forceinline__ void team_begin(TeamSlot<MS>& s, const Vec3 pos, const DevParams* par, const bool need) {
    if constexpr (MS::internal != 0) {
        const int q = threadIdx.x & 3, c = q == 3 ? 2 : q;
        const Vec3 geo = quad_gather(geo_comp(pos, &par->p, c));
        quad_sh_geometry(s.sh, need ? geo : Vec3{1., 0., 0.}, need ? &par->p : nullptr, need);
    }
    if constexpr (MS::external == COR_EXTERNAL_T96) {
        if (need && (threadIdx.x & 3) == 0) t96_slot_start(s.t96, par->t96, pos);
    }
    if constexpr (MS::external == COR_EXTERNAL_TS05) {
        if (need && (threadIdx.x & 3) == 0) ts05_slot_start(s.ts05, par->ts05, pos);
    }
    __syncwarp();
}

template <class MS>
__device__ __forceinline__ Vec3 team_end(const TeamSlot<MS>& s, const DevParams* par, const bool need) {
    const cor_model_params* p = &par->p;
    const int q = threadIdx.x & 3, c = q == 3 ? 2 : q;
    double tot = 0.;
    if constexpr (MS::internal != 0) {
        double b = 0.;
        if (need) b = sh_finish<kFma<MS>>(s.sh, c);
        __syncwarp();
        tot += gsm_comp(quad_gather(b), p, c);
    }
    if constexpr (MS::external == COR_EXTERNAL_T96) {
        if (need) tot += comp(t96_slot_end(s.t96), c);
        __syncwarp();
    }
    if constexpr (MS::external == COR_EXTERNAL_TS05) {
        if (need) tot += comp(ts05_slot_end(s.ts05), c);
        __syncwarp();
    }
    return quad_gather(geo_comp(quad_gather(tot), p, c));
}

// The field at n points by teams (field_kernel's arguments): block b takes
// points b n_slots .. and on.
template <class MS>
__global__ void __launch_bounds__(kTeamThreads)
    team_field_kernel(const DevParams* __restrict__ params, const int n_params, const int32_t* __restrict__ pidx,
                      const double* __restrict__ pos, const int64_t n, double* __restrict__ out, const int n_slots) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ TeamShared ts;
    TeamSlot<MS>* slots = reinterpret_cast<TeamSlot<MS>*>(s_dyn);
    const int tid = threadIdx.x, slot = tid >> 2;
    if (tid < 4) ts.next[tid] = 0;
    for (int64_t i0 = (int64_t)blockIdx.x * n_slots; i0 < n; i0 += (int64_t)gridDim.x * n_slots) {
        const int64_t i = i0 + slot;
        const bool need = slot < n_slots && i < n;
        const DevParams* par = params;
        const bool warp_need = __any_sync(kFull, need);
        if (warp_need) {
            Vec3 x = {0., 0., 0.};
            if (need) {
                const int k = pidx ? pidx[i] : 0;
                par = params + (k < 0 || k >= n_params ? 0 : k);
                x = {DIVRE(pos[3 * i]), DIVRE(pos[3 * i + 1]), DIVRE(pos[3 * i + 2])};
            }
            __syncwarp();
            team_begin<MS>(slots[slot < n_slots ? slot : 0], x, par, need);
        }
        const int64_t left = n - i0;
        const int m = left < n_slots ? (int)left : n_slots;
        __syncthreads();
        team_field<MS>(ts, slots, m == 32 ? kFull : (1u << m) - 1u);
        if (warp_need) {
            const Vec3 b = team_end<MS>(slots[slot < n_slots ? slot : 0], par, need);
            if (need && (tid & 3) == 0) {
                out[3 * i] = b.x;
                out[3 * i + 1] = b.y;
                out[3 * i + 2] = b.z;
            }
        }
    }
}

// The scan by teams: one generation, as trace_kernel's.  `n_slots` (at most
// kTeamSlotsOf<MS>) trajectories per block.

template <class MS>
__global__ void __launch_bounds__(kTeamThreads) team_trace_kernel(const TraceArgs a, const int n_slots) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    __shared__ TeamShared ts;
    TeamSlot<MS>* slots = reinterpret_cast<TeamSlot<MS>*>(s_dyn);
    const int tid = threadIdx.x, slot = tid >> 2, q = tid & 3;
    if (tid < 4) ts.next[tid] = 0;
    if (tid < 32) ts.need[tid] = 0;
    __syncthreads();
    Lane L;
    L.v = 0.;
    L.b = 1.;
    L.nk0 = 1;
    L.vel = L.pos = L.field = L.gsm = Vec3{0., 0., 0.};
    L.par = a.params;
    bool has = false, done = slot >= n_slots;
    unsigned long long n_steps = 0, n_trials = 0, n_traj = 0, n_wd = 0;
    const bool rig_major = a.rig_major && (!a.grid_ok || *(volatile const unsigned int*)a.grid_ok != 0u);
    for (;;) {
        bool need = false;
        if (__any_sync(kFull, has)) {
            const int st = quad_advance<kPlain<MS>>(L, a, has);
            if (has) {
                if (st == 0) {
                    need = true;
                    if (a.step_records && L.step <= a.step_cap && q == 0) {
                        cor_step_record r;
                        r.gsm[0] = L.gsm.x; r.gsm[1] = L.gsm.y; r.gsm[2] = L.gsm.z;
                        r.pos[0] = L.pos.x; r.pos[1] = L.pos.y; r.pos[2] = L.pos.z;
                        r.v = L.v;
                        r.time = L.time;
                        r.length = L.alength;
                        r.step = L.step;
                        r.reserved = 0;
                        a.step_records[L.traj * a.step_cap + (L.step - 1)] = r;
                    }
                } else {
                    if (q == 0) {
                        lane_finish(L, a, st);
                        n_steps += (st == COR_TRAJ_ALLOWED) ? L.step - 1 : L.step;
                        n_trials += L.trials;
                        n_traj += 1;
                        n_wd += (st == COR_TRAJ_WATCHDOG);
                    }
                    has = false;
                }
            }
            __syncwarp();
        }
        bool want = !has && !done;
        if (a.n_restore) {
            uint64_t r = queue_pop(&a.gen->restore_cursor, want && q == 0);
            r = __shfl_sync(kFull, (unsigned long long)r, tid & 28);
            if (want && r < a.n_restore) {
                need = lane_restore(L, a.restore[r], a.jobs, a.params);
                has = true;
                want = false;
            }
        }
        uint64_t t = queue_pop(a.queue, want && q == 0);
        t = __shfl_sync(kFull, (unsigned long long)t, tid & 28);
        if (want) {
            if (t < a.n_traj) {
                lane_init(L, a, t, rig_major);
                has = true;
                need = true;
            } else {
                done = true;
            }
        }
        __syncwarp();
        const bool warp_need = __any_sync(kFull, need);
        if (warp_need) {
            Vec3 pos = {0., 0., 0.};
            if (need) pos = {DIVRE(L.gsm.x), DIVRE(L.gsm.y), DIVRE(L.gsm.z)};
            team_begin<MS>(slots[slot < n_slots ? slot : 0], pos, L.par, need);
        }
        if (q == 0 && slot < 32) ts.need[slot] = need;
        if (__syncthreads_and(done)) break;
        const unsigned mask = __ballot_sync(kFull, ts.need[tid & 31] != 0);
        if (!mask) {
            __syncthreads();
            continue;
        }
        team_field<MS>(ts, slots, mask);
        if (warp_need) {
            const Vec3 f = team_end<MS>(slots[slot < n_slots ? slot : 0], L.par, need);
            if (need) {
                L.field = f;
                L.b = 1.E-09 * sqrt(L.field.x * L.field.x + L.field.y * L.field.y + L.field.z * L.field.z);
            }
            __syncwarp();
        }
    }
    warp_add_u64(reinterpret_cast<unsigned long long*>(&a.counters->accepted_steps), n_steps);
    warp_add_u64(reinterpret_cast<unsigned long long*>(&a.counters->trials), n_trials);
    warp_add_u64(reinterpret_cast<unsigned long long*>(&a.counters->trajectories), n_traj);
    warp_add_u64(reinterpret_cast<unsigned long long*>(&a.counters->watchdog), n_wd);
}

}  // namespace cor
