// step_host.cpp -- TEST INFRASTRUCTURE: one step of a trajectory (lane_advance,
// trace.cuh) compiled as host C++ in both of its forms: the one of the units
// without contraction, with fewer operations, and the general one.
// tests/test_step_forms.py builds this file and calls it via ctypes.
#include "cuda_shim.h"

#include "../../cor-model_gb300/csrc/model_prep.h"
#include "../../cor-model_gb300/csrc/trace.cuh"

using namespace cor;

extern "C" {

// n steps, each from its own state in[16 i ..]: position, velocity, field, B, v,
// time, length, zn, nk1, nk0.  out[12 i ..]: class, position, velocity, v, time,
// length, nk0, step.
void host_step(int plain, const cor_model_params* p, double tu_angle, double gc_reject, double gc_half, double mass,
               uint64_t step_limit, const double* in, int64_t n, double* out) {
    DevParams dp;
    prepare_params(p, 1, &dp);
    TraceArgs a;
    memset(&a, 0, sizeof a);
    a.step_limit = step_limit;
    a.tu_angle = tu_angle;
    a.turn_exact = 1;
    a.gc_reject = gc_reject;
    a.gc_half = gc_half;
    a.mass = mass;
    for (int64_t i = 0; i < n; i++) {
        const double* s = in + 16 * i;
        cor_scan_job job;
        memset(&job, 0, sizeof job);
        job.zn = s[13];
        job.nk1 = (int32_t)s[14];
        Lane L;
        memset(&L, 0, sizeof L);
        L.pos = {s[0], s[1], s[2]};
        L.vel = {s[3], s[4], s[5]};
        L.field = {s[6], s[7], s[8]};
        L.b = s[9];
        L.v = s[10];
        L.time = s[11];
        L.alength = s[12];
        L.nk0 = (int)s[15];
        L.job = &job;
        L.par = &dp;
        const int st = plain ? lane_advance<true>(L, a) : lane_advance<false>(L, a);
        double* o = out + 12 * i;
        const double r[12] = {(double)st, L.pos.x, L.pos.y, L.pos.z, L.vel.x, L.vel.y, L.vel.z, L.v, L.time, L.alength,
                              (double)L.nk0, (double)L.step};
        memcpy(o, r, sizeof r);
    }
}

}  // extern "C"
