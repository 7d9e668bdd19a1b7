// mc_trial.h -- the decision of one trial in the rounds of the one-CTA-per-trotter
// sweep (dense_multi.cu), for the device and, in its test, the host.
//
// A trial accepts when z = rate dE - L < 0, L = -ln u.  z = zA - ring with
// zA = cz q (h + 2F) - L and ring = cb q (qL + qR); unknown neighbour spins leave it
// in [z - sp, z + sp].  It is decided where that interval lies outside [-tol, tol],
// the bound on its fp32 error, and otherwise waits for its neighbours or for its
// FP64 outcome.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define SQ103_HD __host__ __device__ __forceinline__
#else
#define SQ103_HD inline
#endif

namespace sq103 {

// largest factor of the fp32 form: its products with fields up to 1e23 stay finite, so that
// the flips of a batch add up (an infinite z would stay so)
constexpr float kMcCap = 1e15f;
constexpr float kMcMaxL = 1e30f;

// A step's constants: dE's factors of h + 2F and of the spin sum times the rate, the
// largest L, and the part of the tolerance that depends on neither the field nor L.
struct McConst {
    float cz, cb, maxL, tol;
};

// A step outside the fp32 form's range (a rate that is infinite, negative, NaN or too
// large: simulated annealing at G = 0, an infinite beta; a ring coefficient that is NaN or
// too large) gets constants that leave z = 0 within the tolerance, so that every trial
// takes its FP64 outcome.  With coef = -inf (SQA at G = 0, beta = 0) the sign of a nonzero
// spin sum decides, whatever the field, and a sum of zero takes its FP64 outcome.
SQ103_HD McConst mc_const(bool sa, float twoDivM, float coef, float rate) {
    McConst c;
    c.cz = rate * (sa ? 2.f : twoDivM);
    c.cb = sa ? 0.f : rate * coef;
    c.maxL = kMcMaxL;
    c.tol = 4e-6f * fabsf(c.cb) + 2e-6f;
    const bool ringOnly = !sa && coef == -INFINITY;
    if (!(c.cz >= 0.f && c.cz <= kMcCap && (ringOnly || fabsf(c.cb) <= kMcCap))) {
        c.cz = c.cb = c.maxL = 0.f;
        c.tol = kMcCap;
    } else if (ringOnly) {
        c.cz = 0.f;
        c.cb = -1e37f;
        c.tol = 1e37f;
    }
    return c;
}

// a trial's L = -ln u (+inf for u = 0) and tolerance without the field's part
SQ103_HD float mc_L(const McConst &c, float negLogU) { return fminf(negLogU, c.maxL); }
SQ103_HD float mc_tol(const McConst &c, float L) { return c.tol + 1e-6f * L; }

// certain to accept; neither certain to accept nor to reject (a NaN rejects)
SQ103_HD bool mc_accepts(float z, float sp, float tol) { return z + sp < -tol; }
SQ103_HD bool mc_open(float z, float sp, float tol) { return z - sp <= tol; }

// the trial's FP64 outcome: it is decided from here on, whatever its tolerance was
// (an infinite one, of an infinite field say, would leave it open round after round)
SQ103_HD void mc_answer(bool accept, float &zA, float &tol) {
    zA = accept ? -3e38f : 3e38f;
    tol = 0.f;
}

}  // namespace sq103
