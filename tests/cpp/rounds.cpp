// The rounds in which the one-CTA-per-trotter sweep decides a batch of 32 trials
// (dense_multi.cu), restated for one batch on the host with the kernel's own decision
// functions (mc_trial.h).  For every combination of an algorithm, a step (G, beta) and
// a scale of the couplings, ordinary and extreme, it checks that the rounds end, and,
// where the fields stay finite in fp32, that each trial gets the outcome of the same trials
// taken one after another in FP64.  Prints the number of batches; exits 1 on a failure.
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <limits>
#include <vector>

#include "mc_trial.h"

using namespace sq103;

static uint64_t rngState = 12345;
static double uniform() {
    rngState = rngState * 6364136223846793005ull + 1442695040888963407ull;
    return (double)(rngState >> 40) / (double)(1 << 24);
}

struct Trial {
    int x, sum;  // site among kSites, sum of the neighbours' spins
    bool unknown[2];
    float u;
};
constexpr int kSites = 40, kLanes = 32;

struct Batch {
    bool sa;
    int m;
    float G, beta;
    float J[kSites][kSites], h[kSites], q[kSites], F[kSites];
    Trial t[kLanes];
};

// FP64 decision of a trial with field F
static bool outcome64(const Batch &B, double q, double h, double F, int sum, float u) {
    const double t = h + 2. * F;
    double dE, rate;
    if (B.sa) {
        dE = 2. * q * t;
        rate = 1. / (double)B.G;
    } else {
        const double coef = std::log(std::tanh((double)B.G * B.beta / B.m)) / B.beta;
        dE = 2. / B.m * q * t - q * sum * coef;
        rate = B.beta;
    }
    return dE < 0. || std::exp(-dE * rate) > (double)u;
}

// the trials one after another; fields in FP64
static unsigned sequential(const Batch &B) {
    double F[kSites], q[kSites];
    for (int i = 0; i < kSites; ++i) F[i] = B.F[i], q[i] = B.q[i];
    unsigned acc = 0;
    for (int l = 0; l < kLanes; ++l) {
        const int x = B.t[l].x;
        if (!outcome64(B, q[x], B.h[x], F[x], B.t[l].sum, B.t[l].u)) continue;
        acc |= 1u << l;
        for (int i = 0; i < kSites; ++i) F[i] -= 2. * q[x] * B.J[x][i];
        q[x] = -q[x];
    }
    return acc;
}

// the rounds; false if they do not end
static bool rounds(const Batch &B, unsigned &accBits, int &exact) {
    const float twoDivM = 2.f / B.m;
    const float coef = B.sa ? 0.f : logf(tanhf(B.G * B.beta / B.m)) / B.beta;
    const float rate = fminf(B.sa ? 1.f / B.G : B.beta, std::numeric_limits<float>::max());  // (step_const)
    const McConst c = mc_const(B.sa, twoDivM, coef, rate);
    float L[kLanes], qx[kLanes], c2[kLanes], zA[kLanes], tol[kLanes];
    bool unknown[kLanes][2];
    double F64[kSites], q64[kSites];  // what the exact warp sums
    for (int i = 0; i < kSites; ++i) F64[i] = B.F[i], q64[i] = B.q[i];
    for (int l = 0; l < kLanes; ++l) {
        const Trial &t = B.t[l];
        L[l] = mc_L(c, t.u > 0.f ? -logf(t.u) : INFINITY);
        qx[l] = B.q[t.x];
        c2[l] = 2.f * c.cz * qx[l];
        zA[l] = fmaf(c.cz * qx[l], fmaf(2.f, B.F[t.x], B.h[t.x]), -L[l]);
        tol[l] = fmaf(fabsf(c.cz) * 1.52587890625e-5f, fabsf(B.h[t.x]) + 2.f * fabsf(B.F[t.x]) + 1.f, mc_tol(c, L[l]));
        for (int n = 0; n < 2; ++n) unknown[l][n] = !B.sa && t.unknown[n];
    }
    unsigned pending = ~0u;
    accBits = 0;
    exact = 0;
    // a lane waits for its neighbours once, is decided in FP64 once, flips once
    for (int round = 0; round < 3 * kLanes + 2; ++round) {
        int fa = 32, fb = 32;
        for (int l = kLanes - 1; l >= 0; --l) {
            if (!((pending >> l) & 1u)) continue;
            int known = B.t[l].sum, n = unknown[l][0] + unknown[l][1];
            if (n == 2) known = 0;
            if (n == 1) known = B.t[l].sum == 0 ? (unknown[l][0] ? 1 : -1) : B.t[l].sum / 2;
            const float cbq = c.cb * qx[l], z = zA[l] - cbq * (float)known, sp = fabsf(cbq) * (float)n;
            if (mc_accepts(z, sp, tol[l]))
                fa = l;
            else if (mc_open(z, sp, tol[l]))
                fb = l;
        }
        if (fb < fa) {
            pending &= ~((1u << fb) - 1u);
            if (unknown[fb][0] || unknown[fb][1]) {
                unknown[fb][0] = unknown[fb][1] = false;
            } else {
                const Trial &t = B.t[fb];
                mc_answer(outcome64(B, q64[t.x], B.h[t.x], F64[t.x], t.sum, t.u), zA[fb], tol[fb]);
                ++exact;
            }
            continue;
        }
        if (fa == 32) return true;
        accBits |= 1u << fa;
        pending &= fa == 31 ? 0u : ~((2u << fa) - 1u);
        const int xf = B.t[fa].x;
        const float df = -2.f * qx[fa];
        for (int i = 0; i < kSites; ++i) F64[i] += (double)df * B.J[xf][i];
        q64[xf] = -q64[xf];
        if (!pending) return true;
        for (int l = fa + 1; l < kLanes; ++l) {
            const float dJ = df * B.J[xf][B.t[l].x];
            zA[l] = fmaf(c2[l], dJ, zA[l]);
            tol[l] = fmaf(2.f * fabsf(c.cz) * 1.52587890625e-5f, fabsf(dJ), tol[l]);
            if (B.t[l].x == xf) {
                qx[l] = -qx[l];
                c2[l] = -c2[l];
                zA[l] = -(zA[l] + L[l]) - L[l];
            }
        }
    }
    return false;
}

int main() {
    const float inf = std::numeric_limits<float>::infinity(), nan = std::numeric_limits<float>::quiet_NaN();
    const float Gs[] = {5.f, 0.05f, 1e-3f, 1e-30f, 1e-39f, 0.f, -0.f, -1.f, inf, nan};
    const float betas[] = {50.f, 1e-3f, 0.f, 1e30f, 3e38f, inf, -2.f, nan};
    const float scales[] = {1.f, 0.f, 1e-20f, 1e6f, 1e30f, 3e38f, inf, nan};
    long long batches = 0, exactTotal = 0;
    for (int sa = 0; sa < 2; ++sa)
        for (float G : Gs)
            for (float beta : betas)
                for (float scale : scales)
                    for (int rep = 0; rep < 6; ++rep) {
                        Batch B;
                        B.sa = sa;
                        B.m = 2 + 7 * rep;
                        B.G = G;
                        B.beta = beta;
                        const bool one = !(std::fabs(scale) <= 1e20f);  // one coupling of that size, the rest ordinary
                        for (int i = 0; i < kSites; ++i) {
                            B.h[i] = (float)(uniform() - 0.5) * (one ? 1.f : scale);
                            B.q[i] = uniform() < 0.5 ? -1.f : 1.f;
                            for (int j = 0; j <= i; ++j)
                                B.J[i][j] = B.J[j][i] = i == j ? 0.f : (float)(uniform() - 0.5) * 0.5f * (one ? 1.f : scale);
                        }
                        if (one) B.J[3][5] = B.J[5][3] = scale;
                        for (int i = 0; i < kSites; ++i) {
                            double f = 0.;
                            for (int j = 0; j < kSites; ++j) f += (double)B.J[i][j] * B.q[j];
                            B.F[i] = (float)f;
                        }
                        for (Trial &t : B.t) {
                            t.x = (int)(uniform() * (rep & 1 ? 8 : kSites));
                            t.sum = 2 * (int)(uniform() * 3) - 2;
                            t.unknown[0] = uniform() < 0.3;
                            t.unknown[1] = uniform() < 0.3;
                            t.u = uniform() < 0.004 ? 0.f : (float)uniform();
                        }
                        unsigned acc;
                        int exact;
                        ++batches;
                        const bool ended = rounds(B, acc, exact);
                        exactTotal += exact;
                        const bool finite = std::fabs(scale) <= 1e36f;
                        // (u = 0 accepts every finite rate dE in fp32; in FP64 those below 745)
                        bool zeroU = false;
                        for (const Trial &t : B.t) zeroU |= t.u == 0.f;
                        const bool same = !finite || zeroU || acc == sequential(B);
                        if (!ended || !same) {
                            printf("%s: sa=%d G=%g beta=%g scale=%g m=%d\n", ended ? "other outcomes" : "rounds do not end",
                                   sa, G, beta, scale, B.m);
                            return 1;
                        }
                    }
    printf("%lld batches, %lld FP64 decisions\n", batches, exactTotal);
    return 0;
}
