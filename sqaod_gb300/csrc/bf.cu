// bf.cu -- brute-force QUBO search (dense and bipartite graphs).
//
// Dense: E(x) = x^T W x over packed states x (variable i at bit N-1-i,
// sqaodc/common/Common.cpp:79-93).  A state splits into hi = x >> L (the
// first N-L variables) and lo = x & (2^L - 1) (the last L variables,
// L = min(N, 14)):
//   E = E_hh(hi) + E_ll(lo) + sum_{b in lo} x_b C_hi[b],   C_hi[b] = 2 sum_{i in hi} W_{i,b}
// The search runs in three passes: fp32 minimum, collection of every x with
// E32 <= Emin32 + slack, and an FP64 re-evaluation of the candidates (tie-break)
// done by the caller through sq103_dense_bf_refine.  Runs of 64 whole hi values
// (2^20 states) take bf_run_pass, which holds E_ll in registers; the rest of a
// range takes bf_dense_pass: one CTA per hi value, E_ll from a 2^L table, the
// cross term as two table lookups over the halves of lo.  For integer-valued W every fp32 value is
// exact, so Emin and the argmin set equal the reference CPU searcher's
// (sqaodc/cpu/CPUDenseGraphBatchSearch.cpp:26-50).
//
// Bipartite: E(x0, x1) = b0.x0 + b1.x1 + x1^T W x0 (sqaodc/cpu/SharedFormulas.cpp:123-144).
// For one x1, D[j] = b0[j] + sum_{i in x1} W[i][j] and E is the sum of D over the
// bits of x0 plus b1.x1, so the minimum over all x0 is the sum of the negative
// D[j] (bf_bip_min); only the x1 whose minimum is within the slack are searched
// state by state (bf_bip_pass: one CTA per x1, 7-bit-group lookups over x0).  A
// range that does not hold every x0 is searched state by state in both passes.
#include <algorithm>
#include <cstdint>
#include <cstring>

#include "sq_common.cuh"
#include "sq_kernels.h"

namespace sq103 {

constexpr int kLoBits = 14;
constexpr int kBfThreads = 256;

constexpr int kRunBits = 6;                    // hi values per run of bf_run_pass: 64
constexpr int kRunShift = kLoBits + kRunBits;  // a run's states: 2^20
constexpr int kBfGroups = 2048;                // run minima kept (several runs share one in long ranges)

struct BfWorkspace {
    float ell[1 << kLoBits];
    unsigned int minEnc;
    int count;
    int pad[62];
    unsigned int groupMin[kBfGroups];
};

__device__ __forceinline__ unsigned int enc_float(float f) {
    unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float dec_float(unsigned int e) {
    unsigned int u = (e & 0x80000000u) ? (e & 0x7fffffffu) : ~e;
    return __uint_as_float(u);
}

__global__ void bf_init_ws(BfWorkspace *ws) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kBfGroups) ws->groupMin[i] = 0xffffffffu;
    if (i == 0) {
        ws->minEnc = 0xffffffffu;
        ws->count = 0;
    }
}

// E_ll table: lo bit b <-> variable N-1-b.  A CTA takes the 128 lo values that
// share their bits from 7 on: its threads sum the part of those bits, E(upper)
// and the row sums D[c] of the low seven over them, and each value then adds at
// most 28 terms (the 14 x 14 double loop per value took 30 us of FP64; this 7).
__global__ void __launch_bounds__(128) bf_lo_table(const float *W, int N, int L, BfWorkspace *ws) {
    __shared__ double D[7], eU;
    const int t = threadIdx.x, up = blockIdx.x << 7, lo = up | t;
    auto w = [&](int a, int b) { return (double)W[(size_t)(N - 1 - a) * N + (N - 1 - b)]; };
    if (t < 7) {
        double d = 0.;
        for (int b = 7; b < L; ++b)
            if ((up >> b) & 1) d += w(t, b) + w(b, t);
        D[t] = d;
    } else if (t == 32) {
        double e = 0.;
        for (int a = 7; a < L; ++a) {
            if (!((up >> a) & 1)) continue;
            for (int b = 7; b < L; ++b)
                if ((up >> b) & 1) e += w(a, b);
        }
        eU = e;
    }
    __syncthreads();
    if (lo >= (1 << L)) return;
    double e = eU;
    for (int a = 0; a < 7 && a < L; ++a) {
        if (!((t >> a) & 1)) continue;
        e += D[a] + w(a, a);
        for (int b = 0; b < a; ++b)
            if ((t >> b) & 1) e += w(a, b) + w(b, a);
    }
    ws->ell[lo] = (float)e;
}

// ------------------------------------------------------------- whole runs
// A run: 64 consecutive hi values hi = 64 r + u, all 2^14 lo values of each.  A
// thread keeps E_ll of the 64 lo values with its bits 5-12 (lane, warp) in
// registers, bits 0-4 and 13 varying, and per hi adds a 32-entry table over
// bits 0-4 and takes the minimum before the rest, common to the 32, is added:
//   E = (E_ll + tB[lo & 31]) + (tA1[lo >> 10] + tA2[(lo >> 5) & 31]),
// tA1 holding E_hh(hi).  That is one packed addition (two states) and one
// three-input minimum (two more states) per pair, the additions on the FMA pipe
// and the minima on the ALU, so a state costs about 1.5 instructions; the
// per-state lookups of bf_dense_pass cost about 15.  The sums over hi split into
// the run's upper bits (21 short FP64 sums per run) and tables over its six low
// bits (once per CTA).  The rounding is of the same count as bf_dense_pass's and
// exact where that is exact (integer W).
// PASS 0 keeps the minimum of each group of runs; PASS 1 reads them and collects
// x with E <= thr from the runs that have one, eight hi values per item.
// N = 31: 153 and 15 us (748 and 927 us with bf_dense_pass); the pipes of the additions
// and minima are then the limit (dispatch and math-throttle stalls lead).
struct RunShared {
    double t6C[64][kLoBits];  // sum over u's bits of 2 W[hi var][lo var]
    double t6E[64];           // E over u's bits alone
    double cU[kLoBits], dU[kRunBits], eU;
    alignas(16) float C[64][16];  // C_hi of each u; [14] = E_hh
    alignas(16) float tB[64][32];
    float tA2[64][32], tA1[64][16];
    unsigned int minEnc;
    int items[256], nItems;
};

__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float lo2(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// the tables of run r's hi values [u0, u1) (all threads of the CTA)
__device__ __forceinline__ void run_setup(RunShared &S, const float *W, int N, uint64_t r, int u0, int u1) {
    const int H = N - kLoBits, tid = threadIdx.x;
    const uint64_t hi = r << kRunBits;
    // upper bits c >= 6 of hi; hi bit c <-> variable H-1-c, lo bit t <-> variable N-1-t
    if (tid < kLoBits + kRunBits) {
        const int v = tid < kLoBits ? N - 1 - tid : H - 1 - (tid - kLoBits);
        double s = 0.;
        for (int c = kRunBits; c < H; ++c)
            if ((hi >> c) & 1ull) s += (double)W[(H - 1 - c) * N + v];
        (tid < kLoBits ? S.cU[tid] : S.dU[tid - kLoBits]) = 2. * s;
    } else if (tid >= 32 && tid < 64) {
        double e = 0.;
        for (int c = kRunBits + tid - 32; c < H; c += 32) {
            if (!((hi >> c) & 1ull)) continue;
            for (int d = kRunBits; d < H; ++d)
                if ((hi >> d) & 1ull) e += (double)W[(H - 1 - c) * N + (H - 1 - d)];
        }
        for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
        if (tid == 32) S.eU = e;
    }
    __syncthreads();
    for (int i = 16 * u0 + tid; i < 16 * u1; i += kBfThreads) {
        const int u = i >> 4, t = i & 15;
        if (t < kLoBits) S.C[u][t] = (float)(S.cU[t] + S.t6C[u][t]);
    }
    if (tid < u1 - u0) {
        const int u = u0 + tid;
        double e = S.eU + S.t6E[u];
#pragma unroll
        for (int c = 0; c < kRunBits; ++c)
            if ((u >> c) & 1) e += S.dU[c];
        S.C[u][kLoBits] = (float)e;
    }
    __syncthreads();
    // a warp per u, a lane per table entry
    const int warp = tid >> 5, v = tid & 31;
    for (int u = u0 + warp; u < u1; u += kBfThreads / 32) {
        const float *C = S.C[u];
        float sB = 0.f, s2 = 0.f, s1 = C[kLoBits];
#pragma unroll
        for (int b = 0; b < 5; ++b) {
            if ((v >> b) & 1) {
                sB = __fadd_rn(sB, C[b]);
                s2 = __fadd_rn(s2, C[5 + b]);
                if (b < 4) s1 = __fadd_rn(s1, C[10 + b]);
            }
        }
        S.tB[u][v] = sB;
        S.tA2[u][v] = s2;
        if (v < 16) S.tA1[u][v] = s1;
    }
    __syncthreads();
}

template <int PASS>
__global__ void __launch_bounds__(kBfThreads, 2) bf_run_pass(const float *Wg, int N, uint64_t rb, uint64_t re,
                                                             int groupShift, int subBits, float slack,
                                                             BfWorkspace *ws, uint64_t *cand, int cap) {
    extern __shared__ __align__(16) unsigned char bf_smem[];
    RunShared &S = *reinterpret_cast<RunShared *>(bf_smem);
    float *W = reinterpret_cast<float *>(bf_smem + sizeof(RunShared));  // N x N
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, H = N - kLoBits;
    const int kSub = 1 << subBits;  // work items per run
    const uint64_t nItems = (re - rb) << subBits;
    float thr = 0.f;
    if (PASS == 1) thr = dec_float(ws->minEnc) + slack;
    bool ready = false;
    unsigned long long ell[2][16];  // [lo bit 13][pairs over lo bits 0-4]
    // once per CTA: W, the tables over a run's six low hi bits, the thread's E_ll
    auto prepare = [&]() {
        for (int i = tid; i < N * N; i += kBfThreads) W[i] = Wg[i];
#pragma unroll
        for (int s = 0; s < 2; ++s) {
            const float4 *p = reinterpret_cast<const float4 *>(ws->ell + ((s << 13) | (warp << 10) | (lane << 5)));
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const float4 v = p[j];
                ell[s][2 * j] = ((unsigned long long)__float_as_uint(v.y) << 32) | __float_as_uint(v.x);
                ell[s][2 * j + 1] = ((unsigned long long)__float_as_uint(v.w) << 32) | __float_as_uint(v.z);
            }
        }
        __syncthreads();
        // by doubling: the u with highest bit c from the u below 2^c (FP64 is slow: few terms, full warps)
        if (tid < kLoBits) S.t6C[0][tid] = 0.;
        if (tid == 32) S.t6E[0] = 0.;
        for (int c = 0; c < kRunBits; ++c) {
            __syncthreads();
            const float *row = W + (H - 1 - c) * N;
            for (int i = tid; i < 16 << c; i += kBfThreads) {
                const int u = i >> 4, t = i & 15;
                if (t < kLoBits) S.t6C[(1 << c) + u][t] = S.t6C[u][t] + 2. * (double)row[N - 1 - t];
            }
            if (tid >= kBfThreads - (1 << c)) {
                const int u = kBfThreads - 1 - tid;
                double e = S.t6E[u] + (double)row[H - 1 - c];
                for (int d = 0; d < c; ++d)
                    if ((u >> d) & 1) e += 2. * (double)row[H - 1 - d];
                S.t6E[(1 << c) + u] = e;
            }
        }
        ready = true;
        __syncthreads();
    };
    if (PASS == 0) prepare();
    for (uint64_t i0 = blockIdx.x; i0 < nItems; i0 += PASS == 0 ? gridDim.x : (uint64_t)gridDim.x * kBfThreads) {
        int n = 1;
        if (PASS == 1) {
            // the items among the next 256 of this CTA whose runs hold a candidate
            if (tid == 0) S.nItems = 0;
            __syncthreads();
            const uint64_t it = i0 + (uint64_t)tid * gridDim.x;
            if (it < nItems && dec_float(ws->groupMin[(it >> subBits) >> groupShift]) <= thr)
                S.items[atomicAdd(&S.nItems, 1)] = tid;
            __syncthreads();
            n = S.nItems;
            if (n > 0 && !ready) prepare();
        } else if (tid == 0) {
            S.minEnc = 0xffffffffu;
        }
        for (int k = 0; k < n; ++k) {
            const uint64_t it = PASS == 0 ? i0 : i0 + (uint64_t)S.items[k] * gridDim.x;
            const uint64_t r = rb + (it >> subBits);
            const int nu = 64 >> subBits, u0 = (int)(it & (kSub - 1)) * nu, u1 = u0 + nu;
            run_setup(S, W, N, r, u0, u1);
            float lmin = __int_as_float(0x7f800000);
            for (int u = u0; u < u1; ++u) {
                const ulonglong2 *tB = reinterpret_cast<const ulonglong2 *>(S.tB[u]);
                float m0 = __int_as_float(0x7f800000), m1 = m0;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const ulonglong2 t = tB[j];
                    const unsigned long long a = add2(ell[0][2 * j], t.x), b = add2(ell[0][2 * j + 1], t.y);
                    const unsigned long long c = add2(ell[1][2 * j], t.x), d = add2(ell[1][2 * j + 1], t.y);
                    m0 = min3(min3(m0, lo2(a), hi2(a)), lo2(b), hi2(b));
                    m1 = min3(min3(m1, lo2(c), hi2(c)), lo2(d), hi2(d));
                }
                const float a2 = S.tA2[u][lane];
                const float r0 = __fadd_rn(S.tA1[u][warp], a2), r1 = __fadd_rn(S.tA1[u][8 + warp], a2);
                // (rounding is monotone: the minimum of the sums is the sum of the minimum)
                if (PASS == 0) {
                    lmin = min3(lmin, __fadd_rn(m0, r0), __fadd_rn(m1, r1));
                } else if (__fadd_rn(m0, r0) <= thr || __fadd_rn(m1, r1) <= thr) {
                    const uint64_t x0 = ((r << kRunBits) + u) << kLoBits | ((uint64_t)warp << 10) | ((uint64_t)lane << 5);
#pragma unroll
                    for (int s = 0; s < 2; ++s)
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const unsigned long long v = add2(ell[s][j], reinterpret_cast<const unsigned long long *>(S.tB[u])[j]);
                            const float rs = s ? r1 : r0;
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                if (__fadd_rn(h ? hi2(v) : lo2(v), rs) <= thr) {
                                    const int slot = atomicAdd(&ws->count, 1);
                                    if (slot < cap) cand[slot] = x0 | ((uint64_t)s << 13) | (uint64_t)(2 * j + h);
                                }
                        }
                }
            }
            if (PASS == 0) {
                for (int o = 16; o > 0; o >>= 1) lmin = fminf(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
                if (lane == 0) atomicMin(&S.minEnc, enc_float(lmin));
                __syncthreads();
                if (tid == 0) {
                    atomicMin(&ws->groupMin[(r - rb) >> groupShift], S.minEnc);
                    atomicMin(&ws->minEnc, S.minEnc);
                }
            }
            __syncthreads();  // the tables are rebuilt for the next item
        }
    }
}

// per-CTA set-up for the K consecutive hi values hi0 .. hi0 + K - 1 that are <= he:
// each hi value's set-up (C_hi, E_hh) runs in its own group of kBfThreads / K
// threads, all at once: base = E_hh(hi), C_hi, and the cross-term half tables
template <int K>
__device__ void bf_block_setup_k(const float *W, int N, int L, uint64_t hi0, uint64_t he, float *base,
                                 float (*tabHi)[128], float (*tabLo)[128], float (*C)[kLoBits], int Lh, int Ll) {
    static_assert(kBfThreads / K >= 64 && kBfThreads % K == 0, "a group needs two warps");
    constexpr int kGroup = kBfThreads / K;
    const int H = N - L;
    const int tid = threadIdx.x, g = tid / kGroup, t = tid % kGroup;
    const uint64_t hi = hi0 + g;
    if (hi <= he) {
        if (t < L) {
            double s = 0.;
            for (int c = 0; c < H; ++c)
                if ((hi >> c) & 1ull) s += (double)W[(size_t)(H - 1 - c) * N + (N - 1 - t)];
            C[g][t] = (float)(2. * s);
        }
        if (t >= 32 && t < 64) {
            double e = 0.;
            for (int c = t - 32; c < H; c += 32) {
                if (!((hi >> c) & 1ull)) continue;
                const float *row = W + (size_t)(H - 1 - c) * N;
                for (int d = 0; d < H; ++d)
                    if ((hi >> d) & 1ull) e += (double)row[H - 1 - d];
            }
            for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
            if (t == 32) base[g] = (float)e;
        }
    }
    __syncthreads();
    for (int idx = tid; idx < (K << Lh); idx += blockDim.x) {
        const int k = idx >> Lh, u = idx & ((1 << Lh) - 1);
        float s = 0.f;
        for (int b = 0; b < Lh; ++b)
            if ((u >> b) & 1) s += C[k][Ll + b];
        tabHi[k][u] = s;
    }
    for (int idx = tid; idx < (K << Ll); idx += blockDim.x) {
        const int k = idx >> Ll, u = idx & ((1 << Ll) - 1);
        float s = 0.f;
        for (int b = 0; b < Ll; ++b)
            if ((u >> b) & 1) s += C[k][b];
        tabLo[k][u] = s;
    }
    __syncthreads();
}

// PASS 0: minimum; PASS 1: collect x with E <= thr.  A CTA takes kBfHiPerRound hi
// values per round of set-up.
constexpr int kBfHiPerRound = 4;
template <int PASS>
__global__ void __launch_bounds__(kBfThreads) bf_dense_pass(const float *W, int N, int L, uint64_t xb, uint64_t xe,
                                                            float slack, BfWorkspace *ws, uint64_t *cand, int cap) {
    constexpr int K = kBfHiPerRound;
    __shared__ float tabHi[K][128], tabLo[K][128], C[K][kLoBits];
    __shared__ float base[K];
    __shared__ unsigned int blockMin;
    const int Lh = L / 2, Ll = L - Lh;
    const uint64_t hb = xb >> L, he = (xe - 1) >> L;
    float thr = 0.f;
    if (PASS == 1) thr = dec_float(ws->minEnc) + slack;
    const uint32_t mask = (1u << Ll) - 1u;
    for (uint64_t hi0 = hb + (uint64_t)blockIdx.x * K; hi0 <= he; hi0 += (uint64_t)gridDim.x * K) {
        bf_block_setup_k<K>(W, N, L, hi0, he, base, tabHi, tabLo, C, Lh, Ll);
        if (PASS == 0 && threadIdx.x == 0) blockMin = 0xffffffffu;
        __syncthreads();
        float lmin = __int_as_float(0x7f800000);
        for (int k = 0; k < K && hi0 + k <= he; ++k) {
            const float bk = base[k];
            const float *tH = tabHi[k], *tL = tabLo[k];
            const uint64_t x0 = (hi0 + k) << L;
            const uint32_t loB = (uint32_t)(xb > x0 ? xb - x0 : 0);
            const uint32_t loE = (uint32_t)min((uint64_t)1 << L, xe - x0);
            auto visit = [&](uint32_t lo, float e) {
                if (PASS == 0) {
                    lmin = fminf(lmin, e);
                } else if (e <= thr) {
                    int slot = atomicAdd(&ws->count, 1);
                    if (slot < cap) cand[slot] = x0 | lo;
                }
            };
            // four consecutive states per thread: one 16-byte load of the E_ll table and one
            // tabHi lookup for the four; a thread's tabLo entries stay the same across its
            // iterations (the stride 4 * blockDim.x is a multiple of 2^Ll), so they are
            // kept in registers.  Every energy is summed in the same order as one at a time.
            const uint32_t vb = (loB + 3u) & ~3u, ve = loE & ~3u;
            const uint32_t step4 = 4u * blockDim.x;
            if (vb < ve && (step4 & mask) == 0 && !(reinterpret_cast<uintptr_t>(ws->ell) & 15)) {
                for (uint32_t lo = loB + threadIdx.x; lo < vb; lo += blockDim.x)
                    visit(lo, (bk + ws->ell[lo]) + (tH[lo >> Ll] + tL[lo & mask]));
                for (uint32_t lo = ve + threadIdx.x; lo < loE; lo += blockDim.x)
                    visit(lo, (bk + ws->ell[lo]) + (tH[lo >> Ll] + tL[lo & mask]));
                const uint32_t first = vb + 4u * threadIdx.x;
                const float t0 = tL[first & mask], t1 = tL[(first + 1u) & mask];
                const float t2 = tL[(first + 2u) & mask], t3 = tL[(first + 3u) & mask];
                uint32_t lo = first;
                for (; lo + step4 < ve; lo += 2u * step4) {
                    const float4 l = *reinterpret_cast<const float4 *>(&ws->ell[lo]);
                    const float4 q = *reinterpret_cast<const float4 *>(&ws->ell[lo + step4]);
                    const float th = tH[lo >> Ll], tq = tH[(lo + step4) >> Ll];
                    visit(lo, (bk + l.x) + (th + t0));
                    visit(lo + 1u, (bk + l.y) + (th + t1));
                    visit(lo + 2u, (bk + l.z) + (th + t2));
                    visit(lo + 3u, (bk + l.w) + (th + t3));
                    visit(lo + step4, (bk + q.x) + (tq + t0));
                    visit(lo + step4 + 1u, (bk + q.y) + (tq + t1));
                    visit(lo + step4 + 2u, (bk + q.z) + (tq + t2));
                    visit(lo + step4 + 3u, (bk + q.w) + (tq + t3));
                }
                for (; lo < ve; lo += step4) {
                    const float4 l = *reinterpret_cast<const float4 *>(&ws->ell[lo]);
                    const float th = tH[lo >> Ll];  // the four share lo >> Ll (2^Ll is a multiple of 4)
                    visit(lo, (bk + l.x) + (th + t0));
                    visit(lo + 1u, (bk + l.y) + (th + t1));
                    visit(lo + 2u, (bk + l.z) + (th + t2));
                    visit(lo + 3u, (bk + l.w) + (th + t3));
                }
            } else {
                for (uint32_t lo = loB + threadIdx.x; lo < loE; lo += blockDim.x)
                    visit(lo, (bk + ws->ell[lo]) + (tH[lo >> Ll] + tL[lo & mask]));
            }
        }
        if (PASS == 0) {
            for (int o = 16; o > 0; o >>= 1) lmin = fminf(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
            if ((threadIdx.x & 31) == 0) atomicMin(&blockMin, enc_float(lmin));
            __syncthreads();
            if (threadIdx.x == 0) atomicMin(&ws->minEnc, blockMin);
        }
        __syncthreads();
    }
}

// The minimum over all x0 of each of the 32 x1 that share their bits from 5 on
// (X5 = x1 >> 5), warp-wide; lane t returns that of x1 = 32 X5 + t.  Lane j holds
// D[j] (and j + 32), every lane b1.x1; a Gray walk over the low five bits changes
// them by one FP64 row per x1.  The negative D, rounded to fp32, are summed by a
// fixed tree.
__device__ __forceinline__ float bip_min32(const float *b0, const float *b1, const float *W, int N0, int N1,
                                           uint64_t X5) {
    const int lane = threadIdx.x & 31;
    const bool in0 = lane < N0, in1 = lane + 32 < N0;
    double d0 = in0 ? (double)b0[lane] : 0., d1 = in1 ? (double)b0[lane + 32] : 0., s = 0.;
    // x1 bit c <-> variable N1-1-c; the rows of the low bits stay in registers (zero beyond N1)
    float w0[5], w1[5], wb[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        const float *w = W + (size_t)max(N1 - 1 - c, 0) * N0;
        w0[c] = in0 && c < N1 ? w[lane] : 0.f;
        w1[c] = in1 && c < N1 ? w[lane + 32] : 0.f;
        wb[c] = c < N1 ? b1[N1 - 1 - c] : 0.f;
    }
    for (int c = 5; c < N1; ++c)
        if ((X5 >> (c - 5)) & 1ull) {
            const float *w = W + (size_t)(N1 - 1 - c) * N0;
            if (in0) d0 += (double)w[lane];
            if (N0 > 32 && in1) d1 += (double)w[lane + 32];
            s += (double)b1[N1 - 1 - c];
        }
    float res = __int_as_float(0x7f800000);
#pragma unroll
    for (int k = 0; k < 32; ++k) {
        const int g = k ^ (k >> 1);
        if (k) {
            const int c = (k & 1) ? 0 : (k & 2) ? 1 : (k & 4) ? 2 : (k & 8) ? 3 : 4;
            const float sign = (g >> c) & 1 ? 1.f : -1.f;
            d0 += (double)(sign * w0[c]);
            if (N0 > 32) d1 += (double)(sign * w1[c]);
            s += (double)(sign * wb[c]);
        }
        float e = fminf((float)d0, 0.f);
        if (N0 > 32) e = __fadd_rn(e, fminf((float)d1, 0.f));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) e = __fadd_rn(e, __shfl_xor_sync(0xffffffffu, e, o));
        if (lane == g) res = __fadd_rn((float)s, e);
    }
    return res;
}

// the least of them over [x1b, x1e)
__global__ void __launch_bounds__(kBfThreads) bf_bip_min(const float *b0, const float *b1, const float *W, int N0,
                                                         int N1, uint64_t x1b, uint64_t x1e, BfWorkspace *ws) {
    const int lane = threadIdx.x & 31;
    float best = __int_as_float(0x7f800000);
    for (uint64_t X = (x1b >> 5) + (uint64_t)blockIdx.x * (kBfThreads / 32) + (threadIdx.x >> 5); X <= (x1e - 1) >> 5;
         X += (uint64_t)gridDim.x * (kBfThreads / 32)) {
        const float e = bip_min32(b0, b1, W, N0, N1, X);
        const uint64_t x1 = (X << 5) + lane;
        if (x1 >= x1b && x1 < x1e) best = fminf(best, e);
    }
    for (int o = 16; o > 0; o >>= 1) best = fminf(best, __shfl_xor_sync(0xffffffffu, best, o));
    if (lane == 0) atomicMin(&ws->minEnc, enc_float(best));
}

struct BipShared {
    float tab[9][128];
    float D[64];
    float base;
    unsigned int blockMin;
    unsigned int reach[kBfThreads / 32];
};

// one x1: x0 in [x0b, x0e) through 7-bit-group tables (all threads of the CTA).
// COLLECT false: their minimum into ws->minEnc; true: those with E <= thr
template <bool COLLECT>
__device__ __forceinline__ void bip_x1_states(BipShared &S, const float *b0, const float *b1, const float *W, int N0,
                                              int N1, uint64_t x0b, uint64_t x0e, uint64_t x1, float thr,
                                              BfWorkspace *ws, uint64_t *cand, int cap) {
    const int nG = (N0 + 6) / 7;
    int tid = threadIdx.x;
    // x0 bit c <-> variable N0-1-c ; x1 bit c <-> variable N1-1-c
    if (tid < N0) {
        int j = N0 - 1 - tid;  // D indexed by x0 bit position
        double s = (double)b0[j];
        for (int c = 0; c < N1; ++c)
            if ((x1 >> c) & 1ull) s += (double)W[(size_t)(N1 - 1 - c) * N0 + j];
        S.D[tid] = (float)s;
    }
    if (tid == 64) {
        double s = 0.;
        for (int c = 0; c < N1; ++c)
            if ((x1 >> c) & 1ull) s += (double)b1[N1 - 1 - c];
        S.base = (float)s;
    }
    if (!COLLECT && tid == 0) S.blockMin = 0xffffffffu;
    __syncthreads();
    for (int t = tid; t < nG * 128; t += blockDim.x) {
        int g = t >> 7, v = t & 127;
        float s = 0.f;
        for (int k = 0; k < 7; ++k) {
            int bit = g * 7 + k;
            if (bit < N0 && ((v >> k) & 1)) s += S.D[bit];
        }
        S.tab[g][v] = s;
    }
    __syncthreads();
    const float base = S.base;
    float lmin = __int_as_float(0x7f800000);
    auto visit = [&](uint64_t x0, float e) {
        if (!COLLECT) {
            lmin = fminf(lmin, e);
        } else if (e <= thr) {
            int slot = atomicAdd(&ws->count, 1);
            if (slot < cap) {
                cand[2 * slot] = x0;
                cand[2 * slot + 1] = x1;
            }
        }
    };
    auto energy = [&](uint64_t x0) {
        float e = base;
        for (int g = 0; g < nG; ++g) e += S.tab[g][(x0 >> (7 * g)) & 127];
        return e;
    };
    // four consecutive x0 per thread: their first-group entries stay the same across
    // the thread's iterations (the stride 4 * blockDim.x is a multiple of 128), so
    // they are kept in registers, and the four share every higher group's lookup.
    // Each energy adds its groups in the same order as one at a time.
    const uint64_t vb = (x0b + 3) & ~3ull, ve = x0e & ~3ull;
    const uint32_t step4 = 4u * blockDim.x;
    if (nG >= 2 && vb < ve && (step4 & 127u) == 0) {
        for (uint64_t x0 = x0b + tid; x0 < vb && x0 < x0e; x0 += blockDim.x) visit(x0, energy(x0));
        for (uint64_t x0 = ve + tid; x0 < x0e; x0 += blockDim.x) visit(x0, energy(x0));
        const uint64_t first = vb + 4u * tid;
        const float t0 = base + S.tab[0][first & 127], t1 = base + S.tab[0][(first + 1) & 127];
        const float t2 = base + S.tab[0][(first + 2) & 127], t3 = base + S.tab[0][(first + 3) & 127];
        for (uint64_t x0 = first; x0 < ve; x0 += step4) {
            float e0 = t0, e1 = t1, e2 = t2, e3 = t3;
            for (int g = 1; g < nG; ++g) {
                const float tg = S.tab[g][(x0 >> (7 * g)) & 127];  // the same for x0 .. x0 + 3
                e0 += tg;
                e1 += tg;
                e2 += tg;
                e3 += tg;
            }
            visit(x0, e0);
            visit(x0 + 1, e1);
            visit(x0 + 2, e2);
            visit(x0 + 3, e3);
        }
    } else {
        for (uint64_t x0 = x0b + tid; x0 < x0e; x0 += blockDim.x) visit(x0, energy(x0));
    }
    if (!COLLECT) {
        for (int o = 16; o > 0; o >>= 1) lmin = fminf(lmin, __shfl_xor_sync(0xffffffffu, lmin, o));
        if ((tid & 31) == 0) atomicMin(&S.blockMin, enc_float(lmin));
        __syncthreads();
        if (tid == 0) atomicMin(&ws->minEnc, S.blockMin);
    }
    __syncthreads();
}

// every x1 in [x1b, x1e), one per CTA: PASS 0 minimum, PASS 1 collection
template <int PASS>
__global__ void __launch_bounds__(kBfThreads) bf_bip_pass(const float *b0, const float *b1, const float *W, int N0,
                                                          int N1, uint64_t x0b, uint64_t x0e, uint64_t x1b,
                                                          uint64_t x1e, float slack, BfWorkspace *ws,
                                                          uint64_t *cand, int cap) {
    __shared__ BipShared S;
    const float thr = PASS == 1 ? dec_float(ws->minEnc) + slack : 0.f;
    for (uint64_t x1 = x1b + blockIdx.x; x1 < x1e; x1 += gridDim.x)
        bip_x1_states<PASS == 1>(S, b0, b1, W, N0, N1, x0b, x0e, x1, thr, ws, cand, cap);
}

// collection over all x0, after bf_bip_min: the first nWarps warps of a CTA take a unit
// each, a block of 32 x1 or one of its 2^partBits parts, and the CTA searches those of the
// units' x1 whose minimum over all x0 is within reach, thr and the slack once more (the
// minimum and a state's energy are rounded differently).  All may be within reach
// (nonnegative W without biases), so few blocks are spread over the SMs: N0 = 17, N1 = 14
// of that kind took 15.3 ms a search with eight blocks a CTA, 10.8 with about two units per
// SM, 10.4 state by state in both passes.  Parts repeat the block's minima, so they are
// for launches of fewer blocks than that (N0 of 25 and more, few x1).  A search of N0 = N1
// = 15 with one minimum: 111 us (1100 us state by state).
__global__ void __launch_bounds__(kBfThreads) bf_bip_collect(const float *b0, const float *b1, const float *W, int N0,
                                                             int N1, uint64_t x1b, uint64_t x1e, int nWarps,
                                                             int partBits, float slack, BfWorkspace *ws, uint64_t *cand,
                                                             int cap) {
    __shared__ BipShared S;
    constexpr int kWarps = kBfThreads / 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float thr = dec_float(ws->minEnc) + slack;
    const uint64_t Xb = x1b >> 5, units = (((x1e - 1) >> 5) - Xb + 1) << partBits;
    for (uint64_t U0 = (uint64_t)blockIdx.x * nWarps; U0 < units; U0 += (uint64_t)gridDim.x * nWarps) {
        if (warp < nWarps) {
            const uint64_t U = U0 + warp, X = Xb + (U >> partBits), x1 = (X << 5) + lane;
            float e = __int_as_float(0x7f800000);
            if (U < units) e = bip_min32(b0, b1, W, N0, N1, X);  // (every lane: the minima are warp-wide)
            const bool mine = lane >> (5 - partBits) == (int)(U & ((1u << partBits) - 1u));
            const unsigned reach =
                __ballot_sync(0xffffffffu, mine && U < units && x1 >= x1b && x1 < x1e && e <= thr + slack);
            if (lane == 0) S.reach[warp] = reach;
        }
        __syncthreads();
        unsigned todo[kWarps];
#pragma unroll
        for (int w = 0; w < kWarps; ++w) todo[w] = w < nWarps ? S.reach[w] : 0u;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < kWarps; ++w)
            for (unsigned t = todo[w]; t; t &= t - 1u)
                bip_x1_states<true>(S, b0, b1, W, N0, N1, 0, 1ull << N0,
                                    ((Xb + ((U0 + w) >> partBits)) << 5) + (__ffs(t) - 1), thr, ws, cand, cap);
    }
}

// FP64 energies of packed dense states, one warp per state (W float, or double
// for the double-precision searchers)
template <class T>
__global__ void bf_dense_refine(const T *W, int N, const uint64_t *xs, int n, double *E) {
    int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    uint64_t x = xs[w];
    double s = 0.;
    for (int i = lane; i < N; i += 32) {
        if (!((x >> (N - 1 - i)) & 1ull)) continue;
        for (int j = 0; j < N; ++j)
            if ((x >> (N - 1 - j)) & 1ull) s += (double)W[(size_t)i * N + j];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) E[w] = s;
}

template <class T>
__global__ void bf_bip_refine(const T *b0, const T *b1, const T *W, int N0, int N1, const uint64_t *pairs, int n,
                              double *E) {
    int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    uint64_t x0 = pairs[2 * w], x1 = pairs[2 * w + 1];
    double s = 0.;
    for (int j = lane; j < N0; j += 32)
        if ((x0 >> (N0 - 1 - j)) & 1ull) s += (double)b0[j];
    for (int i = lane; i < N1; i += 32) {
        if (!((x1 >> (N1 - 1 - i)) & 1ull)) continue;
        s += (double)b1[i];
        for (int j = 0; j < N0; ++j)
            if ((x0 >> (N0 - 1 - j)) & 1ull) s += (double)W[(size_t)i * N0 + j];
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) E[w] = s;
}

static int bf_grid(uint64_t units, int perSm) {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    uint64_t g = (uint64_t)sms * perSm;
    return (int)(units < g ? units : g);
}

}  // namespace sq103

using namespace sq103;

extern "C" {

SQ103_API size_t sq103_bf_workspace_bytes(int N) {
    (void)N;
    return sizeof(BfWorkspace);
}

SQ103_API int sq103_dense_bf_range(const float *W, int N, uint64_t xBegin, uint64_t xEnd, float slack, void *ws,
                                   uint64_t *cand, int cap, int *count, float *Emin32, void *stream) {
    if (N <= 0 || N > 63 || xEnd <= xBegin || xEnd > (1ull << N)) return kErrBadShape;
    cudaStream_t s = (cudaStream_t)stream;
    BfWorkspace *w = (BfWorkspace *)ws;
    int L = N < kLoBits ? N : kLoBits;
    bf_init_ws<<<(kBfGroups + 255) / 256, 256, 0, s>>>(w);
    bf_lo_table<<<((1 << L) + 127) / 128, 128, 0, s>>>(W, N, L, w);
    // [xBegin, x1) and [x2, xEnd) around the whole runs [x1, x2)
    uint64_t x1 = xEnd, x2 = xEnd;
    if (N >= kRunShift) {
        const uint64_t rb = (xBegin + (1ull << kRunShift) - 1) >> kRunShift, re = xEnd >> kRunShift;
        if (rb < re) {
            x1 = rb << kRunShift;
            x2 = re << kRunShift;
        }
    }
    const size_t runSmem = sizeof(RunShared) + sizeof(float) * N * N;
    const uint64_t runs = (x2 - x1) >> kRunShift;
    int groupShift = 0;
    while ((runs >> groupShift) > (uint64_t)kBfGroups - 1) ++groupShift;
    // few runs are split over hi, down to four values an item, to fill the GPU
    int subBits = 0;
    while (subBits < 4 && (runs << subBits) < (uint64_t)bf_grid(~0ull, 2)) ++subBits;
    if (runs > 0) {
        static SmemLimitOnce limit;
        const cudaError_t e = limit((int)(sizeof(RunShared) + sizeof(float) * 63 * 63), bf_run_pass<0>, bf_run_pass<1>);
        if (e != cudaSuccess) return (int)e;
    }
    for (int pass = 0; pass < 2; ++pass) {
        for (int side = 0; side < 2; ++side) {
            const uint64_t b = side ? x2 : xBegin, e = side ? xEnd : x1;
            if (b >= e) continue;
            const uint64_t nHi = ((e - 1) >> L) - (b >> L) + 1;
            const int grid = bf_grid((nHi + kBfHiPerRound - 1) / kBfHiPerRound, 8);
            if (pass == 0)
                bf_dense_pass<0><<<grid, kBfThreads, 0, s>>>(W, N, L, b, e, slack, w, cand, cap);
            else
                bf_dense_pass<1><<<grid, kBfThreads, 0, s>>>(W, N, L, b, e, slack, w, cand, cap);
        }
        if (runs == 0) continue;
        const uint64_t rb = x1 >> kRunShift, re = x2 >> kRunShift;
        if (pass == 0)
            bf_run_pass<0><<<bf_grid(runs << subBits, 2), kBfThreads, runSmem, s>>>(W, N, rb, re, groupShift, subBits,
                                                                                   slack, w, cand, cap);
        else
            bf_run_pass<1><<<bf_grid(runs << 3, 2), kBfThreads, runSmem, s>>>(W, N, rb, re, groupShift, 3, slack, w,
                                                                             cand, cap);
    }
    unsigned int enc = 0;
    cudaMemcpyAsync(count, &w->count, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&enc, &w->minEnc, sizeof(unsigned int), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return (int)e;
    unsigned int u = (enc & 0x80000000u) ? (enc & 0x7fffffffu) : ~enc;
    memcpy(Emin32, &u, sizeof(float));
    return (int)cudaGetLastError();
}

SQ103_API int sq103_dense_bf_refine(const float *W, int N, const uint64_t *x, int n, double *E, void *stream) {
    if (n <= 0) return 0;
    bf_dense_refine<float><<<(n * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(W, N, x, n, E);
    return (int)cudaGetLastError();
}

SQ103_API int sq103_dense_bf_refine64(const double *W, int N, const uint64_t *x, int n, double *E, void *stream) {
    if (n <= 0) return 0;
    bf_dense_refine<double><<<(n * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(W, N, x, n, E);
    return (int)cudaGetLastError();
}

SQ103_API int sq103_bipartite_bf_range(const float *b0, const float *b1, const float *W, int N0, int N1,
                                       uint64_t x0b, uint64_t x0e, uint64_t x1b, uint64_t x1e, float slack,
                                       void *ws, uint64_t *cand, int cap, int *count, float *Emin32,
                                       void *stream) {
    if (N0 <= 0 || N1 <= 0 || N0 > 63 || N1 > 63 || x0e <= x0b || x1e <= x1b) return kErrBadShape;
    cudaStream_t s = (cudaStream_t)stream;
    BfWorkspace *w = (BfWorkspace *)ws;
    bf_init_ws<<<(kBfGroups + 255) / 256, 256, 0, s>>>(w);
    // over all x0, the minimum per x1 pays from 2^13 values of x1 or 2^25 states on; below,
    // its Gray walks take longer than the states (N0 = N1 = 12: 166 us a search so,
    // 160 us state by state; 13: 164 and 215; N0 = 7, N1 = 15: 160 and 373)
    if (x0b == 0 && x0e == 1ull << N0 && (x1e - x1b >= 1ull << 13 || N0 >= 25 || (x1e - x1b) << N0 >= 1ull << 25)) {
        const int grid = bf_grid((((x1e - 1) >> 5) - (x1b >> 5) + kBfThreads / 32) / (kBfThreads / 32), 8);
        bf_bip_min<<<grid, kBfThreads, 0, s>>>(b0, b1, W, N0, N1, x1b, x1e, w);
        const uint64_t blocks = ((x1e - 1) >> 5) - (x1b >> 5) + 1, full = (uint64_t)bf_grid(~0ull, 2);
        const int nWarps = (int)std::max<uint64_t>(1, std::min<uint64_t>(kBfThreads / 32, blocks / full));
        int partBits = 0;
        while (partBits < 5 && blocks << (partBits + 1) <= full) ++partBits;
        bf_bip_collect<<<bf_grid(((blocks << partBits) + nWarps - 1) / nWarps, 8), kBfThreads, 0, s>>>(
            b0, b1, W, N0, N1, x1b, x1e, nWarps, partBits, slack, w, cand, cap);
    } else {
        const int grid = bf_grid(x1e - x1b, 8);
        bf_bip_pass<0><<<grid, kBfThreads, 0, s>>>(b0, b1, W, N0, N1, x0b, x0e, x1b, x1e, slack, w, cand, cap);
        bf_bip_pass<1><<<grid, kBfThreads, 0, s>>>(b0, b1, W, N0, N1, x0b, x0e, x1b, x1e, slack, w, cand, cap);
    }
    unsigned int enc = 0;
    cudaMemcpyAsync(count, &w->count, sizeof(int), cudaMemcpyDeviceToHost, s);
    cudaMemcpyAsync(&enc, &w->minEnc, sizeof(unsigned int), cudaMemcpyDeviceToHost, s);
    cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return (int)e;
    unsigned int u = (enc & 0x80000000u) ? (enc & 0x7fffffffu) : ~enc;
    memcpy(Emin32, &u, sizeof(float));
    return (int)cudaGetLastError();
}

SQ103_API int sq103_bipartite_bf_refine(const float *b0, const float *b1, const float *W, int N0, int N1,
                                        const uint64_t *pairs, int n, double *E, void *stream) {
    if (n <= 0) return 0;
    bf_bip_refine<float><<<(n * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(b0, b1, W, N0, N1, pairs, n, E);
    return (int)cudaGetLastError();
}

SQ103_API int sq103_bipartite_bf_refine64(const double *b0, const double *b1, const double *W, int N0, int N1,
                                          const uint64_t *pairs, int n, double *E, void *stream) {
    if (n <= 0) return 0;
    bf_bip_refine<double><<<(n * 32 + 255) / 256, 256, 0, (cudaStream_t)stream>>>(b0, b1, W, N0, N1, pairs, n, E);
    return (int)cudaGetLastError();
}

}  // extern "C"
