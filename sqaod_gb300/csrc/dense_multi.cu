// dense_multi.cu -- one CTA per trotter: the dense coloring / SA sweep of one
// large instance across the whole GPU (cooperative launch, all CTAs resident).
//
// It runs the same trials in the same colour order as the one-CTA-per-instance
// kernel in dense.cu, updates the fields in the same order with the same
// rounding, and takes the same (exact) decisions, so both give bit-identical
// spins and fields.
//
// Per CTA (trotter y), 256 threads (224 where four CTAs share an SM):
//   warp 0  decider: the trotter's trials in batches of 32 iterations, lane i =
//           iteration g0 + i.  A lane holds z = rate dE - L, L = -ln u (the trial
//           accepts when z < 0) and a bound on its fp32 error.  A batch is decided
//           in rounds: the lowest accepting lane is final (all undecided lanes
//           below it reject), and a lane above it adds its product with
//           d J[x_f][x_i] to z and changes signs when it shares the flipped site.
//           A batch takes (accepted flips + 1) rounds instead of 32 sequential
//           trials.  The batch's fields start from the resident row F[y][:],
//           which the updaters keep one batch behind, plus the previous
//           batch's flips d_f * J[x_f][x_i].
//           Decisions are published as one 64-bit word per batch (accept
//           bits, decided count, batch tag) with a single relaxed store after
//           every accepting round and at the end of the batch: a reader that
//           sees the tag of the batch it wants sees consistent bits, so no
//           fence is needed.
//   warp 1  helper: polls the two neighbours' accept words (both neighbours,
//           two words ahead, in one round trip) and copies them into shared
//           memory.
//   warps 2-3 prefetchers, alternate batches: this trotter's own trials (PreTrial),
//           the in-batch gathers J[x_j][x_i] (j < i) for the lanes j predicted to
//           accept, the neighbours' sites of the same iterations (a ring of
//           sites and one hashed-site bitmap per batch), and per lane the
//           neighbour iterations of this and the two previous batches that hit its
//           site, into a ring of kPre batch buffers with a ready tag each.
//   warps 4-6 (4-5) updaters: F[y][:] += d * J[x][:] for the flips of the previous
//           batch, in trial order, while the decider works on the next one.
//   last warp exact decisions: a trial whose fp32 outcome the rounding of the
//           resident field could change is decided in FP64 from its exact field
//           (sq_common.cuh); the warp sleeps on a named barrier between requests
//           and answers through a shared word the decider waits on (bounded).
// What bounds it: the decider's chain, about 2500 cycles a batch without flips and
// 1000 per flip at N = 4096, m = 256 (two CTAs per SM), at some ten cycles an
// instruction; DRAM is idle and issue slots are three quarters free.
// Colour order: trial (y, k) must see neighbour n after every neighbour trial
// that precedes it (iteration < k, or = k when n's colour phase comes first:
// even trotters, then trotter m-1 if m is odd, then odd trotters).  The
// decider applies neighbour flips to a ghost bit row of n only up to the
// first trial of its current batch; each lane's bit is corrected for the
// neighbour trials between that point and the lane's own limit, which the
// prefetched lists show to be none for almost every lane.  A lane waits only when such
// a neighbour trial is not yet published.  Every wait is bounded (global
// timer) and ends the kernel with a timeout status instead of hanging; before
// waiting a CTA publishes the trials it has decided, so waits always point to
// strictly earlier trials and cannot form a cycle.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

// the exact warp's helpers inlined: measured 1.8 % faster at N=4096 m=256
#define SQ103_EXACT_ATTR __forceinline__
// the prefetchers' three to seven generators two rounds at a time: N = 1000, m = 250
// 5.75 -> 5.56 ms, 128 uneven instances 27.1 -> 26.2 ms (instruction fetch)
#define SQ103_PHILOX_UNROLL 2
#include "mc_trial.h"
#include "sq_common.cuh"
#include "sq_kernels.h"

namespace sq103 {

constexpr int kPf = 2;                            // prefetcher warps (2 .. 1 + kPf)
constexpr int kUpdWarp0 = 2 + kPf;                // first updater warp
// threads of a CTA: three updater warps at two CTAs per SM, two at four (the registers
// of the third go to the others: N = 2000, m = 500 6.6 -> 6.3 ms; at two per SM the
// third is worth it, N = 4096, m = 256 20.3 -> 19.5 ms)
__host__ __device__ constexpr int mc_threads(int perSm) { return perSm > 2 ? 224 : 256; }
constexpr int kBarExReq = 3;                      // wakes the exact warp (decider + exact warp, 64 threads)
constexpr int kRing = 256;      // neighbour sites kept per neighbour (power of two)
constexpr int kLogWords = 32;   // neighbour accept words kept per neighbour (power of two)
constexpr int kBmBits = 2048;   // bits of a batch's neighbour-site bitmap (hashed sites, power of two)
constexpr int kBmWords = kBmBits / 32;
constexpr int kBmSlots = kRing / 32;  // bitmaps kept per neighbour (one per ring batch)
constexpr int kPre = 4;         // prefetched batches (power of two)
constexpr int kJgStride = 32 * 33;
constexpr int kCand = 2;        // neighbour iterations per lane and batch found by the prefetchers
constexpr int kPredRows = 8;    // predicted accepting lanes whose gathers are kept in registers
constexpr float kFieldDrift = 1.f;  // assumed field change between prefetch and decision
constexpr unsigned long long kWaitLimitNs = 4000000000ull;
constexpr unsigned long long kShortWaitNs = 1000000ull;  // task flag kFlagShortWaits (tests)
// the prefetchers run ahead and mostly wait: they poll gently, which leaves the
// SM's shared load/store path to the decider
constexpr int kPrefetchSleepNs = 32;
constexpr unsigned FULL = 0xffffffffu;
constexpr int kSmallN = 1024;  // rows up to this many spins take the kSmall instance (measured: 1024 faster, 2048 slower)

__device__ __forceinline__ unsigned long long ld_relaxed_u64(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed_u64(unsigned long long *p, unsigned long long v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
// bar.sync and bar.arrive count whole warps: a warp whose lanes reach one apart would
// count more than once and let the other side run early, so the lanes meet first
__device__ __forceinline__ void bar_sync(int id, int n) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int n) {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
__device__ __forceinline__ unsigned smem_addr(const volatile void *p) {
    return (unsigned)__cvta_generic_to_shared((const void *)p);
}
__device__ __forceinline__ int ld_acquire_cta(const volatile int *p) {
    int v;
    asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long ld_acquire_cta64(const volatile unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.acquire.cta.shared.b64 %0, [%1];" : "=l"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta(volatile int *p, int v) {
    asm volatile("st.release.cta.shared.b32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_cta64(volatile unsigned long long *p, unsigned long long v) {
    asm volatile("st.release.cta.shared.b64 [%0], %1;" ::"r"(smem_addr(p)), "l"(v) : "memory");
}

// accept word of batch b: bits 0-31 accept bits, 32-37 decided count, 38-63 b + 1
__device__ __forceinline__ unsigned long long log_word(int b, int cnt, unsigned bits) {
    return ((unsigned long long)(b + 1) << 38) | ((unsigned long long)cnt << 32) | bits;
}

__host__ __device__ __forceinline__ int colour_phase(int y, int m) {
    if ((m & 1) && y == m - 1) return 1;
    return (y & 1) ? 2 : 0;
}

// A prefetched trial (lane i of a batch): its site, h at the site, L = -ln u, and
// the constants of its step: dE's factors of h + 2F and of the spin sum times the
// rate, and the part of the decision's tolerance that does not depend on the
// field; its neighbour candidates, one byte each (two per neighbour, the latest
// first: 32 p + 32 - j for iteration j of the window of batch p).
struct __align__(16) PreTrial {
    int x;
    float h, L, cz;
    float cb, tolC, u;
    uint32_t cand;
};
constexpr uint32_t kNoCand = 127, kManyCand = 0;
constexpr uint32_t kNoCands = 0x7f7f7f7fu;
// bytes of the field row, the h row and the in-batch gathers, up to a 16-byte boundary
__host__ __device__ __forceinline__ constexpr size_t pre_offset(int N) {
    return ((size_t)N * 8 + (size_t)kPre * kJgStride * 4 + 15) & ~(size_t)15;
}

struct McShared {
    volatile unsigned long long logAvail;  // neighbour accept bits known below (lo: neighbour 0, hi: 1) (helper)
    volatile int applied[2];               // neighbour iterations applied to the ghost rows (decider)
    volatile int readyTag[kPre];           // p + 1 once buffer p % kPre holds batch p (prefetchers)
    volatile int ringTag[kPre];            // p + 1 once the neighbours' sites of batch p are in the ring (prefetchers)
    volatile int decDone;                  // batches [0, decDone) no longer read from the buffers (decider)
    volatile int done;
    int nflip;
    // exact decisions (rare): the decider posts a trial, the exact warp answers
    int exX, exBits;       // the trial's site; its FP64 outcomes for qL + qR = -2, 0, +2 (bits 0-2)
    volatile int exDone;   // number of the latest answer (exact warp; the decider counts its requests)
    float exQ, exU;
    int exIter;
};

// every lane loads the flag with acquire semantics (one broadcast access); the
// value of lane 0 keeps control flow uniform
__device__ __forceinline__ int uniform_acquire(const volatile int *p) { return __shfl_sync(FULL, ld_acquire_cta(p), 0); }
__device__ __forceinline__ unsigned long long uniform_acquire64(const volatile unsigned long long *p) {
    return __shfl_sync(FULL, ld_acquire_cta64(p), 0);
}
__device__ __forceinline__ int avail_of(unsigned long long v, int n) { return (int)(n ? v >> 32 : v & 0xffffffffu); }

// bounded wait on a warp-uniform condition; false on timeout
template <int SLEEP_NS = 32, class F>
__device__ __forceinline__ bool wait_until(unsigned long long limitNs, F &&ready) {
    unsigned long long t0 = 0;
    while (!ready()) {
        if (t0 == 0) t0 = global_ns();
        if (global_ns() - t0 > limitNs) return false;
        __nanosleep(SLEEP_NS);
    }
    return true;
}

// Warp-wide.  The spin bit of a neighbour at the lane's site x after its
// iteration Ji, from `bit` (its value after every published iteration below
// j0) and the iterations j in [j0, Ji] that hit x: published ones (j < avail)
// flip it when accepted; need returns the latest unpublished one (-1: none).
// The batch bitmaps flag the lanes whose hashed site an iteration of that
// batch hit; one ballot per flagged lane over the batch's sites finds them.
// j0 and pLast (the batch of the latest Ji) are warp-uniform; only `active`
// lanes take part.
__device__ __forceinline__ void window_bits(int x, int Ji, int j0, int pLast, int avail, bool active,
                                            const uint32_t *bmn, const int *rg, const uint32_t *nl, int Itot,
                                            int &bit, int &need) {
    const int lane = threadIdx.x & 31;
    const int hb = x & (kBmBits - 1);
    need = -1;
    for (int p = j0 >> 5; p <= pLast; ++p) {
        const int jlo = max(j0, 32 * p);
        const bool hit = active && Ji >= jlo && ((bmn[(p & (kBmSlots - 1)) * kBmWords + (hb >> 5)] >> (hb & 31)) & 1u);
        unsigned hits = __ballot_sync(FULL, hit);
        if (!hits) continue;
        const int jl = 32 * p + lane;
        const int sj = jl < Itot ? rg[jl & (kRing - 1)] : -1;
        const uint32_t accw = nl[p & (kLogWords - 1)];  // accept bits, valid below avail
        while (hits) {
            const int i = __ffs(hits) - 1;
            hits &= hits - 1u;
            const int xi = __shfl_sync(FULL, x, i), Jii = __shfl_sync(FULL, Ji, i);
            const unsigned mt = __ballot_sync(FULL, sj == xi && jl >= jlo && jl <= Jii);
            if (lane == i) {
                for (unsigned r = mt; r; r &= r - 1u) {
                    const int j = 32 * p + __ffs(r) - 1;
                    if (j < avail)
                        bit ^= (accw >> (j & 31)) & 1u;
                    else
                        need = j;
                }
            }
        }
    }
}

// Up to kMaxPack independent instances in one cooperative launch (small ones of few
// trotters fill it only in numbers: 64 of m = 8 take 512 CTAs): CTAs
// [base[i], base[i+1]) are the trotters of task t[i], whose accept words live in
// outLog[i] (nWords[i] per trotter).  Instances do not interact (the prologue's
// grid sync is the only common step), so each runs exactly as alone.
constexpr int kMaxPack = 64;  // 12 KB of launch parameters, indexed in place
struct McPack {
    sq103_dense_task t[kMaxPack];
    unsigned long long *outLog[kMaxPack];
    int nWords[kMaxPack];
    int base[kMaxPack + 1];
    int n;
};

// kHooks: the acceptance trace and the test hooks of the task flags are compiled in
// (short waits, a trotter that withholds its accept words).  kSA: simulated
// annealing, without the neighbours' code.  Code that never runs is not free here:
// the warps' roles share the instruction caches, and SA at N = 1501, m = 63 took
// 3.24 ms for 64 steps with the neighbours' code compiled in, 3.12 without.
// kSmall: rows of at most kSmallN spins, where the neighbours' sites hit a lane's
// site often: each prefetcher finds a lane's neighbour candidates from a table
// of the positions at each site of batches p - 2 .. p (one per batch and
// neighbour, in shared memory, cleared after use), with the sites of p - 1 and
// p - 2 drawn again from the neighbours' Philox streams, instead of a ballot per
// hit over the hashed-site bitmaps of the other prefetcher's batches (which
// makes the prefetchers wait for each other).  Both give the same candidates.
// kPerSm: the CTAs per SM the registers are allotted for.  The trotters of a launch
// are all resident, so the limit on m is kPerSm * 152 (where shared memory allows
// as many: N <= 3100 for four).  Two leave 114 registers a thread and the fastest
// decider; four have 72 (up to 24 bytes spilled) and take the launches that exceed two.
// N = 2000, m = 500, 8 steps: 3.7 ms with four per SM; one CTA for the whole
// instance, which such sizes fell back to before, 1090 ms.
template <bool kHooks, bool kSmall, bool kSA, int kPerSm>
__global__ void __launch_bounds__(mc_threads(kPerSm), kPerSm) dense_sweep_multi(const __grid_constant__ McPack P) {
    constexpr int kMcThreads = mc_threads(kPerSm);
    constexpr int kExactWarp = kMcThreads / 32 - 1;  // the last warp: exact decisions
    constexpr int kMcUpdaters = kMcThreads - 32 * kUpdWarp0 - 32;
    constexpr int kBarCount = 32 + kMcUpdaters;      // decider + updaters (barriers 1, 2)
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ McShared S;
    __shared__ sq103_dense_task task;
    __shared__ unsigned long long *sLog;
    __shared__ int sWords, sBase;
    if (threadIdx.x == 0) {
        int lo = 0, hi = P.n - 1;  // the instance whose CTAs [base[i], base[i + 1]) hold this one
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if ((int)blockIdx.x >= P.base[mid])
                lo = mid;
            else
                hi = mid - 1;
        }
        task = P.t[lo];
        sLog = P.outLog[lo];
        sWords = P.nWords[lo];
        sBase = P.base[lo];
    }
    __syncthreads();
    const sq103_dense_task &T = task;
    unsigned long long *const outLog = sLog;
    const int nWords = sWords;
    const int y = (int)blockIdx.x - sBase, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int N = T.N, m = T.m;
    constexpr bool sa = kSA;
    const int nNbr = sa ? 0 : (m == 2 ? 1 : 2);
    const int nbr0 = (y + m - 1) % m, nbr1 = (y + 1) % m;
    const int myPh = colour_phase(y, m);
    const int before0 = colour_phase(nbr0, m) < myPh ? 1 : 0;
    const int before1 = colour_phase(nbr1, m) < myPh ? 1 : 0;
    const int Itot = T.nSteps * N;
    const int nBatches = (Itot + 31) / 32;
    const int nWG = (N + 31) / 32;
    const int ghostStride = (nWG + 1) & ~1;
    const uint32_t tag = sa ? kTagDenseSA : kTagDenseSweep;
    // test hooks (task flags): every wait gives up after 1 ms; trotter 0 never
    // publishes its accept words, so its neighbours' waits run out
    const unsigned long long waitNs = (kHooks && (T.flags & kFlagShortWaits)) ? kShortWaitNs : kWaitLimitNs;
    const bool publish = !(kHooks && (T.flags & kFlagWithholdTrotter0) && y == 0);

    float *Fs = reinterpret_cast<float *>(smem);                        // N
    float *hs = Fs + N;                                                 // N
    float *Jg = hs + N;                                                 // kPre x 32 x 33
    PreTrial *pre = reinterpret_cast<PreTrial *>(smem + pre_offset(N));  // kPre x 32
    uint2 *ghost = reinterpret_cast<uint2 *>(pre + kPre * 32);          // nWG: spin bits of both neighbours
    uint32_t *bm = reinterpret_cast<uint32_t *>(ghost + ghostStride);   // 2 x kBmSlots x kBmWords
    int *ring = reinterpret_cast<int *>(bm + 2 * kBmSlots * kBmWords);  // 2 x kRing
    uint32_t *nlog = reinterpret_cast<uint32_t *>(ring + 2 * kRing);    // 2 x kLogWords
    unsigned *prePred = reinterpret_cast<unsigned *>(nlog + 2 * kLogWords);  // kPre
    int2 *flips = reinterpret_cast<int2 *>(prePred + kPre);             // 32
    int8_t *qs = reinterpret_cast<int8_t *>(flips + 32);                // N
    // kSmall: two site tables of kSmallN words per prefetcher (positions of a batch by site, one per neighbour)
    uint32_t *siteTab = reinterpret_cast<uint32_t *>(qs + ((N + 15) & ~15));

    for (int i = tid; i < kPre * 32; i += kMcThreads) pre[i].x = 0;  // (read before the first batch is ready)
    if (kSmall)
        for (int i = tid; i < kPf * 2 * kSmallN; i += kMcThreads) siteTab[i] = 0u;
    for (int i = tid; i < N; i += kMcThreads) {
        Fs[i] = T.F[(size_t)y * N + i];
        hs[i] = T.h[i];
        qs[i] = T.q[(size_t)y * N + i];
    }
    // a word of a neighbour's spin bits per warp and turn (a thread per word, 32 byte loads
    // after one another, took most of a short launch: N = 128, m = 16, one step, 22.0 us a
    // call before, 19.9 with this)
    for (int n = 0; n < nNbr; ++n) {
        const int8_t *qn = T.q + (size_t)(n ? nbr1 : nbr0) * N;
#pragma unroll 4
        for (int w = warp; w < nWG; w += kMcThreads / 32) {
            const int i = w * 32 + lane;
            const uint32_t bits = __ballot_sync(FULL, i < N && qn[i] > 0);
            if (lane == 0) (n ? ghost[w].y : ghost[w].x) = bits;
        }
    }
    if (tid == 0) {
        S.logAvail = 0;
        S.applied[0] = S.applied[1] = 0;
        for (int i = 0; i < kPre; ++i) S.readyTag[i] = S.ringTag[i] = 0;
        S.decDone = 0;
        S.exDone = 0;
        S.done = 0;
        S.nflip = 0;
    }
    // the accept words carry their batch's tag; zero means "not published"
#pragma unroll 1
    for (int w = tid; w < nWords; w += kMcThreads) outLog[(size_t)y * nWords + w] = 0ull;
    // every CTA has cleared its accept words before any CTA publishes or polls one,
    // and read its neighbours' rows before any CTA can finish and write its own back
    cooperative_groups::this_grid().sync();

    if (warp == 0) {
        // ------------------------------------------------------------ decider
        const uint32_t wordsPerStep = (uint32_t)(((size_t)N * m + 31) / 32);
        const float *const J = T.J;
        const int ldJ = T.ldJ;
        const bool traced = kHooks && T.trace != nullptr;
        unsigned long long *const myLog = outLog + (size_t)y * nWords;
        unsigned long long accepted = 0;
        bool aborted = false;
        unsigned accBits = 0;  // the previous batch's flips (lanes), their sites x and changes d = -2 q
        float d = 0.f;
        int x = 0;                 // the lane's site
        int nd0 = -1, nd1 = -1;    // the unknown neighbour iterations at the lane's site

        int A0 = 0, A1 = 0;  // neighbour iterations applied to the ghost rows
        int exSeq = 0;       // exact-decision requests posted

        // Applies the published neighbour iterations below lim0 / lim1 (their sites
        // are in the ring) to the ghost rows; returns the helper's availability word.
        auto apply_nbr = [&](int lim0, int lim1) {
            const unsigned long long av = uniform_acquire64(&S.logAvail);
            lim0 = min(avail_of(av, 0), lim0);
            lim1 = nNbr > 1 ? min(avail_of(av, 1), lim1) : 0;
            if (lim0 <= A0 && lim1 <= A1) return av;
            // both neighbours a word at a time, their loads in flight together
            for (int w0 = A0 >> 5, w1 = A1 >> 5; w0 * 32 < lim0 || w1 * 32 < lim1; ++w0, ++w1) {
                const int j0 = w0 * 32 + lane, j1 = w1 * 32 + lane;
                const uint32_t a0 = nlog[w0 & (kLogWords - 1)], a1 = nlog[kLogWords + (w1 & (kLogWords - 1))];
                const int s0 = ring[j0 & (kRing - 1)], s1 = ring[kRing + (j1 & (kRing - 1))];
                if (j0 >= A0 && j0 < lim0 && ((a0 >> lane) & 1u)) atomicXor(&ghost[s0 >> 5].x, 1u << (s0 & 31));
                if (j1 >= A1 && j1 < lim1 && ((a1 >> lane) & 1u)) atomicXor(&ghost[s1 >> 5].y, 1u << (s1 & 31));
            }
            A0 = max(A0, lim0);
            A1 = max(A1, lim1);
            __syncwarp();
            if (lane == 0) {
                S.applied[0] = A0;
                S.applied[1] = A1;
            }
            return av;
        };

        // Neighbour spins at the lane's site x for batch b: the ghost rows (iterations
        // < A applied) corrected by the neighbour iterations in [A, Ji] at the site,
        // which the prefetchers listed (the latest kCand of the last three batches).
        // A neighbour more than two batches behind, or a longer list, takes the bitmap
        // scan of window_bits.  sum: the known spins' sum; nd0, nd1: the latest
        // unpublished such iteration of each neighbour (-1: its spin is known).
        auto nbr_spins = [&](int b, int g0, bool valid, uint32_t cand, unsigned long long av, int &sum) {
            const uint2 g = ghost[x >> 5];
            int b0 = (g.x >> (x & 31)) & 1, b1 = (g.y >> (x & 31)) & 1;
            nd0 = nd1 = -1;
            bool slow = A0 < 32 * (b - 2) || (nNbr > 1 && A1 < 32 * (b - 2));
            if (!valid) cand = kNoCands;
            // the candidates not yet applied: bytes up to 32 p + 32 - A (few lanes have one)
            const uint32_t m0 = min(g0 + 32 - A0, 96), m1 = min(g0 + 32 - A1, 96);
            if (__vcmpleu4(cand, m0 | m0 << 8 | m1 << 16 | m1 << 24)) {
#pragma unroll(kSmall ? 4 : 1)
                for (int c = 0; c < 4; ++c) {
                    const int n = c >> 1, v = (cand >> (8 * c)) & 0xff, j = g0 + 32 - v;
                    if (v == (int)kManyCand) {
                        slow = true;
                    } else if (v <= 96 && j >= (n ? A1 : A0)) {
                        int f = 0;
                        if (j < avail_of(av, n))
                            f = (nlog[n * kLogWords + ((j >> 5) & (kLogWords - 1))] >> (j & 31)) & 1u;
                        else if (n)
                            nd1 = max(nd1, j);
                        else
                            nd0 = max(nd0, j);
                        if (n)
                            b1 ^= f;
                        else
                            b0 ^= f;
                    }
                }
            }
            slow = slow && valid;
            if (__any_sync(FULL, slow)) {
#pragma unroll 1
                for (int n = 0; n < nNbr; ++n) {
                    int bit = ((n ? g.y : g.x) >> (x & 31)) & 1, need;
                    window_bits(x, g0 + lane - 1 + (n ? before1 : before0), n ? A1 : A0, b, avail_of(av, n), slow,
                                bm + n * kBmSlots * kBmWords, ring + n * kRing, nlog + n * kLogWords, Itot, bit, need);
                    if (slow) {
                        if (n) {
                            b1 = bit;
                            nd1 = need;
                        } else {
                            b0 = bit;
                            nd0 = need;
                        }
                    }
                }
            }
            if (nNbr == 1) {  // m = 2: the one neighbour on both sides
                b1 = b0;
                nd1 = nd0;
            }
            sum = (nd0 >= 0 ? 0 : 2 * b0 - 1) + (nd1 >= 0 ? 0 : 2 * b1 - 1);
        };

        for (int b = 0; b < nBatches; ++b) {
            const int g0 = b * 32;
            const int buf = b & (kPre - 1);
            const int nValid = min(32, Itot - g0);
            const bool valid = lane < nValid;

            // this batch's trials, once its buffer is ready, and the published neighbour
            // iterations before its first trial (their sites are in the ring once the buffer
            // is ready; while it is not, those of earlier batches are applied, since the
            // prefetchers may need their ring slots)
            // The loads of the trial's site, and the flips handed to the updaters, come before
            // the ghost rows' work, which hides their latency.
            // The fields start from the resident row, which the updaters keep one batch
            // behind, plus the previous batch's flips: a lone flip's coupling is fetched here
            // and added after the neighbour work, several are added below in trial order.
            const bool lone = accBits && !(accBits & (accBits - 1u));
            PreTrial tr;
            unsigned long long av = 0, t0 = 0;
            unsigned pred = 0;  // lanes whose row of in-batch gathers is in jg
            float qx = 0.f, Fv = 0.f, dLone = 0.f, gLone = 0.f;
            for (;;) {
                const int tag = ld_acquire_cta(&S.readyTag[buf]);
                tr = pre[buf * 32 + lane];  // (site 0 beyond the last trial)
                // every lane's own tag: lanes may run apart here (lane 0 has just published), and
                // a lane's trial is valid only if its own load followed the tag
                const bool ready = __all_sync(FULL, tag == b + 1);
                if (ready) {
                    pred = prePred[buf];
                    qx = (float)qs[tr.x];
                    if (lone) {
                        const int f = __ffs(accBits) - 1;
                        dLone = __shfl_sync(FULL, d, f);
                        gLone = __ldg(J + (size_t)__shfl_sync(FULL, x, f) * ldJ + tr.x);
                    }
                    if (b > 0) bar_sync(2, kBarCount);
                    Fv = Fs[tr.x];
                    if (b > 0) {
                        if ((accBits >> lane) & 1u)
                            flips[__popc(accBits & ((1u << lane) - 1u))] = make_int2(x, __float_as_int(d));
                        if (lane == 0) S.nflip = __popc(accBits);
                        __syncwarp();
                        __threadfence_block();
                        bar_arrive(1, kBarCount);
                    }
                }
                if (nNbr > 0) av = apply_nbr(g0 + (ready ? before0 : 0), g0 + (ready ? before1 : 0));
                if (ready) break;
                if (t0 == 0) t0 = global_ns();
                if (global_ns() - t0 > waitNs) {
                    aborted = true;
                    break;
                }
                __nanosleep(32);
            }
            if (aborted) break;
            const int xN = tr.x;
            if (!lone)
                for (unsigned rem = accBits; rem;) {
                    // 4 at a time, their couplings in flight together
                    float j[4], dj[4];
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int f = rem ? __ffs(rem) - 1 : 0;
                        dj[t] = rem ? __shfl_sync(FULL, d, f) : 0.f;
                        j[t] = rem ? __ldg(J + (size_t)__shfl_sync(FULL, x, f) * ldJ + xN) : 0.f;
                        rem &= rem - 1u;
                    }
#pragma unroll
                    for (int t = 0; t < 4; ++t) Fv = __fmaf_rn(dj[t], j[t], Fv);
                }
            x = xN;
            const float *jg = Jg + buf * kJgStride + lane * 33;

            // The trial's decision: mc_trial.h.  The tolerance is the fp32 error bound of
            // sq_common.cuh, the ring's part four times as wide here, for the sums kept over a
            // batch's flips.  A flip adds cz q 2 d J to zA, and changes the signs of a
            // later trial at its site.  (A round that evaluated dE anew, with up to four
            // evaluations for unknown spins, took 970 cycles at two CTAs per SM; the decider is
            // the critical path, at 10 cycles an instruction.  N = 4096, m = 256, 64 steps: 24.2
            // ms before, 20.3 with this; N = 1000, m = 250: 8.0, 6.8.)
            const float kF = fabsf(tr.cz) * 1.52587890625e-5f;
            float c2 = 2.f * tr.cz * qx, ring_ = 0.f, sp = 0.f, zA, tol;
            int sum = 0;
            bool evalNbr = nNbr > 0;  // (one instance of nbr_spins: the loop's code stays small)

            // decide the batch in rounds
            unsigned pending = __ballot_sync(FULL, valid);
            accBits = 0;
            d = 0.f;
            nd0 = nd1 = -1;
            bool first = true;
            for (;;) {
                if (evalNbr) {
                    nbr_spins(b, g0, valid, tr.cand, av, sum);
                    evalNbr = false;
                    const float cbq = tr.cb * qx;
                    ring_ = cbq * (float)sum;
                    sp = fabsf(cbq) * (float)((nd0 >= 0) + (nd1 >= 0));
                }
                if (first) {
                    if (lone) Fv = __fmaf_rn(dLone, gLone, Fv);
                    zA = __fmaf_rn(tr.cz * qx, __fmaf_rn(2.f, Fv, tr.h), -tr.L);
                    tol = __fmaf_rn(kF, fabsf(tr.h) + 2.f * fabsf(Fv) + 1.f, tr.tolC);
                    first = false;
                }
                const float z = zA - ring_;
                const unsigned accM = __ballot_sync(FULL, mc_accepts(z, sp, tol)) & pending;
                const unsigned blkM = __ballot_sync(FULL, mc_open(z, sp, tol)) & pending & ~accM;
                const int fa = accM ? __ffs(accM) - 1 : 32;
                const int fb = blkM ? __ffs(blkM) - 1 : 32;
                if (fb < fa) {
                    // undecided lanes below fb reject
                    pending &= ~((1u << fb) - 1u);
                    if (lane == 0 && publish) st_relaxed_u64(myLog + b, log_word(b, fb, accBits));
                    const int w0 = __shfl_sync(FULL, nd0, fb), w1 = __shfl_sync(FULL, nd1, fb);
                    if (w0 < 0 && w1 < 0) {
                        // fb is too near its threshold: the exact warp decides its trial in FP64
                        // from the exact field (every flip before the trial is in qs), for each
                        // value of the neighbours' spin sum; then the round is evaluated again.
                        // (The decider's arrival on a named barrier wakes the exact warp, which
                        // sleeps there between requests; the decider's wait is bounded.)
                        if (lane == fb) {
                            S.exX = x;
                            S.exQ = qx;
                            S.exU = tr.u;
                            S.exIter = g0 + lane;
                        }
                        ++exSeq;
                        __syncwarp();
                        __threadfence_block();
                        bar_arrive(kBarExReq, 64);
                        if (!wait_until(waitNs, [&] { return uniform_acquire(&S.exDone) == exSeq; })) {
                            aborted = true;
                            break;
                        }
                        if (lane == fb) mc_answer((S.exBits >> ((sum + 2) >> 1)) & 1, zA, tol);
                        continue;
                    }
                    // fb waits for its neighbour trials
                    if (!wait_until(waitNs, [&] {
                            av = uniform_acquire64(&S.logAvail);
                            return avail_of(av, 0) > w0 && (nNbr < 2 || avail_of(av, 1) > w1);
                        })) {
                        aborted = true;
                        break;
                    }
                    evalNbr = true;  // (the ghost rows and A are unchanged within the batch)
                    continue;
                }
                if (fa == 32) break;  // every undecided lane rejects
                // undecided lanes below fa reject; fa flips
                const int xf = __shfl_sync(FULL, x, fa);
                const float df = -2.f * __shfl_sync(FULL, qx, fa);
                accBits |= 1u << fa;
                pending &= ~((2u << fa) - 1u);
                // trials through fa are decided: make them visible to the neighbours
                if (lane == 0 && pending && publish) st_relaxed_u64(myLog + b, log_word(b, fa + 1, accBits));
                if (lane == fa) {
                    qs[x] = (int8_t)(qx > 0.f ? -1 : 1);
                    d = df;
                    if (traced) {
                        const int s = (g0 + lane) / N, k = g0 + lane - s * N;
                        uint32_t bitIdx = (uint32_t)k * (uint32_t)m + (uint32_t)y;
                        atomicOr(&T.trace[(size_t)s * wordsPerStep + (bitIdx >> 5)], 1u << (bitIdx & 31));
                    }
                }
                if (!pending) break;
                if (lane > fa) {
                    const float dJ = df * (((pred >> fa) & 1u) ? jg[fa] : __ldg(J + (size_t)xf * ldJ + x));
                    zA = __fmaf_rn(c2, dJ, zA);
                    tol = __fmaf_rn(2.f * kF, fabsf(dJ), tol);
                    if (x == xf) {
                        qx = -qx;
                        c2 = -c2;
                        zA = -(zA + tr.L) - tr.L;
                        ring_ = -ring_;
                    }
                }
            }
            if (aborted) break;
            __syncwarp();
            if (lane == 0) {
                S.decDone = b + 1;  // this batch's buffer is free
                if (publish) st_relaxed_u64(myLog + b, log_word(b, nValid, accBits));
            }
            accepted += (unsigned long long)__popc(accBits);
        }
        // the last batch's flips, as at the head of the next
        bar_sync(2, kBarCount);
        if ((accBits >> lane) & 1u) flips[__popc(accBits & ((1u << lane) - 1u))] = make_int2(x, __float_as_int(d));
        if (lane == 0) S.nflip = __popc(accBits);
        __syncwarp();
        __threadfence_block();
        bar_arrive(1, kBarCount);
        bar_sync(2, kBarCount);  // the updaters are done with the last flips
        if (lane == 0) {
            if (aborted && T.status) atomicExch(T.status, (int)kErrTimeout);
            if (T.accepted) atomicAdd(T.accepted, accepted);
            S.nflip = -1;
            S.done = 1;
        }
        __syncwarp();
        __threadfence_block();
        bar_arrive(1, kBarCount);
        bar_arrive(kBarExReq, 64);  // the exact warp sees done and leaves
    } else if (warp == 1) {
        // -------------------------------------------------------------- helper
        // lane l < 4 polls word (avail[n] >> 5) + dw of neighbour n = l & 1, dw = l >> 1
        int avail0 = 0, avail1 = 0;
        const int n = lane & 1, dw = lane >> 1;
        const unsigned long long *nbLog = outLog + (size_t)(n ? nbr1 : nbr0) * nWords;
        while (nNbr > 0 && !__shfl_sync(FULL, (int)S.done, 0)) {
            const int an = n ? avail1 : avail0;
            const int w = (an >> 5) + dw;
            unsigned long long v = 0;
            if (lane < 4 && n < nNbr && w * 32 < Itot && w < (S.applied[n] >> 5) + kLogWords)
                v = ld_relaxed_u64(nbLog + w);
            bool moved = false;
#pragma unroll
            for (int nn = 0; nn < 2; ++nn) {
                int &a = nn ? avail1 : avail0;
#pragma unroll
                for (int ww = 0; ww < 2; ++ww) {
                    const unsigned long long vv = __shfl_sync(FULL, v, nn + 2 * ww);
                    const int wv = __shfl_sync(FULL, w, nn + 2 * ww);
                    // words are consumed in order: the second only after the first is complete
                    if (nn >= nNbr || wv != (a >> 5) || (int)(vv >> 38) != wv + 1) break;
                    const int c = (int)((vv >> 32) & 63u);
                    if (wv * 32 + c <= a) break;
                    if (lane == 0) nlog[nn * kLogWords + (wv & (kLogWords - 1))] = (uint32_t)vv;
                    a = wv * 32 + c;
                    moved = true;
                    if (c < min(32, Itot - wv * 32)) break;  // batch still being decided
                }
            }
            if (moved) {
                __syncwarp();
                if (lane == 0)
                    st_release_cta64(&S.logAvail, (unsigned long long)(unsigned)avail0 |
                                                      ((unsigned long long)(unsigned)avail1 << 32));
            }
        }
    } else if (warp == kExactWarp) {
        // --------------------------------------------------------- exact warp
        // Sleeps on a named barrier until the decider posts a flagged trial (or
        // the end of the sweep) and arrives on it: sums
        // its exact field (the integer row sum, as the one-CTA kernel computes it)
        // and decides it in FP64 for each value of the neighbours' spin sum (lane
        // k < 3: the sum 2k - 2).
        for (int seq = 1;; ++seq) {
            bar_sync(kBarExReq, 64);
            if (S.done) break;
            const int xr = S.exX;
            const float qr = S.exQ, ur = S.exU;
            const int sl = S.exIter / N;
            const float Gr = T.G ? T.G[sl] : T.Gs, br = T.beta ? T.beta[sl] : T.betas;
            const double hr = T.h64 ? T.h64[xr] : (double)hs[xr];
            const double F = T.J64 ? exact_field_warp(T.J64 + (size_t)xr * N, qs, N)
                                   : exact_field_warp(T.J + (size_t)xr * T.ldJ, qs, N);
            const int ok = lane < 3 ? exact_accept(sa, true, qr, hr, F, lane == 0 ? -1.f : 1.f, lane == 2 ? 1.f : -1.f,
                                                   m, Gr, br, ur)
                                    : 0;
            const unsigned bits = __ballot_sync(FULL, ok) & 7u;
            if (lane == 0) {
                S.exBits = (int)bits;
                st_release_cta(&S.exDone, seq);
            }
            __syncwarp();
        }
    } else if (warp < kUpdWarp0) {
        // --------------------------------------------------------- prefetchers
        const int pw = warp - 2;
        int s = 0, k = lane + 32 * pw, cs = -1;
        while (k >= N) {
            k -= N;
            ++s;
        }
        StepConst sc = {0.f, 0.f, 0.f};
        McConst mc = {0.f, 0.f, 0.f, 0.f};
        int own0 = -1, own1 = -1;  // kSmall: the neighbours' sites of this warp's last batch (p - 2)
        for (int p = pw; p < nBatches; p += kPf) {
            // buffer p % kPre is free once the decider has finished batch p - kPre,
            // and ring slots j - kRing are applied for the neighbours' iterations j of batch p
            const int jEnd = 32 * p + 32;
            int stop = 0;
            if (!wait_until<kPrefetchSleepNs>(waitNs, [&] {
                    int ok = 0;
                    if (lane == 0) {
                        stop = S.done;
                        ok = stop || (S.decDone > p - kPre && (nNbr < 1 || S.applied[0] + kRing >= jEnd) &&
                                      (nNbr < 2 || S.applied[1] + kRing >= jEnd));
                    }
                    return __shfl_sync(FULL, ok, 0) != 0;
                }))
                break;
            if (__shfl_sync(FULL, stop, 0)) break;
            __threadfence_block();
            const int buf = p & (kPre - 1);
            const int j = 32 * p + lane;
            const bool valid = j < Itot;
            int x = 0;
            float u = 0.f;
            if (valid) {
                u32x4 r = draw(T.seed, (uint32_t)k, (uint32_t)y, T.step0 + (uint32_t)s, tag);
                x = draw_index(r.x, N);
                u = draw_unit(r.y);
                if (s != cs) {
                    const float G = T.G ? T.G[s] : T.Gs, beta = T.beta ? T.beta[s] : T.betas;
                    sc = step_const(T.algo, m, G, beta);
                    mc = mc_const(sa, sc.twoDivM, sc.coef, sc.rate);
                    cs = s;
                }
            }
            // the in-batch gathers J[x_f][x_i] (i > f) are needed only for the lanes f
            // that accept: predict them from the current (a few batches stale) field,
            // spins and ghost rows with a margin for the drift; the decider gathers
            // the row of an accepting lane that was not predicted itself
            unsigned pred;
            {
                const volatile float *vF = Fs, *vh = hs;
                const volatile int8_t *vq = qs;
                const volatile uint32_t *vg = reinterpret_cast<const volatile uint32_t *>(ghost);
                const float qx = (float)vq[x], hx = vh[x], fx = vF[x];
                float qn0 = ((vg[2 * (x >> 5)] >> (x & 31)) & 1u) ? 1.f : -1.f;
                float qn1 = nNbr > 1 ? (((vg[2 * (x >> 5) + 1] >> (x & 31)) & 1u) ? 1.f : -1.f) : qn0;
                const float dE = sa ? dense_sa_dE(qx, hx, fx) : dense_sqa_dE(qx, hx, fx, qn0, qn1, sc.twoDivM, sc.coef);
                const float margin = (sa ? 4.f : 2.f * sc.twoDivM) * kFieldDrift;
                const float dEm = dE - margin;
                pred = __ballot_sync(FULL, valid && (dEm < 0.f || __fmul_rn(dEm, sc.rate) < neg_log_unit(u)));
            }
            float v[kPredRows];
            {
                unsigned r = pred;
#pragma unroll
                for (int t = 0; t < kPredRows; ++t) {
                    if (!r) break;
                    const int f = __ffs(r) - 1;
                    r &= r - 1u;
                    const int xf = __shfl_sync(FULL, x, f);
                    v[t] = (lane > f && valid) ? __ldg(T.J + (size_t)xf * T.ldJ + x) : 0.f;
                }
            }
            // the neighbours' sites of the same iterations (while the gathers are in
            // flight): ring entries and the batch's site bitmaps; then, per lane and
            // neighbour, the latest kCand iterations of batches p - 2 .. p that hit
            // the lane's site up to its limit (-2: more than kCand)
            uint32_t cands = kNoCands;
            auto put_cands = [&](int nn, int c0, int c1) {
                const uint32_t e0 = c0 == -2 ? kManyCand : c0 < 0 ? kNoCand : (uint32_t)(32 * p + 32 - c0);
                const uint32_t e1 = c1 < 0 ? kNoCand : (uint32_t)(32 * p + 32 - c1);
                cands = nn ? (cands & 0xffffu) | (e0 << 16) | (e1 << 24) : (cands & 0xffff0000u) | e0 | (e1 << 8);
            };
            if (nNbr > 0) {
                uint32_t *bp = bm + (p & (kBmSlots - 1)) * kBmWords;
                bp[lane] = 0u;
                bp[lane + 32] = 0u;
                if (nNbr > 1) {
                    bp[kBmSlots * kBmWords + lane] = 0u;
                    bp[kBmSlots * kBmWords + lane + 32] = 0u;
                }
                __syncwarp();
                int cur0 = -1, cur1 = -1;
                if (valid) {
                    cur0 = draw_index(draw(T.seed, (uint32_t)k, (uint32_t)nbr0, T.step0 + (uint32_t)s, tag).x, N);
                    ring[j & (kRing - 1)] = cur0;
                    atomicOr(&bp[(cur0 & (kBmBits - 1)) >> 5], 1u << (cur0 & 31));
                    if (nNbr > 1) {
                        cur1 = draw_index(draw(T.seed, (uint32_t)k, (uint32_t)nbr1, T.step0 + (uint32_t)s, tag).x, N);
                        ring[kRing + (j & (kRing - 1))] = cur1;
                        atomicOr(&bp[kBmSlots * kBmWords + ((cur1 & (kBmBits - 1)) >> 5)], 1u << (cur1 & 31));
                    }
                }
                // batch p - 1 (the other prefetcher's) must be in the ring; its tag's slot
                // may already hold a later batch (batch p - 2 is this warp's own)
                if (!kSmall) {
                    __syncwarp();
                    if (lane == 0) st_release_cta(&S.ringTag[buf], p + 1);
                    if (p > 0 && !wait_until<kPrefetchSleepNs>(
                                     waitNs, [&] { return uniform_acquire(&S.ringTag[(p - 1) & (kPre - 1)]) >= p; }))
                        break;
                }
                __syncwarp();
                const int hb = x & (kBmBits - 1);
                if (kSmall) {
                    // the sites of the neighbours' iterations of batches p - 1 (drawn again: the
                    // ring's entries for it are the other prefetcher's) and p - 2 (this warp's last)
                    int sites[2][3];
#pragma unroll
                    for (int nn = 0; nn < 2; ++nn) {
                        const int j1 = 32 * (p - 1) + lane;
                        int s1 = -1;
                        if (nn < nNbr && j1 >= 0) {
                            const int s2 = k >= 32 ? s : j1 / N, k2 = k >= 32 ? k - 32 : j1 - s2 * N;
                            s1 = draw_index(draw(T.seed, (uint32_t)k2, (uint32_t)(nn ? nbr1 : nbr0),
                                                 T.step0 + (uint32_t)s2, tag).x, N);
                        }
                        sites[nn][0] = nn ? cur1 : cur0;
                        sites[nn][1] = s1;
                        sites[nn][2] = nn ? own1 : own0;
                    }
                    own0 = cur0;
                    own1 = cur1;
                    // per batch: the positions of each site in a table per neighbour (cleared
                    // again after use), read at the lane's own site; latest batch first
                    uint32_t *tab0 = siteTab + pw * 2 * kSmallN, *tab1 = tab0 + kSmallN;
                    int c0[2] = {-1, -1}, c1[2] = {-1, -1}, cnt[2] = {0, 0};
#pragma unroll 1
                    for (int q = 0; q < 3; ++q) {
                        const int s0 = q == 0 ? sites[0][0] : q == 1 ? sites[0][1] : sites[0][2];
                        const int s1 = q == 0 ? sites[1][0] : q == 1 ? sites[1][1] : sites[1][2];
                        if (s0 >= 0) atomicOr(&tab0[s0], 1u << lane);
                        if (s1 >= 0) atomicOr(&tab1[s1], 1u << lane);
                        __syncwarp();
                        unsigned mk[2] = {valid ? tab0[x] : 0u, valid ? tab1[x] : 0u};
                        __syncwarp();
                        if (s0 >= 0) tab0[s0] = 0u;
                        if (s1 >= 0) tab1[s1] = 0u;
                        __syncwarp();
#pragma unroll
                        for (int nn = 0; nn < 2; ++nn) {
                            const int lim = lane - 1 + (nn ? before1 : before0);
                            unsigned m = mk[nn];
                            if (q == 0) m &= lim < 0 ? 0u : (lim >= 31 ? ~0u : (2u << lim) - 1u);
                            cnt[nn] += __popc(m);
                            while (m) {  // from the batch's last iteration
                                const int t = 31 - __clz(m);
                                m &= ~(1u << t);
                                const int jj = 32 * (p - q) + t;
                                if (c0[nn] < 0)
                                    c0[nn] = jj;
                                else if (c1[nn] < 0)
                                    c1[nn] = jj;
                            }
                        }
                    }
#pragma unroll
                    for (int nn = 0; nn < 2; ++nn)
                        if (nn < nNbr) put_cands(nn, cnt[nn] > kCand ? -2 : c0[nn], cnt[nn] > kCand ? -1 : c1[nn]);
                } else {
#pragma unroll
                for (int nn = 0; nn < 2; ++nn) {
                    if (nn >= nNbr) break;
                    const uint32_t *bmn = bm + nn * kBmSlots * kBmWords;
                    const int prev = p > 0 ? ring[nn * kRing + ((32 * (p - 1) + lane) & (kRing - 1))] : -1;
                    const int prev2 = p > 1 ? ring[nn * kRing + ((32 * (p - 2) + lane) & (kRing - 1))] : -1;
                    const int cur = nn ? cur1 : cur0;
                    const int lim = lane - 1 + (nn ? before1 : before0);  // latest iteration of batch p a lane needs
                    auto marked = [&](int q) {
                        return q >= 0 && ((bmn[(q & (kBmSlots - 1)) * kBmWords + (hb >> 5)] >> (hb & 31)) & 1u);
                    };
                    const bool flag = valid && (marked(p) || marked(p - 1) || marked(p - 2));
                    int c0 = -1, c1 = -1;
                    unsigned hits = __ballot_sync(FULL, flag);
                    while (hits) {
                        const int i = __ffs(hits) - 1;
                        hits &= hits - 1u;
                        const int xi = __shfl_sync(FULL, x, i), li = __shfl_sync(FULL, lim, i);
                        const unsigned mc = __ballot_sync(FULL, cur == xi && lane <= li);
                        const unsigned mp = __ballot_sync(FULL, prev == xi);
                        const unsigned mq = __ballot_sync(FULL, prev2 == xi);
                        if (lane == i) {
                            if (__popc(mc) + __popc(mp) + __popc(mq) > kCand) {
                                c0 = -2;
                            } else {
                                // the latest two: batch p first, then p - 1, then p - 2
                                const unsigned ms[3] = {mc, mp, mq};
#pragma unroll
                                for (int q = 0; q < 3; ++q) {
                                    for (unsigned r = ms[q]; r; r &= ~(1u << (31 - __clz(r)))) {
                                        const int jj = 32 * (p - q) + 31 - __clz(r);
                                        if (c0 < 0)
                                            c0 = jj;
                                        else
                                            c1 = jj;
                                    }
                                }
                            }
                        }
                    }
                    put_cands(nn, c0, c1);
                }
                }
            }
            float *jg = Jg + buf * kJgStride + lane * 33;
            {
                unsigned r = pred;
#pragma unroll
                for (int t = 0; t < kPredRows; ++t) {
                    if (!r) break;
                    const int f = __ffs(r) - 1;
                    r &= r - 1u;
                    jg[f] = v[t];
                }
                for (; r; r &= r - 1u) {  // more predicted rows than registers: gather the rest here
                    const int f = __ffs(r) - 1;
                    const int xf = __shfl_sync(FULL, x, f);
                    jg[f] = (lane > f && valid) ? __ldg(T.J + (size_t)xf * T.ldJ + x) : 0.f;
                }
            }
            if (lane == 0) prePred[buf] = pred;
            {
                PreTrial tr;
                tr.x = x;
                tr.h = hs[x];
                tr.L = mc_L(mc, neg_log_unit(u));
                tr.cz = mc.cz;
                tr.cb = mc.cb;
                tr.tolC = mc_tol(mc, tr.L);
                tr.u = u;
                tr.cand = cands;
                pre[buf * 32 + lane] = tr;
            }
            __syncwarp();
            if (lane == 0) st_release_cta(&S.readyTag[buf], p + 1);
            k += 32 * kPf;
            while (k >= N) {
                k -= N;
                ++s;
            }
        }
    } else {
        // ----------------------------------------------------------- updaters
        const int ut = tid - 32 * kUpdWarp0;
        const int n4 = N / 4;
        float4 *F4 = reinterpret_cast<float4 *>(Fs);
        bar_arrive(2, kBarCount);
        for (;;) {
            bar_sync(1, kBarCount);
            const int nf = S.nflip;
            if (nf < 0) break;
            for (int c0 = ut; c0 < n4; c0 += 4 * kMcUpdaters) {
                float4 f[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    int c = c0 + t * kMcUpdaters;
                    if (c < n4) f[t] = F4[c];
                }
                for (int q = 0; q < nf; ++q) {
                    const int2 fl = flips[q];
                    const float d = __int_as_float(fl.y);
                    const float4 *Jr = reinterpret_cast<const float4 *>(T.J + (size_t)fl.x * T.ldJ);
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        int c = c0 + t * kMcUpdaters;
                        if (c < n4) {
                            float4 j = __ldg(Jr + c);
                            f[t].x = __fmaf_rn(d, j.x, f[t].x);
                            f[t].y = __fmaf_rn(d, j.y, f[t].y);
                            f[t].z = __fmaf_rn(d, j.z, f[t].z);
                            f[t].w = __fmaf_rn(d, j.w, f[t].w);
                        }
                    }
                }
#pragma unroll
                for (int t = 0; t < 4; ++t) {
                    int c = c0 + t * kMcUpdaters;
                    if (c < n4) F4[c] = f[t];
                }
            }
            // the last N % 4 fields (J rows start on 16-byte boundaries: ldJ % 4 == 0)
            if (ut < N - 4 * n4) {
                const int i = 4 * n4 + ut;
                float f = Fs[i];
                for (int q = 0; q < nf; ++q) {
                    const int2 fl = flips[q];
                    f = __fmaf_rn(__int_as_float(fl.y), __ldg(T.J + (size_t)fl.x * T.ldJ + i), f);
                }
                Fs[i] = f;
            }
            __threadfence_block();
            bar_arrive(2, kBarCount);
        }
    }
    __syncthreads();
    for (int i = tid; i < N; i += kMcThreads) {
        T.F[(size_t)y * N + i] = Fs[i];
        T.q[(size_t)y * N + i] = qs[i];
    }
}

static size_t multi_smem_bytes(int N) {
    size_t ghostStride = (size_t)((N + 31) / 32 + 1) & ~(size_t)1;
    return pre_offset(N) + (size_t)kPre * 32 * sizeof(PreTrial) + 2 * ghostStride * 4 +
           (size_t)2 * kBmSlots * kBmWords * 4 + 2 * kRing * 4 + 2 * kLogWords * 4 + kPre * 4 +
           32 * 8 + (size_t)((N + 15) & ~15) + 16 + (N <= kSmallN ? (size_t)kPf * 2 * kSmallN * 4 : 0);
}

// every instance: bit 0 kHooks, bit 1 kSmall, bit 2 kSA, bit 3 four CTAs per SM (else two)
template <int I>
static const void *multi_instance() {
    return (const void *)dense_sweep_multi<(I & 1) != 0, (I & 2) != 0, (I & 4) != 0, (I & 8) ? 4 : 2>;
}
static const void *multi_kernel(int i) {
    static const void *const k[16] = {
        multi_instance<0>(),  multi_instance<1>(),  multi_instance<2>(),  multi_instance<3>(),
        multi_instance<4>(),  multi_instance<5>(),  multi_instance<6>(),  multi_instance<7>(),
        multi_instance<8>(),  multi_instance<9>(),  multi_instance<10>(), multi_instance<11>(),
        multi_instance<12>(), multi_instance<13>(), multi_instance<14>(), multi_instance<15>()};
    return k[i];
}

// resident CTAs of rows of N spins, with the registers allotted for two and for four per SM
struct MultiCapacity {
    int two, four;
};

// Callers on several host threads share the kernels' shared memory limits (set once per
// device, to the most that the device allows, and never lowered: another thread's launch
// may need more than this caller's N) and the answers, kept per device and N.
static MultiCapacity multi_capacity(int N) {
    struct Device {
        int sms = 0, maxDyn = -1;
        std::map<int, MultiCapacity> byN;
    };
    static std::mutex mu;
    static std::map<int, Device> devices;
    std::lock_guard<std::mutex> lock(mu);
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return {0, 0};
    }
    Device &d = devices[dev];
    if (d.maxDyn < 0) {
        int optin = 0, maxDyn = 1 << 30;
        cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
        // every instance: the launch takes the one the tasks' flags and sizes ask for
        for (int i = 0; i < 16; ++i) {
            cudaFuncAttributes fa;
            if (cudaFuncGetAttributes(&fa, multi_kernel(i)) != cudaSuccess ||
                cudaFuncSetAttribute(multi_kernel(i), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     optin - (int)fa.sharedSizeBytes) != cudaSuccess) {
                cudaGetLastError();
                return {0, 0};
            }
            maxDyn = std::min(maxDyn, optin - (int)fa.sharedSizeBytes);
        }
        d.maxDyn = maxDyn;
    }
    const size_t smem = multi_smem_bytes(N);
    if (smem > (size_t)d.maxDyn) return {0, 0};
    const auto known = d.byN.find(N);
    if (known != d.byN.end()) return known->second;
    int perSm[2] = {1 << 30, 1 << 30};
    for (int i = 0; i < 16; ++i) {
        int ps = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&ps, multi_kernel(i), mc_threads(i & 8 ? 4 : 2), smem) !=
            cudaSuccess) {
            cudaGetLastError();
            return {0, 0};
        }
        perSm[i >> 3] = std::min(perSm[i >> 3], ps);
    }
    return d.byN[N] = {perSm[0] * d.sms, std::max(perSm[0], perSm[1]) * d.sms};
}

}  // namespace sq103

using namespace sq103;

extern "C" {

SQ103_API unsigned long long sq103_dense_ws_bytes(int N, int m, int nSteps) {
    unsigned long long nWords = ((unsigned long long)nSteps * N + 31) / 32;
    return (unsigned long long)m * nWords * 8 + 256;
}

SQ103_API int sq103_dense_multicta_ok(int N, int m, int algo) {
    if (algo != kColoring && algo != kSANaive) return 0;
    if (N < 64 || m < 2) return 0;
    return m <= multi_capacity(N).four ? 1 : 0;
}

// n instances in one cooperative launch (see McPack)
static int launch_pack(const sq103_dense_task *tasks, int n, void *stream) {
    cudaStream_t st = (cudaStream_t)stream;
    if (n < 1 || n > kMaxPack) return kErrBadShape;
    McPack P = {};
    P.n = n;
    int maxN = 0, ctas = 0;
    bool hooks = false;
    int sas = 0;
    for (int i = 0; i < n; ++i) {
        const sq103_dense_task &t = tasks[i];
        hooks |= (t.flags & (kFlagShortWaits | kFlagWithholdTrotter0)) != 0 || t.trace;
        sas += t.algo == kSANaive;
        const int N = t.N, m = t.m;
        if (t.algo != kColoring && t.algo != kSANaive) return kErrBadShape;
        if (N < 64 || m < 2 || t.nSteps < 1) return kErrBadShape;
        if ((long long)t.nSteps * N >= (1ll << 31)) return kErrBadShape;
        // rows of J are read as float4
        if ((t.ldJ & 3) || (reinterpret_cast<uintptr_t>(t.J) & 15)) return kErrBadShape;
        if (!t.ws || t.wsBytes < sq103_dense_ws_bytes(N, m, t.nSteps)) return kErrCapacity;
        P.t[i] = t;
        P.outLog[i] = reinterpret_cast<unsigned long long *>(t.ws);
        P.nWords[i] = (int)(((long long)t.nSteps * N + 31) / 32);
        P.base[i] = ctas;
        ctas += m;
        maxN = std::max(maxN, N);
    }
    if (sas && sas < n) {  // one algorithm per launch
        std::vector<sq103_dense_task> part[2];
        for (int i = 0; i < n; ++i) part[tasks[i].algo == kSANaive].push_back(tasks[i]);
        const int rc = launch_pack(part[0].data(), (int)part[0].size(), stream);
        return rc != 0 ? rc : launch_pack(part[1].data(), (int)part[1].size(), stream);
    }
    for (int i = n; i <= kMaxPack; ++i) P.base[i] = ctas;
    // every CTA resident at once (cooperative launch); also sets the kernels' shared-memory limits
    const MultiCapacity cap = multi_capacity(maxN);
    if (cap.four < ctas) return kErrCapacity;
    void *args[] = {&P};
    const void *kernel = multi_kernel((hooks ? 1 : 0) | (maxN <= kSmallN ? 2 : 0) | (sas ? 4 : 0) | (ctas <= cap.two ? 0 : 8));
    return (int)cudaLaunchCooperativeKernel(kernel, dim3(ctas), dim3(mc_threads(ctas <= cap.two ? 2 : 4)), args, multi_smem_bytes(maxN), st);
}

// launched from sq103_dense_anneal (dense.cu) when the shape and workspace allow it
int sq103_dense_anneal_multi(const sq103_dense_task *t, void *stream) { return launch_pack(t, 1, stream); }

SQ103_API int sq103_dense_anneal_pack(const sq103_dense_task *tasks, int n, void *stream) {
    if (!tasks) return kErrBadShape;
    return launch_pack(tasks, n, stream);
}

SQ103_API int sq103_dense_multicta_capacity(int N) { return N >= 64 ? multi_capacity(N).four : 0; }

}  // extern "C"
