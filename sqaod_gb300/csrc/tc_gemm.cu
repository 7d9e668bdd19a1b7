// tc_gemm.cu -- local-field refresh on the 5th-generation tensor cores
// (tcgen05), operands staged by TMA, accumulators in TMEM.
//
//   F[y][r] = sum_k q[y][k] B[r][k]      (dense: B = J, symmetric, so F = q J;
//                                          bipartite: B = J or J^T)
//
// The refresh replaces the reference's J.q contractions
// (DeviceDotJqVec4, sqaodc/cuda/DeviceBatchedDot.cuh:247-262, and the cuBLAS
// SGEMMs of CUDABipartiteGraphAnnealer.cu:393-401).
//
// Exactness.  The couplings are held as 31-bit fixed point, B ~ 2^-S * (D0 +
// 2^8 D1 + 2^16 D2 + 2^24 D3), with S chosen from the matrix's largest
// magnitude and every digit D_t a signed integer of magnitude <= 128, exact in
// bf16.  The spins are +-1, so each digit's contraction P_t = q . D_t is a sum
// of integers of magnitude <= 128, and every partial sum is an integer below
// 2^24 for K < 2^17: the fp32 accumulation in TMEM is exact whatever the
// tensor core's adder order, alignment or truncation.  The epilogue combines
// sum_t 2^(8t) P_t in 64-bit integers and rounds once to fp32.  The only error
// left is the quantisation of B (below 2^-29 of the largest |B| per element),
// far below the fp32 rounding of the result.
//
// Energies (tc_digit_gemm<double>).  The FP64 energies need the row sums to FP64
// accuracy.  Four more digit planes hold what the first four round away, 31 bits
// further down (62 below the largest |B|), and a second contraction adds them: both
// sums are exact integers, and the row sum is rounded once, in FP64.
//
// Kernel (one CTA per 128 x 64 output tile, 128 threads):
//   thread 0    TMA producer: per 64-wide K block, the spin tile (128 x 64 bf16)
//               and the four digit tiles (64 x 64 bf16 each) into a 4-stage
//               shared-memory ring (128B swizzle), mbarrier-tracked;
//   thread 32   MMA issuer: per K block 4 tcgen05.mma kind::f16 (M = 128, N = 256,
//               K = 16): the four digit tiles lie one after another in the stage,
//               so one MMA takes all four as 256 rows of B and reads the spins
//               once (four MMAs of N = 64 took 1290 cycles per K block, bound by
//               shared-memory reads: 43 us for 2047 x 3001, m = 200, now 25); tcgen05.commit frees each stage;
//   all 4 warps epilogue: tcgen05.ld of the four accumulators (a trotter row
//               per thread), integer combination, fp32 through a shared tile so
//               that the stores are whole rows (a thread's own row of 64 stored
//               directly took 7 to 12 thousand cycles of a launch).
// Few output tiles (m or R small) would leave most SMs idle and walk the whole K in
// each: a cluster of 2 or 4 CTAs then takes a tile, each a part of K, and adds the
// integer sums through distributed shared memory.  Integer addition is exact, so
// the result does not depend on the split.
// Every mbarrier wait is bounded by the global timer; on timeout the CTA
// records status 1, lets the copies it issued land (bounded), frees TMEM and
// returns.  Two test flags make a wait run out on purpose: the producer skips
// the first K block's copies, and waits give up after 1 ms.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cstdint>

#include "sq_common.cuh"
#include "sq_kernels.h"

namespace sq103 {

constexpr int kTcBM = 128, kTcBN = 64, kTcBK = 64, kTcStages = 4, kTcThreads = 128, kTcDigits = 4;
constexpr int kTcATile = kTcBM * kTcBK * 2;  // 16 KB
constexpr int kTcBTile = kTcBN * kTcBK * 2;  // 8 KB
constexpr int kTcStageBytes = kTcATile + kTcDigits * kTcBTile;
constexpr int kTcSmemBytes = kTcStages * kTcStageBytes + 1024 + 256;
constexpr int kTcOutLd = kTcBN + 1;                                     // row stride of the output tile
constexpr int kTcOutBytes = (kTcBM * kTcOutLd * 8 + 1023) / 1024 * 1024;  // its bytes (FP64 row sums)
constexpr int kTcTmemCols = 256;  // 4 accumulators of 64 fp32 columns
constexpr unsigned long long kTcWaitNs = 2000000000ull, kTcShortWaitNs = 1000000ull;
constexpr int kTcAdd = 4;  // launch flag (see tc_digit_gemm)
constexpr int kTcHeader = 256;  // digit buffer: exponent word, int shift S, then the four planes

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long tc_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// bounded wait for the phase with the given parity; false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned long long limitNs) {
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = tc_now();
    while (!mbar_try_wait(bar, parity))
        if (tc_now() - t0 > limitNs) return false;
    return true;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_addr(dst)),
        "l"((uint64_t)map), "r"(smem_addr(bar)), "r"(x), "r"(y)
        : "memory");
}

__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y, int z) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::
            "r"(smem_addr(dst)),
        "l"((uint64_t)map), "r"(smem_addr(bar)), "r"(x), "r"(y), "r"(z)
        : "memory");
}

// shared-memory matrix descriptor: K-major, 128B swizzle, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;             // leading byte offset (unused with swizzle)
    d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset
    d |= (uint64_t)1 << 46;             // descriptor version
    d |= (uint64_t)2 << 61;             // 128B swizzle
    return d;
}

// instruction descriptor, kind::f16: bf16 x bf16 -> f32, A and B K-major, M x N
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t dtmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// 16 consecutive fp32 columns of the warp's 32 TMEM lanes (one lane per thread)
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}

__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the address of a CTA-local shared address in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t peer_addr(const void *p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_addr(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ long long peer_load64(uint32_t a) {
    long long v;
    asm volatile("ld.shared::cluster.b64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ int peer_load32(uint32_t a) {
    int v;
    asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}

// v 2^-S, rounded once
template <class Out>
__device__ __forceinline__ Out scaled_sum(long long v, int S);
template <>
__device__ __forceinline__ float scaled_sum<float>(long long v, int S) {  // S in [-126, 126]
    return __fmul_rn(__ll2float_rn(v), __int_as_float((127 - S) << 23));
}
template <>
__device__ __forceinline__ double scaled_sum<double>(long long v, int S) {  // S in [-126, 157]
    return __dmul_rn(__ll2double_rn(v), __longlong_as_double((long long)(1023 - S) << 52));
}

// columns [cz, cz + 64 / SPLIT) of the tile from the integer shares of the cluster's
// CTAs, a row per thread, sixteen loads in flight
template <int SPLIT, class Out>
__device__ __forceinline__ void add_shares(const long long *red, Out *out, int cz, int row, int S) {
    constexpr int kCols = 64 / SPLIT, kStep = 16 / SPLIT;
    uint32_t peer[SPLIT];
#pragma unroll
    for (int p = 0; p < SPLIT; ++p) peer[p] = peer_addr(&red[cz * kTcBM + row], (uint32_t)p);
#pragma unroll 1
    for (int c = 0; c < kCols; c += kStep) {
        long long v[kStep][SPLIT];
#pragma unroll
        for (int k = 0; k < kStep; ++k)
#pragma unroll
            for (int p = 0; p < SPLIT; ++p) v[k][p] = peer_load64(peer[p] + (uint32_t)((c + k) * kTcBM * 8));
#pragma unroll
        for (int k = 0; k < kStep; ++k) {
            long long sum = v[k][0];
#pragma unroll
            for (int p = 1; p < SPLIT; ++p) sum += v[k][p];
            out[row * kTcOutLd + cz + c + k] = scaled_sum<Out>(sum, S);
        }
    }
}

// F tile (128 trotters x 64 outputs) = sum_t 2^(8t - S) (q . D_t); gridDim.z CTAs
// (a cluster) share the tile, each K blocks [nK z / gridDim.z, nK (z + 1) / gridDim.z)
// Out float: fields.  double: row sums; flag kTcAdd adds to those in F, and a matrix
// with a non-finite value (its exponent word) gives NaN.
template <class Out>
__global__ void __launch_bounds__(kTcThreads) tc_digit_gemm(const __grid_constant__ CUtensorMap tmA,
                                                            const __grid_constant__ CUtensorMap tmB,
                                                            const int *shiftPtr, Out *F, int ldF, int M, int R,
                                                            int Kp, int flags, int *status) {
    extern __shared__ __align__(16) unsigned char tc_smem_raw[];
    unsigned char *smem = (unsigned char *)(((uintptr_t)tc_smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kTcStages * kTcStageBytes);
    uint64_t *empty = full + kTcStages;
    uint64_t *done = empty + kTcStages;
    uint32_t *tmemSlot = reinterpret_cast<uint32_t *>(done + 1);
    __shared__ int abortFlag, okFlag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * kTcBM, n0 = blockIdx.x * kTcBN;
    const int split = (int)gridDim.z, z = (int)blockIdx.z;
    const int kb0 = Kp / kTcBK * z / split, nK = Kp / kTcBK * (z + 1) / split - kb0;  // this CTA's K blocks
    const unsigned long long waitNs = (flags & 2) ? kTcShortWaitNs : kTcWaitNs;

    if (tid == 0) {
        for (int s = 0; s < kTcStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(tmemSlot)),
                     "r"(kTcTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmemSlot;
    pdl_trigger();
    pdl_wait();  // the spins, and F's last readers

    if (tid == 0) {
        // ---------------------------------------------------------- producer
        // issued[s]: the parity of the latest copy issued into stage s, -1 if none is outstanding
        int issued[kTcStages];
        for (int s = 0; s < kTcStages; ++s) issued[s] = -1;
        for (int kb = 0; kb < nK; ++kb) {
            const int s = kb % kTcStages;
            if (kb >= kTcStages && !mbar_wait(&empty[s], ((kb / kTcStages) - 1) & 1, waitNs)) {
                abortFlag = 1;
                break;
            }
            if ((flags & 1) && kb == 0) continue;  // test hook: stage 0's first copies never come
            unsigned char *a = smem + s * kTcStageBytes;
            mbar_expect_tx(&full[s], kTcStageBytes);
            tma_load_2d(a, &tmA, &full[s], (kb0 + kb) * kTcBK, m0);
#pragma unroll
            for (int t = 0; t < kTcDigits; ++t) tma_load_3d(a + kTcATile + t * kTcBTile, &tmB, &full[s], (kb0 + kb) * kTcBK, n0, t);
            issued[s] = (kb / kTcStages) & 1;
        }
        // let every copy still in flight land before the CTA can leave
        for (int s = 0; s < kTcStages; ++s)
            if (issued[s] >= 0) mbar_wait(&full[s], (uint32_t)issued[s], waitNs);
    } else if (tid == 32) {
        // ---------------------------------------------------------- MMA issuer
        constexpr uint32_t idesc = umma_idesc_bf16(kTcBM, kTcDigits * kTcBN);
        bool ok = true;
        for (int kb = 0; kb < nK; ++kb) {
            const int s = kb % kTcStages;
            if (!mbar_wait(&full[s], (kb / kTcStages) & 1, waitNs) || abortFlag) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a = smem_addr(smem + s * kTcStageBytes);
            const uint64_t adesc = sw128_desc(a);
#pragma unroll
            for (int kk = 0; kk < kTcBK / 16; ++kk)  // K = 16 per MMA: +32 B in the swizzled row
                umma_bf16(tmem, adesc + 2 * kk, sw128_desc(a + kTcATile) + 2 * kk, idesc, (kb | kk) ? 1u : 0u);
            umma_commit(&empty[s]);
        }
        if (!ok) abortFlag = 1;
        umma_commit(done);
    }
    __syncwarp();
    // ---------------------------------------------------------------- epilogue
    const bool got = mbar_wait(done, 0, waitNs);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    bool ok = __syncthreads_and(got ? 1 : 0) && !abortFlag;
    if (!ok && tid == 0 && status) atomicExch(status, (int)kErrTimeout);
    const int S = *shiftPtr;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    // (the ring is idle now) the fp32 tile, rows padded against bank conflicts, and for a
    // split tile this CTA's integer sums, [64 columns][128 rows]
    Out *out = reinterpret_cast<Out *>(smem);
    long long *red = reinterpret_cast<long long *>(smem + kTcOutBytes);
    if (ok) {
        // |P_t| <= 128 Kp: up to 2^22 the sum P + 1.5 2^23 is exact and holds P in its low bits
        const bool narrow = Kp <= (1 << 15);
#pragma unroll 1
        for (int c0 = 0; c0 < kTcBN; c0 += 16) {
            uint32_t p[kTcDigits][16];
#pragma unroll
            for (int t = 0; t < kTcDigits; ++t) tmem_ld16(tmem + lanes + (uint32_t)(t * kTcBN + c0), p[t]);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                long long v;
                if (narrow) {
                    int d[kTcDigits];
#pragma unroll
                    for (int t = 0; t < kTcDigits; ++t)
                        d[t] = __float_as_int(__fadd_rn(__uint_as_float(p[t][j]), 12582912.f)) - 0x4B400000;
                    v = ((long long)(d[3] * 256 + d[2]) << 16) + (d[1] * 256 + d[0]);
                } else {
                    v = 0;
#pragma unroll
                    for (int t = kTcDigits - 1; t >= 0; --t)
                        v = (v << 8) + (long long)__float2int_rn(__uint_as_float(p[t][j]));
                }
                if (split > 1)
                    red[(c0 + j) * kTcBM + tid] = v;
                else
                    out[tid * kTcOutLd + c0 + j] = scaled_sum<Out>(v, S);
            }
        }
    }
    int cols = kTcBN, cz = 0;  // the columns of the tile that this CTA stores
    if (split > 1) {
        if (tid == 0) okFlag = ok ? 1 : 0;
        __syncwarp();
        cluster_sync_all();
        // this CTA's columns: the sums of every CTA's share (none if one gave up)
        for (int p = 0; p < split; ++p) ok = ok && peer_load32(peer_addr(&okFlag, (uint32_t)p));
        cols = kTcBN / split;
        cz = z * cols;
        if (ok) {
            if (split == 2)
                add_shares<2>(red, out, cz, tid, S);
            else
                add_shares<4>(red, out, cz, tid, S);
        }
        __syncwarp();
        cluster_sync_all();  // a CTA's shared memory stays until its peers have read it
    } else {
        __syncthreads();
    }
    if (ok) {
        const int c = cz + tid % cols;  // whole rows of the tile, kTcThreads / cols at a time
        for (int r = tid / cols; r < kTcBM && m0 + r < M; r += kTcThreads / cols)
            if (n0 + c < R) {
                Out v = out[r * kTcOutLd + c], *dst = &F[(size_t)(m0 + r) * ldF + n0 + c];
                if (sizeof(Out) == 8) {
                    if (flags & kTcAdd) v += *dst;
                    if (*reinterpret_cast<const unsigned *>(shiftPtr - 4) == 0x7f800000u) v = (Out)__int_as_float(0x7fffffff);
                }
                *dst = v;
            }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcTmemCols)
                     : "memory");
}

// largest biased exponent of the matrix (atomicMax over the float bit patterns, one per
// block: one per warp of a full grid took 20 us on the one word)
__global__ void __launch_bounds__(256) tc_max_exponent(const float *B, int ld, int rows, int cols, unsigned *out) {
    __shared__ unsigned top;
    if (threadIdx.x == 0) top = 0u;
    __syncthreads();
    unsigned e = 0;
    for (int r = blockIdx.x; r < rows; r += gridDim.x)
#pragma unroll 4
        for (int c = threadIdx.x; c < cols; c += 256) e = max(e, __float_as_uint(B[(size_t)r * ld + c]) & 0x7f800000u);
    e = __reduce_max_sync(0xffffffffu, e);
    if ((threadIdx.x & 31) == 0) atomicMax(&top, e);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(out, top);
}

// shift S: |B| < 2^(E - 126) for the largest biased exponent E, so |B 2^S| < 2^30 with S = 156 - E
__device__ __forceinline__ int tc_shift(unsigned maxExpBits) {
    return min(max(156 - (int)(maxExpBits >> 23), -126), 126);
}

// digit planes D_t[r][k] (r < R rows of output, k < K, row stride ldD, zero padded to ldD):
// B[r][k] = J[r][k] (transpose = 0) or J[k][r] (transpose = 1), J with row stride ldJ
// low: the planes of 2^31 (B 2^S - rint(B 2^S)), the part the planes of B round away (shift S + 31)
__global__ void tc_make_digits(const float *J, int ldJ, int R, int K, int ldD, int transpose, bool low,
                               const unsigned *maxExp, unsigned *header, __nv_bfloat16 *D) {
    const int S = tc_shift(*maxExp);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (low) header[0] = *maxExp;  // (the planes of B hold it already)
        header[4] = (unsigned)(low ? S + 31 : S);
    }
    const float scale = __int_as_float((S + 127) << 23);
    const size_t plane = (size_t)R * ldD;
    for (int r = blockIdx.x; r < R; r += gridDim.x)
    for (int k = threadIdx.x; k < ldD; k += blockDim.x) {
        const size_t i = (size_t)r * ldD + k;
        int v = 0;
        if (k < K) {
            float x = __fmul_rn(transpose ? J[(size_t)k * ldJ + r] : J[(size_t)r * ldJ + k], scale);
            if (low) x = __fmul_rn(__fsub_rn(x, rintf(x)), 2147483648.f);  // exact: |x - rint x| <= 1/2
            v = __float2int_rn(x);
        }
        // balanced base-256 digits: v = d0 + 2^8 d1 + 2^16 d2 + 2^24 d3, d0..d2 in [-128, 127],
        // |d3| <= 64 since |v| < 2^30
#pragma unroll
        for (int t = 0; t < kTcDigits; ++t) {
            const int d = t == kTcDigits - 1 ? v : (int)(int8_t)(v & 0xff);
            D[t * plane + i] = __int2bfloat16_rn(d);
            v = (v - d) >> 8;
        }
    }
}

// *spread = how far, in powers of two, the largest coupling of some row or column of J (R x
// K) lies below the matrix's, of those that hold a coupling the digits round (255 with a
// non-finite coupling).  Up to 5, the digits are as fine as fp32 holds a row's largest
// coupling (2^24 quanta 2^-S or more).  Couplings of one magnitude, and integers below
// 2^30, have no spread; one coupling far above the rest gives the other rows one.
// Blocks below rowBlocks: a warp per row; the rest: 32 columns each.
__global__ void __launch_bounds__(256) tc_spread(const float *J, int ld, int R, int K, const unsigned *maxExp,
                                                 int rowBlocks, int *spread) {
    __shared__ unsigned top[8][32];
    const unsigned E = *maxExp;
    const float scale = __int_as_float((tc_shift(E) + 127) << 23);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned e = 0;  // the largest exponent, bit 0 set when a value is rounded
    auto take = [&](float v) {
        const float x = __fmul_rn(v, scale);
        const unsigned b = __float_as_uint(v) & 0x7f800000u;
        e = max(e & ~1u, b) | (e & 1u) | (x != rintf(x) ? 1u : 0u);
    };
    if ((int)blockIdx.x < rowBlocks) {
        const int r = (int)blockIdx.x * 8 + warp;
        if (r < R)
#pragma unroll 4
            for (int c = lane; c < K; c += 32) take(J[(size_t)r * ld + c]);
        e = __reduce_max_sync(0xffffffffu, e & ~1u) | __reduce_or_sync(0xffffffffu, e & 1u);
    } else {
        const int c = ((int)blockIdx.x - rowBlocks) * 32 + lane;
        if (c < K)
#pragma unroll 4
            for (int r = warp; r < R; r += 8) take(J[(size_t)r * ld + c]);
        top[warp][lane] = e;
        __syncthreads();
        for (int w = 0; w < 8; ++w) e = max(e & ~1u, top[w][lane] & ~1u) | ((e | top[w][lane]) & 1u);
    }
    const int gap = E == 0x7f800000u ? 255 : (e & 1u) ? (int)((E - (e & ~1u)) >> 23) : 0;
    if (gap > 0) atomicMax(spread, gap);  // (few rows of an ordinary matrix have one)
}

// spins (m x K int8, row stride ldq) -> bf16 (m x ldA), zero beyond K
__global__ void tc_spins_bf16(const int8_t *q, int ldq, int m, int K, int ldA, __nv_bfloat16 *A) {
    pdl_trigger();
    pdl_wait();
    const size_t n = (size_t)m * ldA;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int y = (int)(i / ldA), k = (int)(i - (size_t)y * ldA);
        A[i] = __int2bfloat16_rn(k < K ? (int)q[(size_t)y * ldq + k] : 0);
    }
}

static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

static int ld_pad(int K) { return (K + kTcBK - 1) / kTcBK * kTcBK; }

static int grid_for(size_t n) { return (int)std::min<size_t>((n + 255) / 256, (size_t)152 * 16); }

}  // namespace sq103

using namespace sq103;

// F = spins (converted, in spinsBf16) times the digits' matrix, behind the kernel last launched on the stream
template <class Out>
static int launch_gemm(const void *digits, int R, int K, int m, void *spinsBf16, Out *F, int ldF, int flags,
                       int *status, cudaStream_t st) {
    auto enc = tensor_map_encoder();
    if (!enc) return kErrBadShape;
    const int ldD = ld_pad(K);
    const unsigned char *base = static_cast<const unsigned char *>(digits);
    CUtensorMap tmA, tmB;
    {
        cuuint64_t dims[2] = {(cuuint64_t)ldD, (cuuint64_t)m};
        cuuint64_t strides[1] = {(cuuint64_t)ldD * 2};
        cuuint32_t box[2] = {(cuuint32_t)kTcBK, (cuuint32_t)kTcBM};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&tmA, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, spinsBf16, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return kErrBadShape;
    }
    {
        cuuint64_t dims[3] = {(cuuint64_t)ldD, (cuuint64_t)R, (cuuint64_t)kTcDigits};
        cuuint64_t strides[2] = {(cuuint64_t)ldD * 2, (cuuint64_t)R * ldD * 2};
        cuuint32_t box[3] = {(cuuint32_t)kTcBK, (cuuint32_t)kTcBN, 1};
        cuuint32_t estr[3] = {1, 1, 1};
        if (enc(&tmB, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<unsigned char *>(base + kTcHeader), dims,
                strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return kErrBadShape;
    }
    static SmemLimitOnce limit;  // (one per instance of this function: per output type)
    const cudaError_t limitErr = limit(kTcSmemBytes, tc_digit_gemm<Out>);
    if (limitErr != cudaSuccess) return (int)limitErr;
    // K split over a cluster of up to 4 while the tiles times the split stay within one CTA
    // per SM and a CTA has two K blocks or more.  us per refresh with the spins' conversion,
    // by largest split 1, 2, 4, 8: R = K = 1501, m = 63 (24 tiles) 20.5, 20.5, 18.5, 18.4;
    // 2047 x 3001, m = 200 (64 tiles) 28.9, 24.6, 24.6, 24.6; 1024, m = 64 (16 tiles) 18.6,
    // 18.7, 18.6, 26.8 (a cluster of eight waits for eight free SMs of one GPC)
    const int tilesX = (R + kTcBN - 1) / kTcBN, tilesY = (m + kTcBM - 1) / kTcBM;
    int split = 1;
    while (split < 4 && (long long)tilesX * tilesY * split * 2 <= 152 && ldD / kTcBK >= 4 * split) split *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tilesX, tilesY, split);
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = kTcSmemBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)split;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // behind the spins' conversion
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t le = cudaLaunchKernelEx(&cfg, tc_digit_gemm<Out>, tmA, tmB, reinterpret_cast<const int *>(base + 16), F,
                                              ldF, m, R, ldD, flags, status);
    if (le != cudaSuccess) return (int)le;
    return (int)cudaGetLastError();
}

extern "C" {

SQ103_API unsigned long long sq103_tc_digits_bytes(int R, int K) {
    return (unsigned long long)kTcHeader + (unsigned long long)kTcDigits * R * (unsigned long long)ld_pad(K) * 2ull;
}

SQ103_API unsigned long long sq103_tc_spins_bytes(int m, int K) {
    return (unsigned long long)m * (unsigned long long)ld_pad(K) * 2ull;
}

static int make_digits(const float *J, int ldJ, int R, int K, int transpose, const void *high, void *digits, void *stream) {
    if (R <= 0 || K <= 0 || K >= (1 << 17) || !J || !digits || (reinterpret_cast<uintptr_t>(digits) & 255))
        return kErrBadShape;
    cudaStream_t st = (cudaStream_t)stream;
    unsigned char *base = static_cast<unsigned char *>(digits);
    unsigned *header = reinterpret_cast<unsigned *>(base);
    if (!high) {
        cudaError_t e = cudaMemsetAsync(header, 0, sizeof(sq103_tc_header), st);
        if (e != cudaSuccess) return (int)e;
        const int rowsJ = transpose ? K : R, colsJ = transpose ? R : K;
        tc_max_exponent<<<std::min(rowsJ, 152 * 4), 256, 0, st>>>(J, ldJ, rowsJ, colsJ, header);
    }
    tc_make_digits<<<std::min(R, 152 * 16), 256, 0, st>>>(J, ldJ, R, K, ld_pad(K), transpose, high != nullptr,
                                                          high ? static_cast<const unsigned *>(high) : header, header,
                                                          reinterpret_cast<__nv_bfloat16 *>(base + kTcHeader));
    if (!high && !transpose) {
        const int rowBlocks = (R + 7) / 8;
        tc_spread<<<rowBlocks + (K + 31) / 32, 256, 0, st>>>(J, ldJ, R, K, header, rowBlocks,
                                                            &static_cast<sq103_tc_header *>(digits)->spread);
    }
    return (int)cudaGetLastError();
}

SQ103_API int sq103_tc_make_digits(const float *J, int ldJ, int R, int K, int transpose, void *digits, void *stream) {
    return make_digits(J, ldJ, R, K, transpose, nullptr, digits, stream);
}

int sq103_tc_make_low_digits(const float *J, int ldJ, int R, int K, const void *high, void *digits, cudaStream_t st) {
    if (!high) return kErrBadShape;
    return make_digits(J, ldJ, R, K, 0, high, digits, st);
}

SQ103_API int sq103_tc_refresh(const void *digits, int R, int K, const int8_t *q, int ldq, int m, void *spinsBf16,
                               float *F, int ldF, int flags, int *status, void *stream) {
    return sq103_tc_refresh_after(digits, R, K, q, ldq, m, spinsBf16, F, ldF, flags, status, false,
                                  (cudaStream_t)stream);
}

int sq103_tc_refresh_after(const void *digits, int R, int K, const int8_t *q, int ldq, int m, void *spinsBf16,
                           float *F, int ldF, int flags, int *status, bool dependent, cudaStream_t st) {
    if (R <= 0 || K <= 0 || m <= 0 || K >= (1 << 17) || !digits || !q || !spinsBf16 || !F ||
        (reinterpret_cast<uintptr_t>(digits) & 255) || (reinterpret_cast<uintptr_t>(spinsBf16) & 15) ||
        (flags & ~3))
        return kErrBadShape;
    const int ldD = ld_pad(K);
    launch_dependent(dependent, tc_spins_bf16, dim3(grid_for((size_t)m * ldD)), dim3(256), 0, st, q, ldq, m, K, ldD,
                     reinterpret_cast<__nv_bfloat16 *>(spinsBf16));
    return launch_gemm<float>(digits, R, K, m, spinsBf16, F, ldF, flags, status, st);
}

// r (m x R) = the FP64 row sums of q from the digits and the low digits of one matrix
int sq103_tc_row_sums(const void *digits, const void *lowDigits, int R, int K, const int8_t *q, int ldq, int m,
                      void *spinsBf16, double *r, int *status, cudaStream_t st) {
    if (R <= 0 || K <= 0 || m <= 0 || K >= (1 << 17) || !digits || !lowDigits || !q || !spinsBf16 || !r ||
        (reinterpret_cast<uintptr_t>(digits) & 255) || (reinterpret_cast<uintptr_t>(lowDigits) & 255) ||
        (reinterpret_cast<uintptr_t>(spinsBf16) & 15))
        return kErrBadShape;
    const int ldD = ld_pad(K);
    launch_dependent(false, tc_spins_bf16, dim3(grid_for((size_t)m * ldD)), dim3(256), 0, st, q, ldq, m, K, ldD,
                     reinterpret_cast<__nv_bfloat16 *>(spinsBf16));
    const int rc = launch_gemm<double>(digits, R, K, m, spinsBf16, r, R, 0, status, st);
    return rc != 0 ? rc : launch_gemm<double>(lowDigits, R, K, m, spinsBf16, r, R, kTcAdd, status, st);
}

// The dense refresh every path runs (single annealer, batch, server, bench): the
// tensor-core digit contraction when a digit buffer is given, else the SIMT spin
// GEMM.  Which one a path uses is decided by sq103_dense_refresh_uses_tc(N) and
// digits_coarse() of its digits, so every path that anneals the same instance holds the
// same fields.
SQ103_API int sq103_dense_refresh_uses_tc(int N) { return N >= 1024 ? 1 : 0; }

// Bipartite half-step fields on the tensor cores for problems of at least 2^20
// couplings whose output tiles (128 trotters x 64 spins) give each half step a
// grid of at least 64 CTAs; smaller grids leave most SMs idle, and the SIMT
// field kernel is faster there (N0 = N1 = 1024, m = 64: 16 CTAs).
SQ103_API int sq103_bipartite_refresh_uses_tc(int N0, int N1, int m) {
    if ((long long)N0 * (long long)N1 < (1ll << 20) || m < 1) return 0;
    const long long tiles = (long long)((m + 127) / 128) * ((std::min(N0, N1) + 63) / 64);
    return tiles >= 64 ? 1 : 0;
}

// Where the bipartite annealer takes its energies, and its half-step fields when the
// digits hold every row (kEvenSpread), to the tensor cores: as above, and from
// about 80 M products a half-step on (m rounded up to a SIMT tile's 16 rows).  32 steps in
// ms, SIMT and tensor cores: 1024 x 1024, m = 64 (67 M) 1.10, 1.18, m = 65 (84 M) 1.57,
// 1.20; 1100 x 1900, m = 33 (100 M) 2.17, 1.28; 600 x 9000, m = 1 (86 M) 5.33, 1.38; 2300 x
// 2300, m = 1 (85 M) 2.21, 1.26, m = 16 2.50, 1.55, m = 129 6.72, 2.19.  (Below the line
// larger sides gain too: 2048 x 2048, m = 1 1.97, 1.13.)  The flips' tolerance covers the
// digits' rounding, so decisions are exact and the spins the same on either; a path that
// returns energies (server) sums them the way the annealer does.
int sq103_bipartite_tc_pays(int N0, int N1, int m) {
    if ((long long)N0 * (long long)N1 < (1ll << 20) || m < 1) return 0;
    return sq103_bipartite_refresh_uses_tc(N0, N1, m) || (double)((m + 15) / 16 * 16) * N0 * N1 >= 8e7;
}

SQ103_API int sq103_dense_refresh(const float *J, int ldJ, const void *digits, void *spinsBf16, const int8_t *q,
                                  float *F, int N, int m, int *status, void *stream) {
    if (digits) return sq103_tc_refresh(digits, N, N, q, N, m, spinsBf16, F, N, 0, status, stream);
    return sq103_dense_field_refresh(J, ldJ, q, F, N, m, stream);
}

}  // extern "C"
