// sq_kernels.h -- internal declarations shared by the CUDA translation units.
#pragma once

#include "../../include/sqaod_gb300.h"

#include <cuda_runtime.h>

#include <mutex>

namespace sq103 {

// A kernel's dynamic shared memory limit is an attribute of the device's context that
// every host thread shares: it is set to the largest use, once per device, under a lock,
// and never lowered, so a launch of another thread always finds it large enough.
class SmemLimitOnce {
public:
    template <class... Kernels>
    cudaError_t operator()(int bytes, Kernels... kernels) {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        std::lock_guard<std::mutex> lock(mu_);
        const bool known = dev >= 0 && dev < 256;
        if (known && set_[dev]) return cudaSuccess;
        for (const void *k : {(const void *)kernels...}) {
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (e != cudaSuccess) return e;
        }
        if (known) set_[dev] = true;
        return cudaSuccess;
    }

private:
    std::mutex mu_;
    bool set_[256] = {};
};

}  // namespace sq103

// the half-step fields, launched to start while the stream's last kernel runs when
// `dependent` (that kernel must be one of the bipartite anneal's own)
extern "C" int sq103_bipartite_fields_after(const float *J, int N0, int N1, const int8_t *qFixed, int side, float *F,
                                            int m, bool dependent, cudaStream_t st);
extern "C" int sq103_tc_refresh_after(const void *digits, int R, int K, const int8_t *q, int ldq, int m,
                                      void *spinsBf16, float *F, int ldF, int flags, int *status, bool dependent,
                                      cudaStream_t st);

extern "C" int sq103_bipartite_tc_pays(int N0, int N1, int m);
// the head of a digit buffer (device memory): its matrix is rounded to multiples of 2^-shift
struct sq103_tc_header {
    unsigned maxExp;
    int pad0[3];
    int shift;
    int pad1[3];
    int spread;  // of the matrix (tc_spread; 0 in the digits of a transpose)
};
inline const int *sq103_tc_shift_of(const void *digits) { return &static_cast<const sq103_tc_header *>(digits)->shift; }
namespace sq103 {
constexpr int kEvenSpread = 5;  // up to here the digits are as fine as fp32 for every row
// The digits of an uneven matrix with K columns are too coarse for fields where their
// rounding, up to K 2^-(shift + 1) a field, may exceed half of the drift that the dense
// decisions allow for at any field (2^-16 in h + 2F).
__host__ __device__ inline bool digits_coarse(int shift, int spread, int K) {
    return spread > kEvenSpread && (shift <= 0 || (shift < 40 && ((long long)K << 17) > 1ll << shift));
}
}  // namespace sq103
// sq103_dense_refresh where the host has not seen the header: the tensor-core fields, and
// over them the SIMT ones when the digits are coarse
extern "C" int sq103_dense_refresh_checked(const float *J, int ldJ, const void *digits, void *spinsBf16,
                                           const int8_t *q, float *F, int N, int m, int *status, cudaStream_t st);
// the planes of what `high`, the digits of J (R x K, row stride ldJ), round away (same layout and size)
extern "C" int sq103_tc_make_low_digits(const float *J, int ldJ, int R, int K, const void *high, void *digits,
                                        cudaStream_t st);
extern "C" int sq103_tc_row_sums(const void *digits, const void *lowDigits, int R, int K, const int8_t *q, int ldq,
                                 int m, void *spinsBf16, double *r, int *status, cudaStream_t st);
// the FP64 energies from the row sums r (m x N of q J; m x N1 of q0 J^T)
extern "C" int sq103_dense_energy_of_sums(const double *r, const float *h, const double *c64, const int8_t *q, int N,
                                          int m, int maximize, double *E64, float *E32, cudaStream_t st);
extern "C" int sq103_bipartite_energy_of_sums(const double *r, const float *h0, const float *h1, const double *c64,
                                              const int8_t *q0, const int8_t *q1, int N0, int N1, int m, int maximize,
                                              double *E64, cudaStream_t st);

// sets the message returned by sq103_last_error() on this thread
void sq103_set_error(const char *msg);
