// sq_kernels.h -- internal declarations shared by the CUDA translation units.
#pragma once

#include "../../include/sqaod_gb300.h"

#include <cuda_runtime.h>

// the half-step fields, launched to start while the stream's last kernel runs when
// `dependent` (that kernel must be one of the bipartite anneal's own)
extern "C" int sq103_bipartite_fields_after(const float *J, int N0, int N1, const int8_t *qFixed, int side, float *F,
                                            int m, bool dependent, cudaStream_t st);
extern "C" int sq103_tc_refresh_after(const void *digits, int R, int K, const int8_t *q, int ldq, int m,
                                      void *spinsBf16, float *F, int ldF, int flags, int *status, bool dependent,
                                      cudaStream_t st);

// sets the message returned by sq103_last_error() on this thread
void sq103_set_error(const char *msg);
