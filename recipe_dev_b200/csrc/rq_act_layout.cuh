// The int8 activation records of the matvec kernels: their layout in the scratch and in shared memory. No CUDA in it (a host test reads it).
#pragma once
#include <stddef.h>
#include <stdint.h>

#ifdef __CUDACC__
#define RQ_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define RQ_HOST_DEVICE inline
#endif

// Device-side activation scratch, per token (INT8 path).
// Inputs that are whole 256-value units use one padded record per unit, the layout the streaming
// kernel keeps in shared memory:
//   codes[256] int8 | d[8] fp32 @256 | sum16[16] int16 @288 | sum32[8] int16 @320   (336 bytes)
// Other widths use three planes: codes [cols] int8 | d [cols/32] fp32 | sum16 [cols/16] int16.
// d = the step of a 32-value group, sum16 = the sum of the 16 codes of a slice.
#define RQ_ACT_RECORD_INT8 336
RQ_HOST_DEVICE bool rq_act_unit_layout(int64_t cols) { return cols % 256 == 0; }
RQ_HOST_DEVICE size_t rq_act_token_bytes(int64_t cols) {
    return rq_act_unit_layout(cols) ? (size_t)(cols / 256) * RQ_ACT_RECORD_INT8
                                    : (size_t)cols + (size_t)(cols / 32) * 4 + (size_t)(cols / 16) * 2;
}
