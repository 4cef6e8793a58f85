// Between rq_matmul_tc.cu, which prepares a batched product's operands, and rq_matmul_int8.cu, the kernel of int8 activations over Q8_0 and Q4_0.
#pragma once
#include <cuda.h>
#include <stdint.h>

struct RqInt8Params {
    CUtensorMap tile_map;  // the weight's main plane (TMA descriptor; first: 64-byte aligned)
    const uint16_t* scale;
    int64_t rows;
    int blocks32, units, permuted;
    const uint8_t* xs;     // codes: [token tile][half unit][64 tokens x 128 bytes, swizzled], over Q8_0 in the weight's order of 16-byte chunks
    const float* steps;    // [token tile][half unit][4 groups][64 tokens]
    int tokens;
    float* y; int64_t yn, yt;
    int tiles_m, whole, rest_tiles, share;
    float* partial;        // [2 * share][64][256]
    int* arrived;
    int* error_flag;
    unsigned long long wait_ns;
};
int rq_launch_tc_int8(int type, const RqInt8Params& p, int ctas, cudaStream_t s);
