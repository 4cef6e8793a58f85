// The streaming matrix-vector kernel over Q4_0 weights.
#include "rq_gemv_stream.cuh"

template <>
int rqstream::dispatch_type<RQ_Q4_0>(StreamParams& p, bool is_float, int sm_count, int vectors_per_launch, cudaStream_t s) {
    return is_float ? dispatch_stream<RQ_Q4_0, RQ_ACT_FLOAT>(p, sm_count, vectors_per_launch, s) : dispatch_stream<RQ_Q4_0, RQ_ACT_INT8>(p, sm_count, vectors_per_launch, s);
}
