// Matrix-vector product over the stored formats that have no streaming kernel of their own (Q4_1, Q5_0, Q5_1, Q5_K,
// IQ4_NL, Q8_1, Q2_K, Q3_K, Q8_K, IQ4_XS): fp32 activations against the decoded weights, the reference's run decoders
// (recipe.rs:7826-7917: one fused-multiply-add chain per unit of 32 values; the units of a row add up, ll:3451-3492; here
// the additions are regrouped, within the 1e-3 band). A LANE owns a group of 32 values: it fetches the group's bytes in
// words, turns them into eight words of byte codes whatever the format, and makes them weights with the scale and offset of each
// sixteen, for 32 inputs it holds in registers. `.int(8)` never reaches these formats: the reference re-encodes
// them to Q8_0 at load (rq_weight_requantize), and that weight takes the streaming kernel. `.int(4)` stores Q4_1 and dots it
// with int8 activation records: rq_gemv_q41_int8_kernel below.
#include "rq_decode.cuh"
#include "rq_mma.cuh"
#include "rq_pairs.cuh"
#include "rq_ring_rule.cuh"

namespace {

using rqring::kChunkGroups;
using rqring::kGroupFloats;
using rqring::kWarps;

// N words from a 2-byte aligned address (blocks of 18, 22 and 110 bytes): the aligned words around it, shifted together. Nothing past
// the last wanted byte's word is touched. RING: the bytes lie in shared memory.
template <bool RING, typename T> __device__ __forceinline__ T fetch(const T* p) {
    if constexpr (RING) return *p;
    else return __ldg(p);
}
template <int N, bool RING>
__device__ __forceinline__ void load_words2(const uint8_t* p, uint32_t* w) {
    const uintptr_t a = (uintptr_t)p;
    const uint32_t* q = (const uint32_t*)(a & ~(uintptr_t)3);
    const uint32_t shift = (a & 2) ? 16u : 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = fetch<RING>(q + i);
    const uint32_t last = shift ? fetch<RING>(q + N) : 0u;
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(w[i], i + 1 < N ? w[i + 1] : last, shift);
}
template <int N, bool RING>
__device__ __forceinline__ void load_words4(const uint8_t* p, uint32_t* w) {
#pragma unroll
    for (int i = 0; i < N; ++i) w[i] = fetch<RING>((const uint32_t*)p + i);
}
template <bool RING>
__device__ __forceinline__ void load_line(const uint8_t* p, uint32_t* w) {
    const uint4 v = fetch<RING>((const uint4*)p);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
}

// Four fifth bits (the low four of n) as bytes 0x10 / 0x00: bit i moves to 8 i + 4.
__device__ __forceinline__ uint32_t fifth_bits(uint32_t n) { return ((n & 15u) * 0x02040810u) & 0x10101010u; }
// The IQ4 levels of the eight nibbles of a word, biased by 128: bytes of the low nibbles (values 4 j ..) and of the high ones. The
// sixteen levels (recipe.rs:15211) are four words; a byte permute looks four nibbles up in eight levels at a time.
__device__ __forceinline__ void iq4_levels(uint32_t w, uint32_t& low, uint32_t& high) {
    constexpr uint32_t k0 = 0xBFAD9881u ^ 0x80808080u, k1 = 0xF6EADDCFu ^ 0x80808080u, k2 = 0x26190D01u ^ 0x80808080u, k3 = 0x71594535u ^ 0x80808080u;
    uint32_t v[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // nibbles low0 high0 low1 high1 of half h
        const uint32_t n = h ? w >> 16 : w & 0xffffu;
        const uint32_t below = __byte_perm(k0, k1, n & 0x7777u), above = __byte_perm(k2, k3, n & 0x7777u);
        const uint32_t pick = __byte_perm(0x0000FF00u, 0u, (n >> 3) & 0x1111u);
        v[h] = (above & pick) | (below & ~pick);
    }
    low = __byte_perm(v[0], v[1], 0x6420);
    high = __byte_perm(v[0], v[1], 0x7531);
}

// A group's stored bytes in registers, and what they stand for: value v = scale[v / 16] * (code[v] - bias) + offset[v / 16], codes
// as the bytes of eight words in value order.
template <int TYPE> struct GroupBytes;
template <> struct GroupBytes<RQ_Q4_1> {
    static constexpr int bias = 0;
    uint32_t w[5];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) { load_words4<5, RING>(row + (int64_t)g * 20, w); }
    __device__ __forceinline__ void decode(int, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        scale[0] = scale[1] = rq_h2f((uint16_t)(w[0] & 0xffff));
        offset[0] = offset[1] = rq_h2f((uint16_t)(w[0] >> 16));
#pragma unroll
        for (int j = 0; j < 4; ++j) { c[j] = w[1 + j] & 0x0F0F0F0Fu; c[4 + j] = (w[1 + j] >> 4) & 0x0F0F0F0Fu; }
    }
};
template <> struct GroupBytes<RQ_Q5_0> {
    static constexpr int bias = 16;
    uint32_t w[6];  // d | high bits 0..15, high bits 16..31 | nibbles, ..: the fields straddle words
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)g * 22;
        w[0] = *(const uint16_t*)blk;
        load_words2<5, RING>(blk + 2, w + 1);
    }
    __device__ __forceinline__ void decode(int, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        scale[0] = scale[1] = rq_h2f((uint16_t)w[0]);
        offset[0] = offset[1] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            c[j] = (w[2 + j] & 0x0F0F0F0Fu) | fifth_bits(w[1] >> (4 * j));
            c[4 + j] = ((w[2 + j] >> 4) & 0x0F0F0F0Fu) | fifth_bits(w[1] >> (16 + 4 * j));
        }
    }
};
template <> struct GroupBytes<RQ_Q5_1> {
    static constexpr int bias = 0;
    uint32_t w[6];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) { load_words4<6, RING>(row + (int64_t)g * 24, w); }
    __device__ __forceinline__ void decode(int, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        scale[0] = scale[1] = rq_h2f((uint16_t)(w[0] & 0xffff));
        offset[0] = offset[1] = rq_h2f((uint16_t)(w[0] >> 16));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            c[j] = (w[2 + j] & 0x0F0F0F0Fu) | fifth_bits(w[1] >> (4 * j));
            c[4 + j] = ((w[2 + j] >> 4) & 0x0F0F0F0Fu) | fifth_bits(w[1] >> (16 + 4 * j));
        }
    }
};
template <> struct GroupBytes<RQ_Q5_K> {
    static constexpr int bias = 0;
    uint32_t hdr[4], qh[8], qs[8];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)(g >> 3) * 176;  // eleven lines of sixteen bytes
        load_line<RING>(blk, hdr);
        load_line<RING>(blk + 16, qh);
        load_line<RING>(blk + 32, qh + 4);
        load_line<RING>(blk + 48 + 32 * ((g & 7) >> 1), qs);
        load_line<RING>(blk + 64 + 32 * ((g & 7) >> 1), qs + 4);
    }
    __device__ __forceinline__ void decode(int g, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        const int sub = g & 7;
        int sc, mn;
        rq_q4k_scale_min(hdr[1], hdr[2], hdr[3], sub, sc, mn);
        scale[0] = scale[1] = __fmul_rn(rq_h2f((uint16_t)(hdr[0] & 0xffff)), (float)sc);
        offset[0] = offset[1] = -__fmul_rn(rq_h2f((uint16_t)(hdr[0] >> 16)), (float)mn);
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = ((qs[j] >> (4 * (sub & 1))) & 0x0F0F0F0Fu) | (((qh[j] >> sub) & 0x01010101u) << 4);
    }
};
template <> struct GroupBytes<RQ_IQ4_NL> {
    static constexpr int bias = 128;
    uint32_t d, w[4];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)g * 18;
        d = *(const uint16_t*)blk;
        load_words2<4, RING>(blk + 2, w);
    }
    __device__ __forceinline__ void decode(int, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        scale[0] = scale[1] = rq_h2f((uint16_t)d);
        offset[0] = offset[1] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) iq4_levels(w[j], c[j], c[4 + j]);
    }
};
template <> struct GroupBytes<RQ_IQ4_XS> {
    static constexpr int bias = 128;
    uint32_t hdr[2], w[4];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)(g >> 3) * 136;
        load_words4<2, RING>(blk, hdr);
        load_words4<4, RING>(blk + 8 + 16 * (g & 7), w);
    }
    __device__ __forceinline__ void decode(int g, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        const int b = g & 7, high = (hdr[0] >> (16 + 2 * b)) & 3, low = (hdr[1] >> (4 * b)) & 15;
        scale[0] = scale[1] = __fmul_rn(rq_h2f((uint16_t)(hdr[0] & 0xffff)), (float)((low | (high << 4)) - 32));
        offset[0] = offset[1] = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j) iq4_levels(w[j], c[j], c[4 + j]);
    }
};
template <> struct GroupBytes<RQ_Q8_1> {
    static constexpr int bias = 128;
    uint32_t w[9];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) { load_words4<9, RING>(row + (int64_t)g * 36, w); }
    __device__ __forceinline__ void decode(int, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        scale[0] = scale[1] = rq_h2f((uint16_t)(w[0] & 0xffff));
        offset[0] = offset[1] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = w[1 + j] ^ 0x80808080u;
    }
};
template <> struct GroupBytes<RQ_Q8_K> {
    static constexpr int bias = 128;
    uint32_t d, w[8];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)(g >> 3) * 292;
        d = fetch<RING>((const uint32_t*)blk);
        load_words4<8, RING>(blk + 4 + 32 * (g & 7), w);
    }
    __device__ __forceinline__ void decode(int, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        scale[0] = scale[1] = __uint_as_float(d);
        offset[0] = offset[1] = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = w[j] ^ 0x80808080u;
    }
};
template <> struct GroupBytes<RQ_Q2_K> {
    static constexpr int bias = 0;
    uint32_t meta, dd, w[8];
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)(g >> 3) * 84;
        meta = *(const uint16_t*)(blk + 2 * (g & 7));
        load_words4<8, RING>(blk + 16 + 32 * ((g & 7) >> 2), w);
        dd = fetch<RING>((const uint32_t*)(blk + 80));
    }
    __device__ __forceinline__ void decode(int g, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        const float d = rq_h2f((uint16_t)(dd & 0xffff)), dmin = rq_h2f((uint16_t)(dd >> 16));
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int m = (meta >> (8 * h)) & 0xff;
            scale[h] = __fmul_rn(d, (float)(m & 15));
            offset[h] = -__fmul_rn(dmin, (float)(m >> 4));
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = (w[j] >> (2 * (g & 3))) & 0x03030303u;
    }
};
template <> struct GroupBytes<RQ_Q3_K> {
    static constexpr int bias = 4;  // a clear mask bit takes four off the code
    uint32_t mask[8], w[8], sc[3], d;
    template <bool RING> __device__ __forceinline__ void load(const uint8_t* row, int g) {
        const uint8_t* blk = row + (int64_t)(g >> 3) * 110;
        load_words2<8, RING>(blk, mask);
        load_words2<8, RING>(blk + 32 + 32 * ((g & 7) >> 2), w);
        load_words2<3, RING>(blk + 96, sc);
        d = *(const uint16_t*)(blk + 108);
    }
    __device__ __forceinline__ void decode(int g, uint32_t (&c)[8], float (&scale)[2], float (&offset)[2]) const {
        const int sub = g & 7;
        const float df = rq_h2f((uint16_t)d);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int b = 2 * sub + h, at = b & 7;
            const int low = ((at < 4 ? sc[0] : sc[1]) >> (8 * (at & 3) + (b < 8 ? 0 : 4))) & 15, high = (sc[2] >> (8 * (b & 3) + 2 * (b >> 2))) & 3;
            scale[h] = __fmul_rn(df, (float)((low | (high << 4)) - 32));
            offset[h] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) c[j] = ((w[j] >> (2 * (sub & 3))) & 0x03030303u) | (((mask[j] >> sub) & 0x01010101u) << 2);
    }
};

// A group's weights, each put together whole, against its 32 inputs (v).
template <int TYPE>
__device__ __forceinline__ float dot_group(const GroupBytes<TYPE>& raw, int g, const Pair (&v)[16]) {
    constexpr bool kOffset = TYPE == RQ_Q4_1 || TYPE == RQ_Q5_1 || TYPE == RQ_Q5_K || TYPE == RQ_Q2_K;
    uint32_t c[8];
    float scale[2], offset[2];
    raw.decode(g, c, scale, offset);
    Pair acc[2][2];  // per sixteen: inputs 0, 1 and 2, 3 of every four
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const Pair by = pair_of(scale[j >> 2], scale[j >> 2]), plus = pair_of(offset[j >> 2], offset[j >> 2]);
        // 0x4B0000cc is 2^23 + code: the subtraction leaves the code less its bias, exactly
        constexpr float kOff = -8388608.0f - (float)GroupBytes<TYPE>::bias;
        Pair lo = pair_add(pair_of(__byte_perm(c[j], 0x4B000000u, 0x7650), __byte_perm(c[j], 0x4B000000u, 0x7651)), pair_of(kOff, kOff));
        Pair hi = pair_add(pair_of(__byte_perm(c[j], 0x4B000000u, 0x7652), __byte_perm(c[j], 0x4B000000u, 0x7653)), pair_of(kOff, kOff));
        lo = kOffset ? pair_fma(lo, by, plus) : pair_mul(lo, by);
        hi = kOffset ? pair_fma(hi, by, plus) : pair_mul(hi, by);
        acc[j >> 2][0] = j & 3 ? pair_fma(lo, v[2 * j], acc[j >> 2][0]) : pair_mul(lo, v[2 * j]);
        acc[j >> 2][1] = j & 3 ? pair_fma(hi, v[2 * j + 1], acc[j >> 2][1]) : pair_mul(hi, v[2 * j + 1]);
    }
    const Pair both = pair_add(pair_add(acc[0][0], acc[0][1]), pair_add(acc[1][0], acc[1][1]));
    return pair_at(both, 0) + pair_at(both, 1);
}

// CTAs the registers are cut for: what is in flight per SM counts more than what a warp has in flight by itself, until the formats of many
// words a group begin to spill with four rows. (4096 x 4096, a row a warp, four CTAs: Q4_1 6.8 us, Q5_0 7.5, Q2_K 7.3; left to the
// compiler 8.6, 9.7, 9.8. Q5_K 14336 x 4096, four rows: two CTAs 22.9, three 35.6.)
template <int TYPE, int ROWS>
constexpr int ctas_per_sm() {
    return ROWS == 1 ? 4 : (ROWS == 4 && rqring::many_words(TYPE) ? 2 : 3);
}

// A warp owns ROWS rows, its lanes the groups g, g + 32, ..: a lane reads its group's 32 inputs from shared memory once and uses them
// for all of its rows, whose bytes are all in flight before the first is decoded. A weight is put together whole (scale * code + offset,
// rounded once, as the decoders do) before it meets its input: scaled and offset sums kept apart cost two multiplies less per four weights,
// but cancel against each other (2.3e-7 against 64 bits where decoding value by value has 1.0e-7, Q5_K over 512 inputs), and a code
// times a large input can leave the range that the weight's own product stays in. Per four
// weights: two or three instructions to isolate the codes, four to place them, six packed ones. Measured, Q5_K 14336 x 4096, one token: 26.5 us (28.2 with the sums kept apart; with a ring,
// below, 21.2); decoding value by value, every header field once per value, took 175.6.
template <int TYPE, int ROWS>
__global__ void __launch_bounds__(kWarps * 32, ctas_per_sm<TYPE, ROWS>()) rq_gemv_generic_kernel(const uint8_t* __restrict__ main_plane, int64_t rows, int64_t row_bytes, int groups, const float* x,
                                                                        int64_t sk, int64_t st, float* __restrict__ y, int64_t yn, int64_t yt) {
    extern __shared__ __align__(16) float xs[];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, token = blockIdx.y;
    const float* xt = x + (int64_t)token * st;
    const int64_t row0 = ((int64_t)blockIdx.x * kWarps + warp) * ROWS;
    const uint8_t* base[ROWS];
    float sum[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        base[r] = main_plane + (row0 + r < rows ? row0 + r : rows - 1) * row_bytes;  // rows past the end are computed and dropped
        sum[r] = 0.f;
    }
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int g0 = 0; g0 < groups; g0 += kChunkGroups) {
        const int here = min(kChunkGroups, groups - g0);
        if (g0) __syncthreads();
        for (int k = threadIdx.x; k < here * 32; k += kWarps * 32) xs[(k >> 5) * kGroupFloats + (k & 31)] = __ldcg(xt + ((int64_t)g0 * 32 + k) * sk);
        __syncthreads();
        for (int i = lane; i < here; i += 32) {
            const int g = g0 + i;
            GroupBytes<TYPE> raw[ROWS];
#pragma unroll
            for (int r = 0; r < ROWS; ++r) raw[r].template load<false>(base[r], g);
            Pair v[16];  // the group's inputs
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const ulonglong2 four = *(const ulonglong2*)(xs + i * kGroupFloats + 4 * j);
                v[2 * j] = four.x;
                v[2 * j + 1] = four.y;
            }
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                sum[r] += dot_group<TYPE>(raw[r], g, v);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], off);
        if (lane == 0 && row0 + r < rows) y[(row0 + r) * yn + (int64_t)token * yt] = sum[r];
    }
}

// The same product where a row and 32 of its groups are whole 16-byte lines: a warp owns a range of rows (an equal share, to one row) and
// brings up to four of them at a time, 32 groups of each, into a ring of its own in shared memory with bulk copies, which start before the wait
// for the kernel before (the kernels that write weights let nothing behind them start early: rq_layout.cu, rq_requant.cu). The kernel above
// leaves a warp waiting for memory between its dots (a quarter of the issue slots used): its registers hold one round's bytes, and its CTAs
// come to an SM in whole numbers (448 of them to 148). The same additions in the same order. What bounds it is instruction issue (codes
// turned into fp32 by conversions instead of byte permutes: 22.9). us without / with it: Q5_K 14336 x 4096 26.5 / 21.2, 60000 x 2560 64.4 / 55.4; Q4_1 14336 x 4096
// 19.8 / 16.7; Q8_1 21.5 / 17.4. Which calls take it: rq_ring_rule.cuh.
constexpr int kRingRows = rqring::kRows, kRingMax = rqring::kMaxStages;
template <int TYPE>
__global__ void __launch_bounds__(kWarps * 32, rqring::kCtas) rq_gemv_ring_kernel(const uint8_t* __restrict__ main_plane, int64_t rows, int row_bytes, int chunk_bytes, int stages, int groups, const float* x, int64_t sk,
                                                                    int64_t st, float* __restrict__ y, int64_t yn, int64_t yt, int* error_flag, unsigned long long wait_ns) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t full[kWarps][kRingMax];
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, token = blockIdx.y;
    float* const xs = (float*)smem;
    const int slot_bytes = kRingRows * chunk_bytes;
    uint8_t* const ring = smem + ((groups * kGroupFloats * 4 + 127) & ~127) + warp * stages * slot_bytes;
    const int64_t warps = (int64_t)gridDim.x * kWarps, me = (int64_t)blockIdx.x * kWarps + warp;
    const int64_t row_end = rows * (me + 1) / warps;
    int64_t next_row = rows * me / warps, row = next_row;  // of the copies; of the dots
    const int chunks = (groups + 31) >> 5;
    int next_chunk = 0;
    if (lane == 0) {
        for (int i = 0; i < stages; ++i) rqmma::mbar_init(&full[warp][i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    // the next four rows' next 32 groups into `slot`: a lane a row
    auto issue = [&](int slot) {
        if (next_row >= row_end) return;
        const int n = (int)min((int64_t)kRingRows, row_end - next_row), at = next_chunk * chunk_bytes, bytes = min(chunk_bytes, row_bytes - at);
        if (lane == 0) rqmma::mbar_expect_tx(&full[warp][slot], (uint32_t)(n * bytes));
        __syncwarp();
        if (lane < n) rqmma::bulk_g2s(ring + slot * slot_bytes + lane * chunk_bytes, main_plane + (next_row + lane) * row_bytes + at, (uint32_t)bytes, &full[warp][slot]);
        if (++next_chunk == chunks) { next_chunk = 0; next_row += n; }
    };
    for (int i = 0; i < stages; ++i) issue(i);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float* const xt = x + (int64_t)token * st;
    for (int k = threadIdx.x; k < groups * 32; k += kWarps * 32) xs[(k >> 5) * kGroupFloats + (k & 31)] = __ldcg(xt + (int64_t)k * sk);
    __syncthreads();
    int slot = 0;
    uint32_t phase = 0;
    bool dead = false;
    while (row < row_end) {
        const int n = (int)min((int64_t)kRingRows, row_end - row);
        float sum[kRingRows];
#pragma unroll
        for (int r = 0; r < kRingRows; ++r) sum[r] = 0.f;
        for (int g0 = 0; g0 < groups; g0 += 32) {
            if (!rqmma::mbar_wait_warp(&full[warp][slot], phase, wait_ns, dead)) {
                // The slot is still being written: nothing more goes into a slot or out to y, and the warp leaves once the copies it has under way
                // have landed (within the limit again).
                atomicExch(error_flag, 22);
                const int64_t begin = rows * me / warps;
                const int issued = (int)((next_row - begin + kRingRows - 1) / kRingRows) * chunks + next_chunk, used = (int)((row - begin) / kRingRows) * chunks + g0 / 32;
                for (int in_flight = issued - used; in_flight > 0 && rqmma::mbar_wait(&full[warp][slot], phase, wait_ns); --in_flight)
                    if (++slot == stages) { slot = 0; phase ^= 1; }
                return;
            }
            const uint8_t* const from = ring + slot * slot_bytes;
            if (g0 + lane < groups) {
                Pair v[16];  // the group's inputs
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const ulonglong2 four = *(const ulonglong2*)(xs + (g0 + lane) * kGroupFloats + 4 * j);
                    v[2 * j] = four.x;
                    v[2 * j + 1] = four.y;
                }
#pragma unroll
                for (int r = 0; r < kRingRows; ++r) {
                    if (r < n) {
                        GroupBytes<TYPE> raw;
                        raw.template load<true>(from + r * chunk_bytes, lane);
                        sum[r] += dot_group<TYPE>(raw, lane, v);
                    }
                }
            }
            // the slot's bytes have met their inputs: it may be filled again, once the reads are in order before the copies
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            issue(slot);
            if (++slot == stages) { slot = 0; phase ^= 1; }
        }
#pragma unroll
        for (int r = 0; r < kRingRows; ++r) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) sum[r] += __shfl_xor_sync(0xffffffffu, sum[r], off);
            if (lane == 0 && r < n) y[(row + r) * yn + (int64_t)token * yt] = sum[r];
        }
        row += n;
    }
}

// `.int(4)`: int8 activation records against Q4_1 blocks (block32 slice kind 3, build.rs:777-796). Per 16-value slice
// r = q8_d * (d * f32(dot) + m * f32(sum of the slice's activation codes)); slice 0 takes the low nibbles, slice 1 the high
// ones. A warp owns a row, lane l the blocks l, l + 32, ..; dots by dp4a over the nibbles in place; fixed xor tree.
__global__ void __launch_bounds__(kWarps * 32) rq_gemv_q41_int8_kernel(const uint8_t* __restrict__ blocks, int64_t rows, int64_t cols, const uint8_t* records,
                                                                         size_t token_bytes, float* __restrict__ y, int64_t yn, int64_t yt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, token = blockIdx.y;
    const uint8_t* tok = records + (size_t)token * token_bytes;
    const bool unit = rq_act_unit_layout(cols);
    const int64_t nb = cols >> 5;
    // Programmatic dependent launch: the records (read by plain loads, through a pointer the compiler may not take for one to constants) come from the quantiser launched before this kernel; the weights are
    // constants of the model, so the first round's weight loads go out before the wait for that kernel.
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    bool records_ready = false;
    for (int64_t row = (int64_t)blockIdx.x * kWarps + warp; row < rows; row += (int64_t)gridDim.x * kWarps) {
        float sum = 0.f;
        // four blocks per lane and round, their twenty weight words loaded before the first is used: the row is read once,
        // from HBM, and a round trip per block would leave the warp waiting on latency
        for (int64_t b0 = 0; b0 < nb; b0 += 128) {
            uint32_t wq[4][5];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t b = b0 + 32 * i + lane;
                const uint32_t* blk = (const uint32_t*)(blocks + (row * nb + (b < nb ? b : nb - 1)) * 20);  // 20-byte stride from a 256-byte aligned base: words are aligned
#pragma unroll
                for (int w = 0; w < 5; ++w) wq[i][w] = __ldcs(blk + w);
            }
            if (!records_ready) {
                asm volatile("griddepcontrol.wait;" ::: "memory");
                records_ready = true;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int64_t b = b0 + 32 * i + lane;
                if (b >= nb) break;
                const float d = rq_h2f((uint16_t)(wq[i][0] & 0xffff)), m = rq_h2f((uint16_t)(wq[i][0] >> 16));
                int cl[4], ch[4];
                float q8_d; uint32_t sums;
                if (unit) {
                    const uint8_t* rec = tok + (size_t)(b >> 3) * RQ_ACT_RECORD_INT8;  // records are 16-byte aligned
                    const uint4 lo = *(const uint4*)(rec + 32 * (b & 7)), hi = *((const uint4*)(rec + 32 * (b & 7)) + 1);
                    cl[0] = (int)lo.x; cl[1] = (int)lo.y; cl[2] = (int)lo.z; cl[3] = (int)lo.w;
                    ch[0] = (int)hi.x; ch[1] = (int)hi.y; ch[2] = (int)hi.z; ch[3] = (int)hi.w;
                    q8_d = ((const float*)(rec + 256))[b & 7];
                    sums = ((const uint32_t*)(rec + 288))[b & 7];
                } else {
                    const int* codes = (const int*)(tok + b * 32);  // a token's planes start on a multiple of 8 bytes
#pragma unroll
                    for (int w = 0; w < 4; ++w) { cl[w] = codes[w]; ch[w] = codes[4 + w]; }
                    q8_d = ((const float*)(tok + cols))[b];
                    sums = ((const uint32_t*)(tok + cols + nb * 4))[b];
                }
                int dot_lo = 0, dot_hi = 0;
#pragma unroll
                for (int w = 0; w < 4; ++w) {
                    const uint32_t q = wq[i][1 + w];
                    dot_lo = __dp4a((int)(q & 0x0F0F0F0Fu), cl[w], dot_lo);
                    dot_hi = __dp4a((int)((q >> 4) & 0x0F0F0F0Fu), ch[w], dot_hi);
                }
                const float r0 = __fmul_rn(q8_d, __fadd_rn(__fmul_rn(d, (float)dot_lo), __fmul_rn(m, (float)(int16_t)(sums & 0xffff))));
                const float r1 = __fmul_rn(q8_d, __fadd_rn(__fmul_rn(d, (float)dot_hi), __fmul_rn(m, (float)(int16_t)(sums >> 16))));
                sum += r0;
                sum += r1;
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0) y[row * yn + (int64_t)token * yt] = sum;
    }
}

template <int TYPE, int ROWS>
int launch_generic_rows(const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens, float* y, int64_t yn, int64_t yt, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)((w->rows + kWarps * ROWS - 1) / (kWarps * ROWS)), (unsigned)tokens);
    cfg.blockDim = dim3(kWarps * 32);
    const int groups = (int)(w->cols >> 5);
    cfg.dynamicSmemBytes = (size_t)(groups < kChunkGroups ? groups : kChunkGroups) * kGroupFloats * 4;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const int64_t row_bytes = w->cols / rq_block_values(TYPE) * rq_block_bytes(TYPE);
    RQ_CUDA(cudaLaunchKernelEx(&cfg, rq_gemv_generic_kernel<TYPE, ROWS>, (const uint8_t*)w->main, w->rows, row_bytes, groups, x, sk, st, y, yn, yt));
    return RQ_OK;
}
// RQ_ERR_UNSUPPORTED: the kernel without a ring (rq_ring_rule.cuh says which calls, and why).
template <int TYPE>
int launch_ring(const rq_ctx* ctx, const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens, float* y, int64_t yn, int64_t yt, cudaStream_t s) {
    const int stages = rqring::stages(TYPE, ctx->sm_count, w->rows, w->cols, tokens);
    if (!stages || ((uintptr_t)w->main & 15)) return RQ_ERR_UNSUPPORTED;
    const int groups = (int)(w->cols >> 5);
    const int64_t row_bytes = w->cols / rqring::block_values(TYPE) * rqring::block_bytes(TYPE);
    constexpr int chunk_bytes = rqring::chunk_bytes(TYPE);
    const size_t inputs = rqring::input_bytes(w->cols), slot = (size_t)kWarps * rqring::kRows * chunk_bytes;
    auto kernel = rq_gemv_ring_kernel<TYPE>;
    static bool configured[64] = {};
    if (ctx->device >= 64 || !configured[ctx->device]) {
        RQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rqring::kSmem));
        if (ctx->device < 64) configured[ctx->device] = true;
    }
    cudaLaunchConfig_t cfg = {};
    const int64_t ctas = (w->rows + kWarps - 1) / kWarps, most = (int64_t)ctx->sm_count * rqring::kCtas;
    cfg.gridDim = dim3((unsigned)(ctas < most ? ctas : most), (unsigned)tokens);
    cfg.blockDim = dim3(kWarps * 32);
    cfg.dynamicSmemBytes = inputs + stages * slot;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, (const uint8_t*)w->main, w->rows, (int)row_bytes, chunk_bytes, stages, groups, x, sk, st, y, yn, yt, ctx->error_flag, ctx->wait_limit_ns));
    return RQ_OK;
}
template <int TYPE>
int launch_generic(const rq_ctx* ctx, const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens, float* y, int64_t yn, int64_t yt, cudaStream_t s) {
    if constexpr (rqring::whole_lines(TYPE)) {
        const int rc = launch_ring<TYPE>(ctx, w, x, sk, st, tokens, y, yn, yt, s);
        if (rc != RQ_ERR_UNSUPPORTED) return rc;
    }
    const int sm_count = ctx->sm_count;
    // rows per warp: as many as leave every SM two CTAs (a row's sums do not depend on it)
    const int64_t warps = (int64_t)sm_count * 2 * kWarps / (tokens < 8 ? tokens : 8);
    if (w->rows >= 4 * warps) return launch_generic_rows<TYPE, 4>(w, x, sk, st, tokens, y, yn, yt, s);
    if (w->rows >= 2 * warps) return launch_generic_rows<TYPE, 2>(w, x, sk, st, tokens, y, yn, yt, s);
    return launch_generic_rows<TYPE, 1>(w, x, sk, st, tokens, y, yn, yt, s);
}

}  // namespace

int rq_launch_gemv_generic(rq_ctx* ctx, const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens, float* y, int64_t yn, int64_t yt, cudaStream_t s) {
    if (tokens > 65535) return rq_fail(RQ_ERR_LIMIT, "matvec: %d tokens over a %d-type weight, at most 65535 per call", tokens, w->type);
    switch (w->type) {
#define RQ_CASE(T) case T: return launch_generic<T>(ctx, w, x, sk, st, tokens, y, yn, yt, s);
        RQ_DECODE_ONLY_TYPES(RQ_CASE)
#undef RQ_CASE
        default: return rq_fail(RQ_ERR_INVALID, "matvec: type %d", w->type);
    }
}

int rq_launch_gemv_q41_int8(rq_ctx* ctx, const rq_weight* w, const uint8_t* records, int tokens, float* y, int64_t yn, int64_t yt, cudaStream_t s) {
    if (tokens > 65535) return rq_fail(RQ_ERR_LIMIT, "matvec: %d tokens over a Q4_1 weight, at most 65535 per call", tokens);
    const int64_t ctas = (w->rows + kWarps - 1) / kWarps;
    const int64_t cap = (int64_t)ctx->sm_count * 8;
    dim3 grid((unsigned)(ctas < cap ? ctas : cap), (unsigned)tokens);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(kWarps * 32);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RQ_CUDA(cudaLaunchKernelEx(&cfg, rq_gemv_q41_int8_kernel, (const uint8_t*)w->main, w->rows, w->cols, records, rq_act_token_bytes(w->cols), y, yn, yt));
    return RQ_OK;
}
