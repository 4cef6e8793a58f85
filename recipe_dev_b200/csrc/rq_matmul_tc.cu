// Batched product over the four stored formats on the 5th-generation tensor cores, with EXACT INTEGER weight operands.
//
//   Y[t][n] = sum_k W[n][k] * X[t][k]
//
// A stored value factors into an fp16 scale and small integers:
//   Q4_K : w = d * (sc_g * (q - 8)) - (dmin * m_g - 8 * d * sc_g)   sc_g, m_g six bits, q four bits: |sc_g * (q - 8)| <= 504
//   Q6_K : w = d * (s_j * (q - 32))                                 s_j int8, q six bits: |s_j * (q - 32)| <= 4096
//   Q8_0 : w = d_b * q        Q4_0 : w = d_b * (q - 8)              d_b per 32 values
// fp16 holds every integer up to 2048 exactly, so the tensor core is fed the integers themselves (Q6_K: the fp16 rounding of
// the integer plus its exact residual, -1 / 0 / 1) and the scale is applied outside it, when a sum leaves tensor memory.
// Activations are fp32 and go in as fp16 pairs hi + lo (22 mantissa bits), prepared once per call (rq_tc_prep_kernel) in the
// tensor core's 128-byte-swizzled K-major image; INT8 calls over the K-quants feed code * step through the same path. INT8 calls
// over Q8_0 and Q4_0 (CODES) feed the codes themselves: their scale changes every 32 inputs anyway, as the activations' step does,
// so a sum of 32 products is an exact integer that both scale on its way out -- half the products, half the activation bytes,
// the matvec kernel's arithmetic, and no fp16 range to stay in. Beyond 64 tokens they have a kernel of 8-bit products (rq_matmul_int8.cu), which this file prepares.
//
// One CTA per SM, persistent. Work is counted in UNITS, 256 inputs of one row tile (128 * MH rows) x one token tile: every CTA
// takes the same number of whole tiles and then an equal share of the units that are left, whatever tile they fall in (where few are
// left, only so many CTAs as a tile is worth cutting for: rq_matmul_cut.cuh); a tile that is shared by several CTAs is added up, in unit order, by whichever of them is the last to leave its sums (the same bits on
// every run; a kernel of its own would be one more launch in the chain). Roles in a CTA:
//   * raw copies: one TMA tile of 128 rows x one unit of stored bytes at a time (Q8_0: half a unit) into a ring;
//   * activation copies: one bulk copy per 64-wide slice, B_hi | B_lo of the token tile, into a ring;
//   * staging groups of four warps (thread = row): stored bytes -> 64 fp16 integers -> operand slot in TENSOR MEMORY
//     (tcgen05.st; the A operand of tcgen05.mma may live there, so the unpacked weights never touch shared memory). A group has
//     one slice of every unit (MH = 1, four groups) or one row half (MH = 2, two);
//   * two issuing warps, alternate slices (MH = 2: a row half each): the products of a step into one of a ring of accumulators,
//     one tcgen05.commit. One thread issues a product of 16 .. 32 columns every 33 cycles, of 64 / 96 / 128 every 41 / 56 / 71;
//   * eight drain warps: accumulator -> scale * sum -> fp32 registers, round-to-nearest, then Y or the partial sums.
//
// The tensor core adds into its fp32 accumulator by TRUNCATION, a bias that grows with the length of the chain (measured: 7e-7
// relative over 256 inputs, 1.2e-5 over 4096), so a sum stays in tensor memory for one 64-wide slice (32 inputs for the
// formats whose scale changes there) and the small cross terms go first or into columns of their own.
//
// Two forms. MH = 1 (token tiles of up to 64): B_hi and B_lo are one operand of 2 * bn columns, so a slice is four (Q6_K:
// eight) instructions and the low products have accumulators of their own. MH = 2 (token tiles of up to 128 or, where that leaves few tiles to
// many CTAs, of up to 96: rq_matmul_cut.cuh; of 96 over the 32-value formats, whose two sums a slice take the columns): two row halves share each activation tile, which halves the activation bytes a
// CTA pulls from L2 (they, at 4 bytes per input and token, are what the large shapes would be bound by); products of hi and lo
// share an accumulator, a row half has four drain warps with up to 128 fp32 sums a thread (setmaxnreg).
//
// What bounds it, from cycles counted around every wait: 512 tokens, the tensor cores are busy for half of the time and the rest is
// accumulators being drained (three of 128 columns are what tensor memory holds); a few tokens, a third is the wait for the
// activation image, the rest the chain staging -> products -> drain of a slice. Measured on one B200, calls back to back,
// before (staging groups took slices in turn; a lone lane looked at barriers; columns were tested for in sixteens; tiles of 96;
// the minimum terms read their headers again) and
// now: Q4_K 14336 x 4096 16 / 64 / 90 / 512 tokens 34.2 / 49.4 / 55.6 / 188 us -> 27.7 / 41.2 / 45.9 / 118 (a burst; 199 -> 139 under load, where clocks fall); Q6_K 4096 x 14336 int8 64
// tokens 50.8 -> 44.3; Q8_0 14336 x 4096 int8 20 tokens 49.0 -> 35.4, 4096 x 8192 fp32 200 tokens 84.3 -> 61.2. The shared tiles' sums as the last thing a CTA does, by drain and staging warps together, were slower (64 tokens 48.8): a CTA is
// then the last of both of its tiles more often.
//
// The Q4_K minimum term, sum_g (8 * d * sc_g - dmin * m_g) * (sum of x over group g), is a second, 32 times smaller product: per
// window of four superblocks one more slice (the terms' fp16 values and, behind them, their residuals) whose "activations" are the group
// sums, twice.
//
// Every wait is bounded; a wait that runs out records a code in the context's error word and the thread stops waiting. Before the CTA frees its
// tensor memory and exits, the issuing and copying warps wait once more, within the same limit, for the products and copies that they have under way.
#include "rq_internal.cuh"
#include "rq_matmul_cut.cuh"
#include "rq_matmul_int8.cuh"
#include "rq_mma.cuh"
#include "rq_pairs.cuh"

using namespace rqmma;
using namespace rqcut;

namespace {

constexpr int kDone = 32;                    // ring of "step finished" barriers, indexed by the step (see the kernel)
constexpr float kMinScale = 256.0f, kMinUnscale = 1.0f / 256.0f;  // the minimum term's weights are scaled so that their fp16 residuals are no subnormals

constexpr int kIssuers = 2;                  // with the two copying warps: one warpgroup
template <int MH, bool CODES> __host__ __device__ constexpr int tc_threads() { return (Shape<MH, CODES>::drain_warps + 4 * Shape<MH, CODES>::groups + 4) * 32; }

struct TcParams {
    CUtensorMap tile_map;  // the weight's main plane as a [rows][row bytes] byte matrix (TMA descriptor; first: 64-byte aligned)
    const uint8_t* main;
    const uint16_t* scale;
    int64_t rows;
    int blocks32;          // 32-value blocks per row
    int units;             // 256-value units per row (a last one may be partial for the 32-value formats)
    int permuted;          // Q8_0 / Q4_0: the plane's chunks are permuted (rows of whole units)
    const uint8_t* xs;     // activation images: [token tile][image tile][hi | lo][bn rows x 128 bytes, swizzled] (CODES: one fp16 tile of codes)
    const float* steps;    // CODES: [token tile][slice][half][bn]
    int image_tiles;       // 4 * units, then one per window of four superblocks (Q4_K)
    int bn, tokens;
    float* y; int64_t yn, yt;
    int tiles_m, whole, rest_tiles, share;  // row tiles; whole tiles per CTA; tiles shared out by units, and among how many CTAs
    float* partial;        // [2 * share][bn][128 * MH]
    int* arrived;          // per shared tile, how many of its CTAs have left their sums (zeroed by the preparation kernel)
    int raw_slots, b_slots, a_slots, accs;
    int* error_flag;
    unsigned long long wait_ns;
};

__device__ __forceinline__ __half2 as_half2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
// fp32 pair -> fp16 hi and lo words
__device__ __forceinline__ void split2(float a, float b, uint32_t& hi, uint32_t& lo) {
    const __half2 h2 = __floats2half2_rn(a, b);
    const float2 back = __half22float2(h2);
    hi = as_u32(h2);
    lo = as_u32(__floats2half2_rn(a - back.x, b - back.y));
}
// a TMA tile of 128-byte rows written with the 128-byte swizzle
__device__ __forceinline__ uint4 swizzled_chunk(const uint8_t* tile, int row, int chunk) { return *(const uint4*)(tile + swizzled(row, chunk)); }

// ------------------------------------------------------------------------------------------
// 64 inputs of one row (slice `sl` of unit `u`): the stored bytes, and 32 of them at a time (`half`) as fp16 integers (sixteen words),
// inputs in the order 0 2 1 3 within every four: the order the nibbles of a word come out in. 0x6400 | n is the fp16 number
// 1024 + n; the subtraction that follows and the product with a scale are exact. The loads come before the arithmetic: a store to
// tensor memory between them would hold the second half's loads back.
// ------------------------------------------------------------------------------------------
template <int TYPE> struct Stored {
    uint4 v[TYPE == RQ_Q6_K || TYPE == RQ_Q8_0 ? 4 : (TYPE == RQ_Q4_K ? 3 : 2)];
    uint32_t scales;
    __device__ __forceinline__ void load(const uint8_t* tile, int r, int u, int sl, bool permuted) {
        if (TYPE == RQ_Q4_K) {
            const uint8_t* blk = tile + r * 144;
            v[0] = *(const uint4*)blk;
            v[1] = *(const uint4*)(blk + 16 + 32 * sl);
            v[2] = *(const uint4*)(blk + 32 + 32 * sl);
        } else if (TYPE == RQ_Q6_K) {
            const int ch = sl >> 1, sel = sl & 1;
            const uint8_t* body = tile + r * 208;
#pragma unroll
            for (int i = 0; i < 2; ++i) { v[i] = *(const uint4*)(body + 64 * ch + 16 * i); v[2 + i] = *(const uint4*)(body + 128 + 32 * ch + 16 * i); }
            scales = *(const uint32_t*)(body + 192 + 8 * ch + 4 * sel);  // int8 scales of the inputs 0..15, 16..31, 32..47, 48..63
        } else if (TYPE == RQ_Q8_0) {
            const int x = permuted ? u & 7 : 0;
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = swizzled_chunk(tile, r, (4 * (sl & 1) + i) ^ x);  // the tile holds half a unit: chunks 0..7
        } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) v[i] = swizzled_chunk(tile, r, (2 * sl + i) ^ (permuted ? u & 7 : 0));  // a block: low nibbles are its first sixteen values
        }
    }
    // Q6_K: the second half's low bits, once the first half's are spent (the operands and their residuals take the registers)
    __device__ __forceinline__ void load_second(const uint8_t* tile, int r, int sl) {
        if (TYPE == RQ_Q6_K) {
#pragma unroll
            for (int i = 0; i < 2; ++i) v[i] = *(const uint4*)(tile + r * 208 + 64 * (sl >> 1) + 32 + 16 * i);
        }
    }
    __device__ __forceinline__ void expand(int sl, int half, uint32_t (&o)[16], uint32_t (&res)[16]) const {
        if (TYPE == RQ_Q4_K) {
            const uint4& hdr = v[0];
            // the six-bit scale of sub-block 2 sl + half, without a branch: bytes 0 .. 3 of the first four, split ones after
            const int at = 8 * ((2 * sl + half) & 3);
            const uint32_t packed = sl < 2 ? hdr.y & 0x3f3f3f3fu : (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u);
            const int sc = (packed >> at) & 0xff;
            // a nibble in bits 4 .. 7 under an exponent of 0x6400 is 1024 + 16 q: times sc / 16, less 72 sc, is sc * (q - 8) -- sc / 16, 72 sc
            // (a multiple of eight below 4608) and the result (at most 504) are fp16 numbers, so the fused operation is exact
            const __half2 mul = __half2half2(__hmul(__int2half_rn(sc), __float2half_rn(0.0625f))), off = __half2half2(__int2half_rn(-72 * sc));
            const uint32_t w[8] = {v[1].x, v[1].y, v[1].z, v[1].w, v[2].x, v[2].y, v[2].z, v[2].w};
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t a = ((half ? w[j] : w[j] << 4) & 0x00F000F0u) | 0x64006400u;       // inputs 4j, 4j + 2
                const uint32_t b = ((half ? w[j] >> 8 : w[j] >> 4) & 0x00F000F0u) | 0x64006400u;  // inputs 4j + 1, 4j + 3
                o[2 * j] = as_u32(__hfma2(as_half2(a), mul, off));
                o[2 * j + 1] = as_u32(__hfma2(as_half2(b), mul, off));
            }
        } else if (TYPE == RQ_Q6_K) {
            const int sel = sl & 1, g = 2 * sel + half;
            const uint32_t lw[8] = {v[0].x, v[0].y, v[0].z, v[0].w, v[1].x, v[1].y, v[1].z, v[1].w}, hw[8] = {v[2].x, v[2].y, v[2].z, v[2].w, v[3].x, v[3].y, v[3].z, v[3].w};
            const __half2 s_first = __half2half2(__int2half_rn((int)(int8_t)(scales >> (16 * half))));
            const __half2 s_second = __half2half2(__int2half_rn((int)(int8_t)(scales >> (16 * half + 8))));
            const __half2 k1056 = __half2half2(__float2half_rn(1056.0f));
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const __half2 s2 = j < 4 ? s_first : s_second;
                const uint32_t q4 = ((lw[j] >> (4 * sel)) & 0x0F0F0F0Fu) | (((hw[j] >> (2 * g)) & 0x03030303u) << 4);  // four six-bit codes
                const uint32_t a = __byte_perm(q4, 0x64646464u, 0x4240), b = __byte_perm(q4, 0x64646464u, 0x4341);  // bytes 0, 2 and 1, 3 under 0x64
                const __half2 ca = __hsub2(as_half2(a), k1056), cb = __hsub2(as_half2(b), k1056);  // q - 32
                const __half2 ha = __hmul2(ca, s2), hb = __hmul2(cb, s2);
                o[2 * j] = as_u32(ha);
                o[2 * j + 1] = as_u32(hb);
                res[2 * j] = as_u32(__hfma2(ca, s2, __hneg2(ha)));  // the product less its rounding: -1, 0 or 1
                res[2 * j + 1] = as_u32(__hfma2(cb, s2, __hneg2(hb)));
            }
        } else if (TYPE == RQ_Q8_0) {
            const uint4 &q0 = v[2 * half], &q1 = v[2 * half + 1];
            const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
            const __half2 k1152 = __half2half2(__float2half_rn(1152.0f));
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const uint32_t c = w[j] ^ 0x80808080u;  // code + 128
                o[2 * j] = as_u32(__hsub2(as_half2(__byte_perm(c, 0x64646464u, 0x4240)), k1152));  // bytes 0, 2 under 0x64; then 1, 3
                o[2 * j + 1] = as_u32(__hsub2(as_half2(__byte_perm(c, 0x64646464u, 0x4341)), k1152));
            }
        } else {
            const uint4& q = v[half];
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
            const __half2 k1032 = __half2half2(__float2half_rn(1032.0f));
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                o[2 * j] = as_u32(__hsub2(as_half2((w[j] & 0x000F000Fu) | 0x64006400u), k1032));
                o[2 * j + 1] = as_u32(__hsub2(as_half2(((w[j] >> 8) & 0x000F000Fu) | 0x64006400u), k1032));
                o[8 + 2 * j] = as_u32(__hsub2(as_half2(((w[j] >> 4) & 0x000F000Fu) | 0x64006400u), k1032));
                o[8 + 2 * j + 1] = as_u32(__hsub2(as_half2(((w[j] >> 12) & 0x000F000Fu) | 0x64006400u), k1032));
            }
        }
    }
};

// Q4_K: 2^8 * (dmin * m_g - 8 * d * sc_g) of a superblock's eight sub-blocks (what is left of the minimum once the codes are
// centred: for weights spread about zero an order of magnitude smaller than dmin * m_g, and so are the truncations of its sums)
// as fp16, and the residuals of that rounding.
__device__ __forceinline__ void minimum_terms(const uint4& hdr, uint32_t (&hi)[4], uint32_t (&lo)[4]) {
    // both products are exact in fp32 (an fp16 times an integer below 64); their difference is rounded once
    const float dmin = __fmul_rn(kMinScale, rq_h2f((uint16_t)(hdr.x >> 16))), d8 = __fmul_rn(-8.0f * kMinScale, rq_h2f((uint16_t)(hdr.x & 0xffff)));
    const uint32_t sc[2] = {hdr.y & 0x3f3f3f3fu, (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u)};
    const uint32_t mn[2] = {hdr.z & 0x3f3f3f3fu, ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float t[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int at = 16 * (j & 1) + 8 * i;
            t[i] = __fmaf_rn(dmin, (float)((mn[j >> 1] >> at) & 0xff), __fmul_rn(d8, (float)((sc[j >> 1] >> at) & 0xff)));
        }
        split2(t[0], t[1], hi[j], lo[j]);
    }
}

// ------------------------------------------------------------------------------------------
// X -> the tensor core's operand images. A warp takes one unit of one token row: lane l the eight inputs 8 l .. 8 l + 7, so reads
// and writes are whole lines. INT8 quantises on the way with the reference's arithmetic: the extreme of a group of STEP inputs
// is the FIRST input of strictly largest magnitude, signed; inverse = -127 / extreme and d = 1 / inverse are IEEE divides,
// code = clamp(rint(x * inverse)); the image holds code * d. STEP 0: fp32 activations. CODES: the image holds the codes, and the
// matvec kernels' records of the same inputs are left beside it for INT8_CACHED calls; STEP -1 reads those records instead of x. Rows
// past the last token and inputs past the last column are zeros.
// ------------------------------------------------------------------------------------------
enum Image { kPairs, kCodes, kBytes };  // fp16 hi | lo; the codes as fp16; the codes as bytes (rq_matmul_int8.cu), half a unit a tile
template <int STEP, Image IMAGE>
__global__ void __launch_bounds__(256) rq_tc_prep_kernel(const float* x, int64_t sk, int64_t st, int cols, int units, int tokens, int padded, int bn, int image_tiles,
                                                          int windows, int permuted, uint8_t* records, uint8_t* xs, float* steps,
                                                          int* arrived, int shared_tiles) {
    constexpr bool CODES = IMAGE != kPairs;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, unit = blockIdx.x;
    const int row = (blockIdx.z * gridDim.y + blockIdx.y) * 8 + (threadIdx.x >> 5);  // the padded rows are a multiple of sixteen
    if (row >= padded) return;  // a last layer of the grid that is not full (more rows than one layer takes)
    const int nt = row / bn, r = row - nt * bn, k0 = unit * 256 + 8 * lane;
    const bool vec = sk == 1 && (st & 3) == 0 && ((uintptr_t)x & 15) == 0;
    // eight inputs: a 16-byte chunk of the image, or half of one (chunks in the order that the weight's plane has them in)
    uint8_t* hi = IMAGE == kBytes ? xs + ((size_t)nt * image_tiles + 2 * unit + (lane >> 4)) * (size_t)bn * 128 + swizzled(r, ((lane >> 1) ^ (permuted ? unit : 0)) & 7) + 8 * (lane & 1)
                                  : xs + ((size_t)nt * image_tiles + 4 * unit + (lane >> 3)) * (CODES ? 1 : 2) * (size_t)bn * 128 + swizzled(r, lane & 7);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (blockIdx.x == 0 && row < 8)
        for (int i = threadIdx.x; i < shared_tiles; i += 256) arrived[i] = 0;
    float v[8], d = 0.f;
    uint32_t packed[2] = {0, 0};
    // CODES: where this lane's eight codes, their group's step and the sums lie in the token's records
    const bool inside = row < tokens && k0 < cols;
    uint8_t *rec_codes = nullptr, *rec_step = nullptr, *rec_sum16 = nullptr;
    if (CODES && inside) {
        uint8_t* tok = records + (size_t)row * rq_act_token_bytes(cols);
        if (rq_act_unit_layout(cols)) {
            uint8_t* rec = tok + (size_t)unit * RQ_ACT_RECORD_INT8;
            rec_codes = rec + 8 * lane; rec_step = rec + 256 + 4 * (lane >> 2); rec_sum16 = rec + 288 + 2 * (lane >> 1);
        } else {
            rec_codes = tok + k0; rec_step = tok + cols + 4 * (k0 >> 5); rec_sum16 = tok + cols + 4 * (cols >> 5) + 2 * (k0 >> 4);
        }
    }
    if (STEP < 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.f;
        if (inside) {
            const uint2 c = __ldcg((const uint2*)rec_codes);
            packed[0] = c.x;
            packed[1] = c.y;
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = (float)(int8_t)((j < 4 ? c.x : c.y) >> (8 * (j & 3)));
            d = __ldcg((const float*)rec_step);
        }
    } else if (inside) {  // a width is a whole number of 32-value blocks: a lane's eight inputs are all inside or all outside
        const float* src = x + (int64_t)row * st + (int64_t)k0 * sk;
        if (vec) {
            *(float4*)v = __ldcg((const float4*)src);
            *(float4*)(v + 4) = __ldcg((const float4*)src + 1);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __ldcg(src + j * sk);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
    if (STEP > 0) {
        float best = 0.f;  // a NaN is never larger, so it never becomes the extreme
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (fabsf(v[j]) > fabsf(best)) best = v[j];
#pragma unroll
        for (int off = 1; off <= STEP / 16; off <<= 1) {  // 4 lanes or 32 hold a group
            const float other = __shfl_xor_sync(0xffffffffu, best, off);
            // of two equal magnitudes the earlier input's wins
            if ((lane & off) ? fabsf(other) >= fabsf(best) : fabsf(other) > fabsf(best)) best = other;
        }
        const bool nonzero = fabsf(best) > 0.f;
        const float inverse = nonzero ? __fdiv_rn(-127.0f, best) : 0.f;
        d = nonzero ? __fdiv_rn(1.0f, inverse) : 0.f;
        int sum = 0;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int code = __float2int_rn(__fmul_rn(v[j], inverse));
            code = code < -128 ? -128 : (code > 127 ? 127 : code);
            v[j] = CODES ? (float)code : __fmul_rn((float)code, d);
            sum += code;
            packed[j >> 2] |= (uint32_t)(code & 0xff) << (8 * (j & 3));
        }
        if (CODES) {
            const int sum16 = sum + __shfl_xor_sync(0xffffffffu, sum, 1), sum32 = sum16 + __shfl_xor_sync(0xffffffffu, sum16, 2);
            if (inside) {
                *(uint2*)rec_codes = make_uint2(packed[0], packed[1]);
                if ((lane & 1) == 0) *(int16_t*)rec_sum16 = (int16_t)sum16;
                if ((lane & 3) == 0) {
                    *(float*)rec_step = d;
                    if (rq_act_unit_layout(cols)) *(int16_t*)(rec_codes - 8 * lane + 320 + 2 * (lane >> 2)) = (int16_t)sum32;
                }
            }
        }
    }
    if (CODES) {
        if ((lane & 3) == 0) steps[(((size_t)nt * units + unit) * 8 + (lane >> 2)) * bn + r] = d;
    }
    if (IMAGE == kBytes) {
        *(uint2*)hi = make_uint2(packed[0], packed[1]);
        return;
    }
    uint32_t hw[4], lw[4];
    split2(v[0], v[2], hw[0], lw[0]);  // the order the weights' nibble pairs come in
    split2(v[1], v[3], hw[1], lw[1]);
    split2(v[4], v[6], hw[2], lw[2]);
    split2(v[5], v[7], hw[3], lw[3]);
    *(uint4*)hi = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    if (!CODES) *(uint4*)(hi + (size_t)bn * 128) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
    if (windows) {
        // the unit's eight group sums: one 16-byte chunk of the window's image tile
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[j];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        const float next = __shfl_down_sync(0xffffffffu, s, 4);
        uint32_t h, l;
        split2(s, next, h, l);  // in lanes 0, 8, 16, 24: groups 0 1 | 2 3 | 4 5 | 6 7
        // (twice: the window's operand is the terms' fp16 values and, behind them, their residuals)
        uint8_t* sums = xs + ((size_t)nt * image_tiles + 4 * units + (unit >> 2)) * 2 * (size_t)bn * 128;
        if ((lane & 7) == 0) {
#pragma unroll
            for (int again = 0; again < 8; again += 4) {
                const int at = swizzled(r, again + (unit & 3)) + 4 * (lane >> 3);
                *(uint32_t*)(sums + at) = h;
                *(uint32_t*)(sums + (size_t)bn * 128 + at) = l;
            }
        }
        if (unit == units - 1) {  // groups past the last superblock of the window count as zeros
            const int chunk = lane & 7;
            if ((chunk & 3) > (unit & 3) && lane < 16) *(uint4*)(sums + (lane < 8 ? 0 : (size_t)bn * 128) + swizzled(r, chunk)) = make_uint4(0, 0, 0, 0);
        }
    }
}

// sixteen columns at two places of this warp's 32 lanes; thirty-two at one
__device__ __forceinline__ void tmem_ld16_pair(uint32_t a, uint32_t b, uint32_t (&u)[16], uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%33];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=&r"(u[0]), "=&r"(u[1]), "=&r"(u[2]), "=&r"(u[3]), "=&r"(u[4]), "=&r"(u[5]), "=&r"(u[6]), "=&r"(u[7]), "=&r"(u[8]), "=&r"(u[9]), "=&r"(u[10]), "=&r"(u[11]),
          "=&r"(u[12]), "=&r"(u[13]), "=&r"(u[14]), "=&r"(u[15]), "=&r"(v[0]), "=&r"(v[1]), "=&r"(v[2]), "=&r"(v[3]), "=&r"(v[4]), "=&r"(v[5]), "=&r"(v[6]), "=&r"(v[7]),
          "=&r"(v[8]), "=&r"(v[9]), "=&r"(v[10]), "=&r"(v[11]), "=&r"(v[12]), "=&r"(v[13]), "=&r"(v[14]), "=&r"(v[15])
        : "r"(a), "r"(b)
        : "memory");
}

template <int N> struct Columns { static constexpr int value = N; };
template <Image I> struct ImageOf { static constexpr Image value = I; };

template <int TYPE, int MH, bool CODES>
__global__ void __launch_bounds__(tc_threads<MH, CODES>(), 1) rq_tc_kernel(const __grid_constant__ TcParams p) {
    using F = Format<TYPE>;
    using S = Shape<MH, CODES>;
    using Order = Slices<TYPE>;
    constexpr int kDrainWarps = S::drain_warps, kGroups = S::groups, kStageFirst = kDrainWarps, kMiscFirst = kDrainWarps + 4 * kGroups;
    static_assert(32 * kDrainWarps * S::drain_regs + 128 * kGroups * S::stage_regs + 128 * S::other_regs <= tc_threads<MH, CODES>() * S::launch_regs, "more registers than the launch has: the increase would wait forever");
    static_assert(kDrainWarps == 8 && kGroups == (MH == 1 ? 4 : 2), "a staging group has one slice of every unit (MH = 1) or one row half (MH = 2)");
    constexpr int kHalves = F::halves;
    static_assert(MH == 1 || !CODES, "codes and two row halves: rq_matmul_int8.cu");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // swizzled tiles want 1024-byte alignment
    // A STEP is one operand tile's products: (slice, row half), numbered in issue order. A step's commit
    // arrives on done[step % kDone]: the drain warps wait for it (the sums are complete), the staging warps for the step that read
    // their operand slot, the activation copies for the last step that read theirs. What the drain warps have read they say on
    // drained[step % kDone], and a staged tile (slice, row half) is announced on a_full[tile % kDone].
    // Indexing by step keeps every parity wait within one phase whatever the rings' lengths: no thread is ever kDone steps ahead
    // of anyone (activation slots x steps per slot < kDone).
    __shared__ __align__(8) uint64_t done[kDone], drained[kDone], a_full[kDone], raw_full[kMaxRaw], raw_empty[kMaxRaw], b_full[kMaxB];
    __shared__ __align__(8) uint64_t ended[kIssuers];  // an issuing warp's products are all complete
    __shared__ uint32_t tmem_base_slot;
    __shared__ int last_piece;
    // CODES: the activations' steps of a few slices, a ring of its own (the drain warps read it, well after the products are done)
    constexpr int kStepSlots = CODES ? 8 : 1;
    __shared__ __align__(16) float step_ring[kStepSlots][2][S::cols];
    __shared__ __align__(8) uint64_t steps_full[kStepSlots], steps_empty[kStepSlots];
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // visibly the same for the whole warp: the compiler budgets registers by role only then
    const int bn = p.bn, b_bytes = bn * (CODES ? 128 : 256), a_mask = p.a_slots - 1, sums = p.accs / kHalves;  // sums: steps that have accumulators of their own
    const int acc_cols = MH == 1 && !CODES ? 2 * bn : bn;
    uint8_t* raw = smem + (size_t)p.b_slots * b_bytes;
    // Q4_K: the headers of a window's four superblocks, each left by the thread that will turn them into the window's minimum terms (read
    // again from global memory when those are due they cost a trip to memory in the middle of the chain).
    uint4* const stash = (uint4*)(raw + (size_t)p.raw_slots * F::raw_bytes + (MH == 1 ? (size_t)bn * 512 : 0));

    if (tid == 0) {
        for (int s = 0; s < kDone; ++s) { mbar_init(&done[s], 1); mbar_init(&drained[s], 4); mbar_init(&a_full[s], 4); }
        for (int s = 0; s < kMaxRaw; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], MH == 1 ? 4 * F::raw_slices : 4); }
        for (int s = 0; s < kMaxB; ++s) mbar_init(&b_full[s], 1);
        for (int s = 0; s < kIssuers; ++s) mbar_init(&ended[s], 1);
        for (int s = 0; s < kStepSlots; ++s) { mbar_init(&steps_full[s], 1); mbar_init(&steps_empty[s], 4); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kMiscFirst) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = tmem_base_slot, a_ring = tmem_base + 512u - (uint32_t)(p.a_slots * F::a_cols);
    Walk walk(p.whole, p.rest_tiles, p.units, p.share, (int)gridDim.x, (int)blockIdx.x);
    int tile, u0, u1;

    if (warp < kDrainWarps) {
        // ------------------------------------------------------------ drain warps
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(S::drain_regs));
        // Warp w may read accumulator rows 32 (w % 4) .., so four warps, a SET, drain a sum's columns. MH = 1: the even and the odd slices, joined at
        // the end of the tile; MH = 2: a row half each.
        const int quarter = warp & 3, set = warp >> 2, half0 = MH == 2 ? set : 0;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        float* const joined = (float*)(raw + (size_t)p.raw_slots * F::raw_bytes);  // MH = 1: [bn][128]
        int slice_base = 0;  // slices of the segments before this one
        Ring acc_at(sums, set);  // the accumulators of this set's next slice
        bool dead = false;
        // The number of columns is known where the loops are unrolled: with a test for each sixteen of them the sums went through copies, and a
        // drain of 128 columns took 1340 cycles instead of 550 (512 tokens: 135 us).
        auto run_tiles = [&](auto columns) {
            constexpr int kMine = decltype(columns)::value;
            while (walk.next(tile, u0, u1)) {
                const int mt = tile % p.tiles_m, nt = tile / p.tiles_m;
                // the CTAs that share this tile, in unit order (some divisions: before the sums are there, not behind them)
                const bool whole = u0 == 0 && u1 == p.units;
                const int t = tile - p.whole * (int)gridDim.x;
                int c0 = 0, c1 = 0;
                if (!whole) {
                    const Deal deal(p.share, p.rest_tiles, p.units);
                    c0 = deal.first(t);
                    c1 = deal.last(t, (int)blockIdx.x);
                }
                Pair sum[kMine / 2];
#pragma unroll
                for (int i = 0; i < kMine / 2; ++i) sum[i] = 0;
                // CODES: the products are exact, so what a sum loses it loses where its terms (32 inputs each) are added up, and up to 448 of them one
                // after another in one fp32 register lose more than the matvec kernel's tree does. Every few slices the sums go into totals,
                // and what that addition rounds off stays in the register as the start of the next run (the shorter the segment, the more the
                // additions inside a run weigh). Error against 64 bits, 4096 x 14336 and 509 tokens: 2.0e-7 without, 0.75e-7 so, the matvec
                // kernel 0.90e-7. The totals lie in tensor memory. (In registers they
                // spill; a compensated sum at every slice is slower.)
                const int own = 2 * (u1 - u0);  // (a set's slices of this segment)
                const int run_length = own <= 16 ? 2 : (own <= 64 ? 4 : 8);
                int run = 0;
                bool flushed = false;
                [[maybe_unused]] const uint32_t totals = tmem_base + lane_base + (uint32_t)(p.accs * acc_cols + set * bn);
                const Pair minus = pair_of(-1.0f, -1.0f);
                auto flush = [&]() {
                    run = 0;
                    Pair lost = 0;
                    auto into = [&](Pair total, Pair& s) -> Pair {  // total + s; s = what that rounds off
                        const Pair t = pair_add(total, s);
                        s = pair_fma(minus, pair_fma(minus, total, t), s);
                        lost = pair_add(lost, s);
                        return t;
                    };
#pragma unroll
                    for (int c = 0; c < kMine; c += 16) {
                        uint32_t v[16];
                        if (flushed) {
                            tmem_ld16(totals + c, v);
#pragma unroll
                            for (int j = 0; j < 16; j += 2) {
                                const Pair t = into(pair_of(v[j], v[j + 1]), sum[(c + j) / 2]);
                                v[j] = __float_as_uint(pair_at(t, 0));
                                v[j + 1] = __float_as_uint(pair_at(t, 1));
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(pair_at(sum[(c + j) / 2], j & 1));
#pragma unroll
                            for (int j = 0; j < 8; ++j) sum[c / 2 + j] = 0;
                        }
                        tmem_st16(totals + c, v);
                    }
                    tmem_st_wait();
                    flushed = true;
                    // an infinite total has no rounding error to carry on
                    if (!(fabsf(pair_at(lost, 0) + pair_at(lost, 1)) <= 3.402823466e38f)) {
#pragma unroll
                        for (int i = 0; i < kMine / 2; ++i) {
                            const float e0 = pair_at(sum[i], 0), e1 = pair_at(sum[i], 1);
                            sum[i] = pair_of(fabsf(e0) <= 3.402823466e38f ? e0 : 0.f, fabsf(e1) <= 3.402823466e38f ? e1 : 0.f);
                        }
                    }
                };
                // this lane's row, kept inside the weight for the scale loads (found anew by each: held, it cost Q8_0 and Q4_0 4 % in spilled registers)
                auto my_row = [&]() -> int64_t { return min((int64_t)(mt * MH + half0) * 128 + quarter * 32 + lane, p.rows - 1); };
                // Slice `all` of the CTA's: d[0] (and d[1]: the second half slice's) scale its sums
                auto drain = [&](int all, const float (&d)[2]) {
                    const int step = MH == 1 ? all : 2 * all + half0;
                    if (!mbar_wait_warp(&done[step % kDone], (step / kDone) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 14);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t acc0 = tmem_base + lane_base + (uint32_t)(acc_at.slot * kHalves * acc_cols), acc1 = acc0 + (uint32_t)((kHalves - 1) * acc_cols);
                    const Pair scale0 = pair_of(d[0], d[0]), scale1 = pair_of(d[1], d[1]);
                    if constexpr (CODES) {
                        const int slot = all % kStepSlots;
                        if (!mbar_wait_warp(&steps_full[slot], (all / kStepSlots) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 20);
                        const float *d8 = &step_ring[slot][0][0], *e8 = d8 + bn;
#pragma unroll
                        for (int c = 0; c < kMine; c += 16) {
                            uint32_t t[16], u[16];
                            tmem_ld16_pair(acc0 + c, acc1 + c, t, u);
#pragma unroll
                            for (int j = 0; j < 16; j += 4) {
                                const float4 s4 = *(const float4*)(d8 + c + j), r4 = *(const float4*)(e8 + c + j);
                                const Pair sv[2] = {pair_of(s4.x, s4.y), pair_of(s4.z, s4.w)}, rv[2] = {pair_of(r4.x, r4.y), pair_of(r4.z, r4.w)};
#pragma unroll
                                for (int q = 0; q < 2; ++q) {
                                    const Pair even = pair_mul(pair_mul(sv[q], scale0), pair_of(t[j + 2 * q], t[j + 2 * q + 1]));
                                    Pair& to = sum[(c + j) / 2 + q];
                                    to = pair_add(to, pair_fma(pair_mul(rv[q], scale1), pair_of(u[j + 2 * q], u[j + 2 * q + 1]), even));
                                }
                            }
                        }
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&steps_empty[slot]);
                    } else {
#pragma unroll
                        for (int h = 0; h < kHalves; ++h) {
                            const uint32_t at = h ? acc1 : acc0;
                            const Pair scale = h ? scale1 : scale0;
#pragma unroll
                            for (int c = 0; c < kMine; c += 16) {
                                {
                                    uint32_t t[16];
                                    if (MH == 1) {  // hi and lo of a token
                                        uint32_t u[16];
                                        tmem_ld16_pair(at + c, at + bn + c, t, u);
#pragma unroll
                                        for (int j = 0; j < 16; j += 2) sum[(c + j) / 2] = pair_fma(scale, pair_add(pair_of(t[j], t[j + 1]), pair_of(u[j], u[j + 1])), sum[(c + j) / 2]);
                                    } else {
                                        tmem_ld16(at + c, t);
#pragma unroll
                                        for (int j = 0; j < 16; j += 2) sum[(c + j) / 2] = pair_fma(scale, pair_of(t[j], t[j + 1]), sum[(c + j) / 2]);
                                    }
                                }
                            }
                        }
                    }
                    // this warp has read the accumulators: the tensor core may overwrite them
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&drained[step % kDone]);
                    acc_at.skip(2);
                    if (CODES && ++run == run_length) flush();
                };
                if constexpr (F::kquant) {
                    auto d_of = [&](int u) -> float {
                        if (TYPE == RQ_Q4_K) return rq_h2f(__ldg((const uint16_t*)(p.main + (my_row() * p.units + u) * 144)));
                        return rq_h2f(__ldg(p.scale + my_row() * p.units + u));
                    };
                    float d_next = d_of(u0);
                    int all = slice_base;
                    for (int u = u0; u < u1; ++u) {
                        const float d = d_next;
                        if (u + 1 < u1) d_next = d_of(u + 1);  // the next unit's scale is on its way
                        const int n = Order::closes(u, u1) ? 5 : 4;
#pragma unroll 1
                        for (int sl = 0; sl < n; ++sl, ++all)
                            // MH = 1: this set's slices are the even or the odd ones of the CTA's
                            if (MH == 2 || (all & 1) == set) {
                                const float scale[2] = {sl < 4 ? d : -kMinUnscale, 0.f};
                                drain(all, scale);
                            }
                    }
                } else {
                    // a unit's eight fp16 scales, the next unit's on their way: one load where rows are whole units (a load of two bytes goes to
                    // 32 lines, as one of sixteen does)
                    const bool wide = (p.blocks32 & 7) == 0 && ((uintptr_t)p.scale & 15) == 0;
                    auto d_of = [&](int u) -> uint4 {
                        const uint16_t* at = p.scale + my_row() * p.blocks32 + 8 * u;
                        if (wide) return __ldg((const uint4*)at);
                        uint32_t w[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int b = 8 * u + 2 * i;
                            w[i] = (b < p.blocks32 ? (uint32_t)__ldg(at + 2 * i) : 0u) | (b + 1 < p.blocks32 ? (uint32_t)__ldg(at + 2 * i + 1) << 16 : 0u);
                        }
                        return make_uint4(w[0], w[1], w[2], w[3]);
                    };
                    uint4 next = d_of(u0);
                    int all = slice_base;  // (a multiple of four)
#pragma unroll 1
                    for (int u = u0; u < u1; ++u, all += 4) {
                        const uint4 d = next;
                        if (u + 1 < u1) next = d_of(u + 1);
#pragma unroll 1
                        for (int sl = MH == 1 ? set : 0; sl < 4; sl += MH == 1 ? 2 : 1) {
                            const uint32_t w = sl < 2 ? (sl == 0 ? d.x : d.y) : (sl == 2 ? d.z : d.w);
                            const float scale[2] = {rq_h2f((uint16_t)(w & 0xffff)), rq_h2f((uint16_t)(w >> 16))};
                            drain(all + sl, scale);
                        }
                    }
                }
                slice_base += Order::count(u0, u1);
                const int r0 = quarter * 32 + lane;
                if (CODES && flushed) {  // the totals and what is in the registers
#pragma unroll
                    for (int c = 0; c < kMine; c += 16) {
                        uint32_t v[16];
                        tmem_ld16(totals + c, v);
#pragma unroll
                        for (int j = 0; j < 16; j += 2) sum[(c + j) / 2] = pair_add(pair_of(v[j], v[j + 1]), sum[(c + j) / 2]);
                    }
                }
                // MH = 1: each set gives the other half of the columns and keeps the sums of the even and odd slices of its own half
                constexpr int kLeave = MH == 1 ? kMine / 2 : kMine;  // tokens that a thread carries out
                Pair left[kLeave / 2];
                if (MH == 1) {
                    const int give = (1 - set) * kLeave, keep = set * kLeave;
#pragma unroll
                    for (int j = 0; j < kLeave; ++j) joined[(give + j) * 128 + r0] = pair_at(set ? sum[j / 2] : sum[(kLeave + j) / 2], j & 1);
                    asm volatile("bar.sync 3, %0;" ::"n"(kDrainWarps * 32) : "memory");
#pragma unroll
                    for (int j = 0; j < kLeave; j += 2)
                        left[j / 2] = pair_add(set ? sum[(kLeave + j) / 2] : sum[j / 2], pair_of(joined[(keep + j) * 128 + r0], joined[(keep + j + 1) * 128 + r0]));
                    asm volatile("bar.sync 3, %0;" ::"n"(kDrainWarps * 32) : "memory");
                } else {
#pragma unroll
                    for (int j = 0; j < kLeave / 2; ++j) left[j] = sum[j];
                }
                const int from = MH == 1 ? set * kLeave : 0;  // the first of them
                const int tokens_here = dead ? 0 : min(kLeave, p.tokens - nt * bn - from);
                // how many of this thread's tokens count, and where they go (found anew by each, as the row)
                auto live = [&]() { return (int64_t)(mt * MH + half0) * 128 + r0 < p.rows ? tokens_here : 0; };
                auto out = [&]() { return p.y + ((int64_t)(mt * MH + half0) * 128 + r0) * p.yn + (int64_t)(nt * bn + from) * p.yt; };
                if (whole) {
                    const int n = live();
                    float* at = out();
#pragma unroll
                    for (int j = 0; j < kLeave; ++j) {
                        if (j < n) *at = pair_at(left[j / 2], j & 1);
                        at += p.yt;
                    }
                } else {
                    const size_t tile_floats = (size_t)bn * 128 * MH, place0 = (size_t)from * 128 * MH + half0 * 128 + r0;
                    auto piece_of = [&](int c) { return p.partial + (size_t)Deal::place(c, c0) * tile_floats + place0; };
                    {
                        const int n = live();
                        float* const piece = piece_of((int)blockIdx.x);
#pragma unroll
                        for (int j = 0; j < kLeave; ++j)
                            if (j < n) piece[j * 128 * MH] = pair_at(left[j / 2], j & 1);
                    }
                    __threadfence();
                    asm volatile("bar.sync 2, %0;" ::"n"(kDrainWarps * 32) : "memory");
                    if (tid == 0) {
                        asm volatile("griddepcontrol.wait;" ::: "memory");  // the counters were zeroed by the kernel before this one
                        last_piece = atomicAdd(p.arrived + t, 1) == c1 - c0;
                    }
                    asm volatile("bar.sync 2, %0;" ::"n"(kDrainWarps * 32) : "memory");
                    if (last_piece) {
                        __threadfence();
                        // A few tokens at a time, two pieces at a time: 64 loads in flight, in the registers that the sums have left (a branch for each
                        // load would make each wait for the one before; the padding tokens' places exist and hold nothing that is used). Tiles of 48 tokens, 24
                        // a thread: 12 at a time (Q6_K 8192 x 1024, 48 tokens, by 8 / 12 / 24: 13.0 / 11.6 / 11.9 us; 1670 x 12800, 34 tokens: 26.2 / 23.8 / 29.1).
                        constexpr int kAtOnce = kLeave % 32 == 0 ? 32 : (kLeave % 16 == 0 ? 16 : (kLeave % 12 == 0 ? 12 : 8));
                        const int n = live();
#pragma unroll 1
                        for (int j0 = 0; j0 < n; j0 += kAtOnce) {
                            Pair total[kAtOnce / 2];
#pragma unroll
                            for (int q = 0; q < kAtOnce / 2; ++q) total[q] = 0;
#pragma unroll 1
                            for (int c = c0; c <= c1; c += 2) {
                                const bool two = c < c1;
                                const float* one = piece_of(c) + (size_t)j0 * 128 * MH;
                                const float* other = two ? piece_of(c + 1) + (size_t)j0 * 128 * MH : one;
                                float v[kAtOnce], w[kAtOnce];
#pragma unroll
                                for (int q = 0; q < kAtOnce; ++q) {
                                    v[q] = __ldcg(one + q * 128 * MH);
                                    w[q] = __ldcg(other + q * 128 * MH);
                                }
#pragma unroll
                                for (int q = 0; q < kAtOnce; q += 2)
                                    total[q / 2] = pair_add(total[q / 2], two ? pair_add(pair_of(v[q], v[q + 1]), pair_of(w[q], w[q + 1])) : pair_of(v[q], v[q + 1]));
                            }
                            float* at = out() + (int64_t)j0 * p.yt;
#pragma unroll
                            for (int q = 0; q < kAtOnce; ++q) {
                                if (j0 + q < n) *at = pair_at(total[q / 2], q & 1);
                                at += p.yt;
                            }
                        }
                    }
                }
            }
        };
        if constexpr (MH == 2) {
            if (bn == 96) run_tiles(Columns<96>());
            else if (F::kquant && bn == 128) run_tiles(Columns<F::kquant ? 128 : 64>());
            else run_tiles(Columns<64>());
        } else {
            switch (bn) {
                case 16: run_tiles(Columns<16>()); break;
                case 32: run_tiles(Columns<32>()); break;
                case 48: run_tiles(Columns<48>()); break;
                default: run_tiles(Columns<64>()); break;
            }
        }
    } else if (warp < kMiscFirst) {
        // ------------------------------------------------------------ staging groups: stored bytes -> integer operands in tensor memory
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::stage_regs));
        const int group = (warp - kStageFirst) >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t a_lane = a_ring + ((uint32_t)((warp & 3) * 32) << 16);
        uint4* const left = stash + (MH == 1 ? 0 : group * 128) + r;  // [4] of this thread's, 128 * MH apart
        Ring raw_at(p.raw_slots);
        bool dead = false;
        // the operand slot of a step, once the step that read it is done
        auto wait_slot = [&](int step) {
            int freed = step - p.a_slots;
            if (freed >= 0) {
                if (!mbar_wait_warp(&done[freed % kDone], (freed / kDone) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 11);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            }
        };
        auto staged = [&](int step) {
            tmem_st_wait();
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&a_full[step % kDone]);  // one arrival per warp (an arrival is an atomic on the barrier)
        };
        auto wait_raw = [&]() {
            if (!mbar_wait_warp(&raw_full[raw_at.slot], raw_at.phase, p.wait_ns, dead)) atomicExch(p.error_flag, 18);
        };
        // This warp has read its rows of a slot: said behind the stores that needed them (said behind the loads, some lanes were given the
        // slot's next bytes).
        auto release_raw = [&]() {
            if (lane == 0) mbar_arrive(&raw_empty[raw_at.slot]);
        };
        // the window's minimum terms: inputs 8 j .. of the operand are superblock j's (zeros outside u0 .. u1), 32 + 8 j .. their residuals
        auto stage_minimum = [&](int u, int step) {
            wait_slot(step);
            const uint32_t at = a_lane + (uint32_t)((step & a_mask) * F::a_cols);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int of = (u & ~3) + j;
                const uint4 hdr = of >= u0 && of < u1 ? left[j * (128 * MH)] : make_uint4(0, 0, 0, 0);
                uint32_t hi[4], lo[4];
                minimum_terms(hdr, hi, lo);
                tmem_st4(at + 4 * j, hi);
                tmem_st4(at + 16 + 4 * j, lo);
            }
            staged(step);
        };
        // slice sl of unit u, whose stored bytes are at src
        auto stage = [&](int sl, int u, const uint8_t* src, int step) {
            Stored<TYPE> w;
            w.load(src, r, u, sl, p.permuted != 0);
            if (TYPE == RQ_Q4_K && sl == 0) left[(u & 3) * (128 * MH)] = w.v[0];
            const uint32_t at = a_lane + (uint32_t)((step & a_mask) * F::a_cols);
            uint32_t o[16], res[16];
            w.expand(sl, 0, o, res);
            wait_slot(step);
            tmem_st16(at, o);
            if (F::residual) tmem_st16(at + 32, res);
            w.load_second(src, r, sl);
            w.expand(sl, 1, o, res);
            tmem_st16(at + 16, o);
            if (F::residual) tmem_st16(at + 48, res);
            staged(step);
        };
        if constexpr (MH == 1) {
            // a group has the same slice of every unit; group 0 the minimum terms too, of the headers that it sees
            constexpr int kPer = 4 / F::raw_slices;
            raw_at.skip(group / F::raw_slices);
            int first = 0;  // the unit's first slice, of the CTA's
            while (walk.next(tile, u0, u1)) {
#pragma unroll 1
                for (int u = u0; u < u1; ++u, first += 4, raw_at.skip(kPer)) {
                    wait_raw();
                    stage(group, u, raw + (size_t)raw_at.slot * F::raw_bytes, first + group);
                    release_raw();
                    if (Order::closes(u, u1)) {
                        if (group == 0) stage_minimum(u, first + 4);
                        ++first;
                    }
                }
            }
        } else {
            // a group has a row half: every second operand tile, every second tile of stored bytes
            raw_at.skip(group);
            int step = group;
            while (walk.next(tile, u0, u1)) {
#pragma unroll 1
                for (int u = u0; u < u1; ++u) {
                    const uint8_t* src = raw;
#pragma unroll 1
                    for (int sl = 0; sl < 4; ++sl, step += 2) {
                        if (sl % F::raw_slices == 0) {
                            wait_raw();
                            src = raw + (size_t)raw_at.slot * F::raw_bytes;
                        }
                        stage(sl, u, src, step);
                        if (sl % F::raw_slices == F::raw_slices - 1) { release_raw(); raw_at.skip(2); }
                    }
                    if (Order::closes(u, u1)) { stage_minimum(u, step); step += 2; }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(S::other_regs));
        // These warps wait as a whole and one lane acts: a look at a barrier by a lone lane is not suspended, it is repeated every 160 cycles, and
        // sees an arrival 100 to 200 cycles later than a whole warp does (Q4_K 14336 x 4096, 512 tokens: 154 us so, 135 with whole warps).
        const bool leader = elect_one();  // (the same lane every time)
        // The copying warps leave only after every copy that they issued has landed: the last `slots` of n on a ring of barriers (bounded).
        auto landed = [&](uint64_t* full, int slots, int n) {
            bool dead = false;
            for (int i = max(0, n - slots); i < n && !dead; ++i)
                if (!mbar_wait_warp(&full[i % slots], (i / slots) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 24);
        };
        if (warp < kMiscFirst + kIssuers) {
            // ------------------------------------------------------------ the issuing warps
            const int me = warp - kMiscFirst;
            const uint32_t idesc = instr_desc(bn), idesc2 = instr_desc(acc_cols);
            constexpr int kSkip = MH == 1 ? kIssuers : 1;  // slices from one of this warp's to the next (steps: two)
            Ring b_at(p.b_slots, MH == 1 ? me : 0), acc_at(sums, me);
            int ks = MH == 1 ? me : 0, end = 0;
            bool dead = false;
            while (walk.next(tile, u0, u1)) {
                end += Order::count(u0, u1);
#pragma unroll 1
                for (; ks < end; ks += kSkip, b_at.skip(kSkip), acc_at.skip(2)) {
                    const int step = MH == 1 ? ks : 2 * ks + me, bslot = b_at.slot;
                    if (!mbar_wait_warp(&b_full[bslot], b_at.phase, p.wait_ns, dead)) atomicExch(p.error_flag, 17);
                    const uint32_t bbase = smem_u32(smem + (size_t)bslot * b_bytes);
                    const uint64_t b_hi = smem_desc(bbase), b_lo = smem_desc(bbase + bn * 128);
                    if (step >= sums && !mbar_wait_warp(&drained[(step - sums) % kDone], ((step - sums) / kDone) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 15);
                    if (!mbar_wait_warp(&a_full[step % kDone], (step / kDone) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 13);
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t a_hi = a_ring + (uint32_t)((step & a_mask) * F::a_cols), a_res = a_hi + 32;
                    if (leader && !dead) {
#pragma unroll
                        for (int h = 0; h < kHalves; ++h) {
                            const uint32_t acc = tmem_base + (uint32_t)((acc_at.slot * kHalves + h) * acc_cols);
                            constexpr int kk_n = 4 / kHalves;
                            // kk: 16-wide steps, 32 bytes along K (in 16-byte units of the descriptor's start address), eight columns of A
                            if (CODES) {
#pragma unroll
                                for (int k = 0; k < kk_n; ++k) { const int kk = h * kk_n + k; mma_f16_ts(acc, a_hi + 8 * kk, b_hi + 2 * kk, idesc, k ? 1u : 0u); }
                            } else if (MH == 1) {
                                // columns [0, bn): A x B_hi; [bn, 2 bn): A x B_lo and, small as well, the residual x B_hi
#pragma unroll
                                for (int k = 0; k < kk_n; ++k) { const int kk = h * kk_n + k; mma_f16_ts(acc, a_hi + 8 * kk, b_hi + 2 * kk, idesc2, k ? 1u : 0u); }
                                if (F::residual)
#pragma unroll
                                    for (int kk = 0; kk < kk_n; ++kk) mma_f16_ts(acc + bn, a_res + 8 * kk, b_hi + 2 * kk, idesc, 1u);
                            } else {
                                // the cross terms (2^-11 of the sum) first, while the accumulator is small
#pragma unroll
                                for (int k = 0; k < kk_n; ++k) {
                                    const int kk = h * kk_n + k;
                                    mma_f16_ts(acc, a_hi + 8 * kk, b_lo + 2 * kk, idesc, k ? 1u : 0u);
                                    if (F::residual) mma_f16_ts(acc, a_res + 8 * kk, b_hi + 2 * kk, idesc, 1u);
                                }
#pragma unroll
                                for (int k = 0; k < kk_n; ++k) { const int kk = h * kk_n + k; mma_f16_ts(acc, a_hi + 8 * kk, b_hi + 2 * kk, idesc, 1u); }
                            }
                        }
                        // one commit: the sums are complete and, after the last step that reads them, the operand and activation slots are free
                        mma_commit(&done[step % kDone]);
                    }
                    __syncwarp();
                }
            }
            // nothing may be in flight when tensor memory is freed. (The drain warps have waited for every step by then, unless one of their waits ran out.)
            if (leader) mma_commit(&ended[me]);
            __syncwarp();
            dead = false;
            if (!mbar_wait_warp(&ended[me], 0, p.wait_ns, dead)) atomicExch(p.error_flag, 23);
        } else if (warp == kMiscFirst + kIssuers) {
            // ------------------------------------------------------------ activation copies (the images were written by the kernel before this one)
            asm volatile("griddepcontrol.wait;" ::: "memory");
            Ring b_at(p.b_slots), steps_at(kStepSlots);
            int ks_all = 0, images = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const uint8_t* src = p.xs + (size_t)(tile / p.tiles_m) * p.image_tiles * b_bytes;
                int u = u0, sl = 0;
                for (int left = Order::count(u0, u1); left > 0; --left, ++ks_all) {
                    if (ks_all >= p.b_slots) {
                        // the last steps that read the slot, one of each row half (they come from different warps)
#pragma unroll
                        for (int m = 0; m < MH && !dead; ++m) {
                            const int freed = (ks_all - p.b_slots) * MH + m;
                            if (!mbar_wait_warp(&done[freed % kDone], (freed / kDone) & 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 16); }
                        }
                        if (dead) break;
                    }
                    const int image = sl < 4 ? 4 * u + sl : 4 * p.units + (u >> 2);
                    if (++sl >= 4 && !(sl == 4 && Order::closes(u, u1))) { sl = 0; ++u; }
                    if (leader) {
                        mbar_expect_tx(&b_full[b_at.slot], (uint32_t)b_bytes);
                        bulk_g2s(smem + (size_t)b_at.slot * b_bytes, src + (size_t)image * b_bytes, (uint32_t)b_bytes, &b_full[b_at.slot]);
                    }
                    b_at.next();
                    ++images;
                    if (CODES) {
                        if (ks_all >= kStepSlots && !mbar_wait_warp(&steps_empty[steps_at.slot], steps_at.phase ^ 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 16); break; }
                        if (leader) {
                            mbar_expect_tx(&steps_full[steps_at.slot], (uint32_t)(8 * bn));
                            bulk_g2s(&step_ring[steps_at.slot][0][0], p.steps + ((size_t)(tile / p.tiles_m) * p.image_tiles + image) * 2 * bn, (uint32_t)(8 * bn), &steps_full[steps_at.slot]);
                        }
                        steps_at.next();
                    }
                }
            }
            landed(b_full, p.b_slots, images);
            if (CODES) landed(steps_full, kStepSlots, ks_all);
        } else {
            // ------------------------------------------------------------ stored bytes: constants of the model, nothing to wait for before the first fetches
            Ring at(p.raw_slots);
            int n = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const int mt = tile % p.tiles_m;
                constexpr int kPer = 4 / F::raw_slices;  // TMA tiles per unit and row half
                for (int t = u0 * kPer; t < u1 * kPer && !dead; ++t)
                    for (int m = 0; m < MH; ++m, ++n) {
                        if (n >= p.raw_slots && !mbar_wait_warp(&raw_empty[at.slot], at.phase ^ 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 19); break; }
                        if (leader) {
                            mbar_expect_tx(&raw_full[at.slot], F::raw_bytes);
                            tma_load_2d(raw + (size_t)at.slot * F::raw_bytes, &p.tile_map, t * F::box_bytes, (mt * MH + m) * 128, &raw_full[at.slot]);
                        }
                        at.next();
                    }
            }
            landed(raw_full, p.raw_slots, n);
        }
        __syncwarp();
    }
    // free the tensor memory: everyone is past its use
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMiscFirst) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

template <int TYPE, int MH, bool CODES>
int launch_tc(const TcParams& p, int ctas, size_t smem, cudaStream_t s) {
    auto kernel = rq_tc_kernel<TYPE, MH, CODES>;
    static bool configured[64] = {};
    int dev = 0;
    RQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        RQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (CODES ? 218 : 225) * 1024));  // 227 KB less the static part
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(tc_threads<MH, CODES>());
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RQ_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    return RQ_OK;
}
template <int TYPE>
int launch_tc(const TcParams& p, int mh, bool codes, int ctas, size_t smem, cudaStream_t s) {
    if constexpr (!Format<TYPE>::kquant) {
        if (codes) return launch_tc<TYPE, 1, true>(p, ctas, smem, s);
    }
    return mh == 1 ? launch_tc<TYPE, 1, false>(p, ctas, smem, s) : launch_tc<TYPE, 2, false>(p, ctas, smem, s);
}

}  // namespace

size_t rq_matmul_scratch_bytes(const rq_ctx* ctx, int64_t rows, int64_t cols, int tokens) { return scratch_bound(ctx->sm_count, rows, cols, tokens); }

// RQ_ERR_UNSUPPORTED (no error text) = not one of the four formats; INT8_CACHED: no records of this call's column, or no room for the
// image beside them (a cached call allocates nothing). act_mode FLOAT, INT8 (step 32 / 256), over Q8_0 / Q4_0 also INT8_CACHED.
int rq_launch_matmul(rq_ctx* ctx, const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens, float* y, int64_t yn, int64_t yt, int act_mode, int step, cudaStream_t s) {
    if (!w->has_tile_map || !rq_type_has_fast_path(w->type)) return RQ_ERR_UNSUPPORTED;
    const bool codes = act_mode != RQ_ACT_FLOAT && (w->type == RQ_Q8_0 || w->type == RQ_Q4_0);
    // fp32 activations over an odd number of 32-value blocks stay with the matvec kernel, as they were: it has no fp16 range to keep to
    if (!codes && w->cols % BK) return RQ_ERR_UNSUPPORTED;
    const TcCut cut = tc_cut(w->type, codes, ctx->sm_count, w->rows, w->cols, tokens);
    const bool bytes = codes && cut.mh == 2;
    const bool cached = act_mode == RQ_ACT_INT8_CACHED;
    if (cached && (!codes || ctx->act_cols != w->cols || ctx->act_tokens != tokens || ctx->act_step != step || scratch_bytes(cut) > ctx->act_scratch_bytes)) return RQ_ERR_UNSUPPORTED;
    int rc = rq_ensure_act_scratch(ctx, scratch_bytes(cut), s);
    if (rc) return rc;
    uint8_t* xs = ctx->act_scratch + cut.records_bytes;
    if (!cached) ctx->act_cols = 0;  // whatever int8 records the scratch held for INT8_CACHED calls are gone
    float* partial = (float*)(xs + cut.xs_bytes + cut.steps_bytes);
    int* arrived = (int*)((uint8_t*)partial + cut.partial_bytes);
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    {
        const int padded = cut.n_tiles * cut.bn;
        cudaLaunchConfig_t cfg = {};
        const unsigned groups = (unsigned)(padded / 8), deep = (groups + 65534) / 65535;
        cfg.gridDim = dim3((unsigned)cut.units, (groups + deep - 1) / deep, deep);
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        auto prep_of = [&](auto image) {
            constexpr Image kImage = decltype(image)::value;
            if constexpr (kImage != kPairs)
                if (cached) return rq_tc_prep_kernel<-1, kImage>;
            return step == 256 ? rq_tc_prep_kernel<256, kImage> : rq_tc_prep_kernel<32, kImage>;
        };
        auto prep = act_mode == RQ_ACT_FLOAT ? rq_tc_prep_kernel<0, kPairs> : !codes ? prep_of(ImageOf<kPairs>()) : (bytes ? prep_of(ImageOf<kBytes>()) : prep_of(ImageOf<kCodes>()));
        RQ_CUDA(cudaLaunchKernelEx(&cfg, prep, x, sk, st, (int)w->cols, cut.units, tokens, padded, cut.bn, cut.image_tiles, cut.windows, bytes && w->type == RQ_Q8_0 && rq_plane_permuted(w->type, w->cols) ? 1 : 0, ctx->act_scratch, xs, (float*)(xs + cut.xs_bytes), arrived, cut.rest_tiles));
    }
    if (bytes) {
        RqInt8Params q;
        q.tile_map = w->tile_map; q.scale = w->scale; q.rows = w->rows;
        q.blocks32 = (int)(w->cols / 32); q.units = cut.units; q.permuted = rq_plane_permuted(w->type, w->cols) ? 1 : 0;
        q.xs = xs; q.steps = (const float*)(xs + cut.xs_bytes); q.tokens = tokens; q.y = y; q.yn = yn; q.yt = yt;
        q.tiles_m = cut.tiles_m; q.whole = cut.whole; q.rest_tiles = cut.rest_tiles; q.share = cut.share;
        q.partial = partial; q.arrived = arrived; q.error_flag = ctx->error_flag; q.wait_ns = ctx->wait_limit_ns;
        rc = rq_launch_tc_int8(w->type, q, cut.ctas, s);
        if (rc == RQ_OK) { ctx->act_cols = w->cols; ctx->act_tokens = tokens; ctx->act_step = step; }
        return rc;
    }
    TcParams p;
    p.tile_map = w->tile_map;
    p.main = w->main; p.scale = w->scale; p.rows = w->rows;
    p.blocks32 = (int)(w->cols / 32); p.units = cut.units; p.permuted = rq_plane_permuted(w->type, w->cols) ? 1 : 0;
    p.xs = xs; p.image_tiles = cut.image_tiles; p.bn = cut.bn; p.tokens = tokens; p.y = y; p.yn = yn; p.yt = yt;
    p.tiles_m = cut.tiles_m; p.whole = cut.whole; p.rest_tiles = cut.rest_tiles; p.share = cut.share;
    p.steps = (const float*)(xs + cut.xs_bytes);
    p.partial = partial; p.arrived = arrived;
    p.raw_slots = cut.raw_slots; p.b_slots = cut.b_slots; p.a_slots = cut.a_slots; p.accs = cut.accs;
    p.error_flag = ctx->error_flag; p.wait_ns = ctx->wait_limit_ns;
    switch (w->type) {
        case RQ_Q4_K: rc = launch_tc<RQ_Q4_K>(p, cut.mh, codes, cut.ctas, cut.smem, s); break;
        case RQ_Q6_K: rc = launch_tc<RQ_Q6_K>(p, cut.mh, codes, cut.ctas, cut.smem, s); break;
        case RQ_Q8_0: rc = launch_tc<RQ_Q8_0>(p, cut.mh, codes, cut.ctas, cut.smem, s); break;
        default: rc = launch_tc<RQ_Q4_0>(p, cut.mh, codes, cut.ctas, cut.smem, s); break;
    }
    if (rc == RQ_OK && codes) { ctx->act_cols = w->cols; ctx->act_tokens = tokens; ctx->act_step = step; }
    return rc;
}
