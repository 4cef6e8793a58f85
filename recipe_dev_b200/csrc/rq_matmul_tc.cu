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
// tensor core's 128-byte-swizzled K-major image; INT8 calls feed code * step through the same path.
//
// One CTA per SM, persistent. Work is counted in UNITS, 256 inputs of one row tile (128 * MH rows) x one token tile: every CTA
// takes the same number of whole tiles and then an equal share of the units that are left, whatever tile they fall in; a tile
// that is shared by several CTAs is added up by rq_tc_sum_kernel in unit order (the same bits on every run). Roles in a CTA:
//   * raw copies: one TMA tile of 128 rows x one unit of stored bytes at a time (Q8_0: half a unit) into a ring;
//   * activation copies: one bulk copy per 64-wide slice, B_hi | B_lo of the token tile, into a ring;
//   * staging groups of four warps (thread = row): stored bytes -> 64 fp16 integers -> operand slot in TENSOR MEMORY
//     (tcgen05.st; the A operand of tcgen05.mma may live there, so the unpacked weights never touch shared memory). The groups
//     take operand tiles in turn, so that their chains of latencies (barrier, load, unpack, store, fence) overlap;
//   * one issuing thread: per slice and row half, the products into one of a ring of accumulators, one tcgen05.commit;
//   * eight drain warps: accumulator -> scale * sum -> fp32 registers, round-to-nearest, then Y or the partial sums.
//
// The tensor core adds into its fp32 accumulator by TRUNCATION, a bias that grows with the length of the chain (measured: 7e-7
// relative over 256 inputs, 1.2e-5 over 4096), so a sum stays in tensor memory for one 64-wide slice (32 inputs for the
// formats whose scale changes there) and the small cross terms go first or into columns of their own.
//
// Two forms. MH = 1 (token tiles of up to 64): B_hi and B_lo are one operand of 2 * bn columns, so a slice is four (Q6_K:
// eight) instructions and the low products have accumulators of their own; the time goes to unpacking and to the weights'
// bytes, so three staging groups. MH = 2 (token tiles of up to 96): two row halves share each activation tile, which halves
// the activation bytes a CTA pulls from L2 (they, at 4 bytes per input and token, are what the large shapes would be bound
// by); products of hi and lo share an accumulator, drained by all eight warps with 96 fp32 sums a thread (setmaxnreg).
//
// The Q4_K minimum term, sum_g (8 * d * sc_g - dmin * m_g) * (sum of x over group g), is a second, 32 times smaller product: per
// window of eight superblocks two more slices (the terms' fp16 hi and lo) whose "activations" are the group sums.
//
// Every wait is bounded; a wait that runs out records a code in the context's error word, the thread stops waiting and the CTA
// still frees its tensor memory before it exits.
#include "rq_internal.cuh"
#include "rq_mma.cuh"

using namespace rqmma;

namespace {

constexpr int kDrainWarps = 8;
constexpr int kDone = 32;                    // ring of "step finished" barriers, indexed by the step (see the kernel)
constexpr int kMaxRaw = 8, kMaxB = 8, kMaxA = 8, kMaxAcc = 8;
constexpr float kMinScale = 256.0f, kMinUnscale = 1.0f / 256.0f;  // the minimum term's weights are scaled so that their fp16 residuals are no subnormals

template <int MH> struct Shape;
template <> struct Shape<1> { static constexpr int groups = 3, cols = 32; };   // staging groups; accumulator columns (tokens) a drain thread holds
template <> struct Shape<2> { static constexpr int groups = 2, cols = 48; };
template <int MH> __host__ __device__ constexpr int tc_threads() { return (kDrainWarps + 4 * Shape<MH>::groups + 4) * 32; }

template <int TYPE> struct Format {
    static constexpr bool kquant = TYPE == RQ_Q4_K || TYPE == RQ_Q6_K;
    static constexpr bool residual = TYPE == RQ_Q6_K;            // a second operand tile
    static constexpr int halves = kquant ? 1 : 2;                // sums that leave tensor memory per 64-wide slice
    static constexpr int box_bytes = TYPE == RQ_Q4_K ? 144 : (TYPE == RQ_Q6_K ? 208 : 128);  // stored bytes of a row in one TMA tile
    static constexpr int raw_slices = TYPE == RQ_Q8_0 ? 2 : 4;   // slices in one TMA tile
    static constexpr int raw_bytes = 128 * box_bytes;
    static constexpr int a_cols = residual ? 64 : 32;            // tensor-memory columns of an operand slot
};

struct TcParams {
    CUtensorMap tile_map;  // the weight's main plane as a [rows][row bytes] byte matrix (TMA descriptor; first: 64-byte aligned)
    const uint8_t* main;
    const uint16_t* scale;
    int64_t rows;
    int blocks32;          // 32-value blocks per row
    int units;             // 256-value units per row (a last one may be partial for the 32-value formats)
    int permuted;          // Q8_0 / Q4_0: the plane's chunks are permuted (rows of whole units)
    const uint8_t* xs;     // activation images: [token tile][image tile][hi | lo][bn rows x 128 bytes, swizzled]
    int image_tiles;       // 4 * units, then one per window of eight superblocks (Q4_K)
    int bn, tokens;
    float* y; int64_t yn, yt;
    int tiles_m, whole, rest_tiles;  // row tiles; whole tiles per CTA; tiles shared out by units
    float* partial;        // [2 * CTAs][bn][128 * MH]
    int raw_slots, b_slots, a_slots, accs;
    int* error_flag;
    unsigned long long wait_ns;
};

// The tiles and unit ranges of one CTA, in the order every role walks them.
struct Walk {
    const int whole, units;
    int i, at, end;  // whole tiles taken; position among the shared units (fewer than CTAs x units of them: 32 bits)
    __device__ __forceinline__ Walk(int whole_, int rest, int units_) : whole(whole_), units(units_), i(0) {
        const int64_t total = (int64_t)rest * units_;
        at = (int)(blockIdx.x * total / gridDim.x);
        end = (int)((blockIdx.x + 1) * total / gridDim.x);
    }
    __device__ __forceinline__ bool next(int& tile, int& u0, int& u1) {
        if (i < whole) { tile = i * gridDim.x + blockIdx.x; u0 = 0; u1 = units; ++i; return true; }
        if (at >= end) return false;
        const int t = at / units;
        tile = whole * gridDim.x + t;
        u0 = at - t * units;
        u1 = min(units, u0 + end - at);
        at += u1 - u0;
        return true;
    }
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
// 32 consecutive inputs of one row (`half` of the 64-wide slice `sl` of unit `u`) from the stored bytes in shared memory, as 32
// fp16 integers (sixteen words), inputs in the order 0 2 1 3 within every four: the order the nibbles of a word come out in.
// 0x6400 | n is the fp16 number 1024 + n; the subtraction that follows and the product with a scale are exact.
// ------------------------------------------------------------------------------------------
template <int TYPE>
__device__ __forceinline__ void unpack32(const uint8_t* tile, int r, int u, int sl, int half, bool permuted, uint32_t (&o)[16], uint32_t (&res)[16]) {
    if (TYPE == RQ_Q4_K) {
        const uint8_t* blk = tile + r * 144;
        const uint4 hdr = *(const uint4*)blk;
        const uint4 q0 = *(const uint4*)(blk + 16 + 32 * sl), q1 = *(const uint4*)(blk + 32 + 32 * sl);
        int sc, mn;
        rq_q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * sl + half, sc, mn);
        const __half2 sc2 = __half2half2(__int2half_rn(sc)), k1032 = __half2half2(__float2half_rn(1032.0f));
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t a = ((w[j] >> (4 * half)) & 0x000F000Fu) | 0x64006400u;      // inputs 4j, 4j + 2
            const uint32_t b = ((w[j] >> (4 * half + 8)) & 0x000F000Fu) | 0x64006400u;  // inputs 4j + 1, 4j + 3
            o[2 * j] = as_u32(__hmul2(__hsub2(as_half2(a), k1032), sc2));
            o[2 * j + 1] = as_u32(__hmul2(__hsub2(as_half2(b), k1032), sc2));
        }
    } else if (TYPE == RQ_Q6_K) {
        const int ch = sl >> 1, sel = sl & 1, g = 2 * sel + half;
        const uint8_t* body = tile + r * 208;
        const uint4 l0 = *(const uint4*)(body + 64 * ch + 32 * half), l1 = *(const uint4*)(body + 64 * ch + 32 * half + 16);
        const uint4 h0 = *(const uint4*)(body + 128 + 32 * ch), h1 = *(const uint4*)(body + 128 + 32 * ch + 16);
        const uint32_t scales = *(const uint16_t*)(body + 192 + 8 * ch + 2 * g);  // two int8 scales: inputs 0..15 and 16..31 of the group
        const uint32_t lw[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w}, hw[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
        const __half2 s_first = __half2half2(__int2half_rn((int)(int8_t)(scales & 0xff)));
        const __half2 s_second = __half2half2(__int2half_rn((int)(int8_t)(scales >> 8)));
        const __half2 k1056 = __half2half2(__float2half_rn(1056.0f));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const __half2 s2 = j < 4 ? s_first : s_second;
            const uint32_t q4 = ((lw[j] >> (4 * sel)) & 0x0F0F0F0Fu) | (((hw[j] >> (2 * g)) & 0x03030303u) << 4);  // four six-bit codes
            const uint32_t a = (q4 & 0x00FF00FFu) | 0x64006400u, b = ((q4 >> 8) & 0x00FF00FFu) | 0x64006400u;
            const __half2 ca = __hsub2(as_half2(a), k1056), cb = __hsub2(as_half2(b), k1056);  // q - 32
            const __half2 ha = __hmul2(ca, s2), hb = __hmul2(cb, s2);
            o[2 * j] = as_u32(ha);
            o[2 * j + 1] = as_u32(hb);
            res[2 * j] = as_u32(__hfma2(ca, s2, __hneg2(ha)));  // the product less its rounding: -1, 0 or 1
            res[2 * j + 1] = as_u32(__hfma2(cb, s2, __hneg2(hb)));
        }
    } else if (TYPE == RQ_Q8_0) {
        const int x = permuted ? u & 7 : 0, c = 4 * (sl & 1) + 2 * half;  // the tile holds half a unit: chunks 0..7
        const uint4 q0 = swizzled_chunk(tile, r, c ^ x), q1 = swizzled_chunk(tile, r, (c + 1) ^ x);
        const uint32_t w[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        const __half2 k1152 = __half2half2(__float2half_rn(1152.0f));
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t v = w[j] ^ 0x80808080u;  // code + 128
            o[2 * j] = as_u32(__hsub2(as_half2((v & 0x00FF00FFu) | 0x64006400u), k1152));
            o[2 * j + 1] = as_u32(__hsub2(as_half2(((v >> 8) & 0x00FF00FFu) | 0x64006400u), k1152));
        }
    } else {
        const uint4 q = swizzled_chunk(tile, r, (2 * sl + half) ^ (permuted ? u & 7 : 0));  // a block: low nibbles are its first sixteen values
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

// Q4_K: 2^8 * (dmin * m_g - 8 * d * sc_g) of a superblock's eight sub-blocks (what is left of the minimum once the codes are
// centred: for weights spread about zero an order of magnitude smaller than dmin * m_g, and so are the truncations of its sums)
// as fp16; `low`: the residual of that rounding.
__device__ __forceinline__ void minimum_terms(const uint4& hdr, bool low, uint32_t* out) {
    const float dmin = rq_h2f((uint16_t)(hdr.x >> 16)), d8 = __fmul_rn(8.0f, rq_h2f((uint16_t)(hdr.x & 0xffff)));
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        int s0, m0, s1, m1;
        rq_q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * j, s0, m0);
        rq_q4k_scale_min(hdr.y, hdr.z, hdr.w, 2 * j + 1, s1, m1);
        // both products are exact in fp32 (an fp16 times an integer below 64); their difference is rounded once
        const float a = __fmul_rn(__fsub_rn(__fmul_rn(dmin, (float)m0), __fmul_rn(d8, (float)s0)), kMinScale);
        const float b = __fmul_rn(__fsub_rn(__fmul_rn(dmin, (float)m1), __fmul_rn(d8, (float)s1)), kMinScale);
        uint32_t h, l;
        split2(a, b, h, l);
        out[j] = low ? l : h;
    }
}

// ------------------------------------------------------------------------------------------
// X -> the tensor core's operand images. A warp takes one unit of one token row: lane l the eight inputs 8 l .. 8 l + 7, so reads
// and writes are whole lines. INT8 quantises on the way with the reference's arithmetic: the extreme of a group of STEP inputs
// is the FIRST input of strictly largest magnitude, signed; inverse = -127 / extreme and d = 1 / inverse are IEEE divides,
// code = clamp(rint(x * inverse)); the image holds code * d. STEP 0: fp32 activations. Rows past the last token and inputs past
// the last column are zeros.
// ------------------------------------------------------------------------------------------
template <int STEP>
__global__ void __launch_bounds__(256) rq_tc_prep_kernel(const float* __restrict__ x, int64_t sk, int64_t st, int cols, int units, int tokens, int bn, int padded_rows, int image_tiles,
                                                          int windows, uint8_t* __restrict__ xs) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int lane = threadIdx.x & 31, unit = blockIdx.x;
    const int row = blockIdx.y * 8 + (threadIdx.x >> 5);
    if (row >= padded_rows) return;
    const int nt = row / bn, r = row - nt * bn, k0 = unit * 256 + 8 * lane;
    const bool vec = sk == 1 && (st & 3) == 0 && ((uintptr_t)x & 15) == 0;
    uint8_t* hi = xs + ((size_t)nt * image_tiles + 4 * unit + (lane >> 3)) * 2 * (size_t)bn * 128 + swizzled(r, lane & 7);
    asm volatile("griddepcontrol.wait;" ::: "memory");
    float v[8];
    if (row < tokens && k0 < cols) {  // a width is a whole number of 32-value blocks: a lane's eight inputs are all inside or all outside
        const float* src = x + (int64_t)row * st + (int64_t)k0 * sk;
        if (vec) {
            *(float4*)v = __ldg((const float4*)src);
            *(float4*)(v + 4) = __ldg((const float4*)src + 1);
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = __ldg(src + j * sk);
        }
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.f;
    }
    if (STEP != 0) {
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
        const float d = nonzero ? __fdiv_rn(1.0f, inverse) : 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            int code = __float2int_rn(__fmul_rn(v[j], inverse));
            code = code < -128 ? -128 : (code > 127 ? 127 : code);
            v[j] = __fmul_rn((float)code, d);
        }
    }
    uint32_t hw[4], lw[4];
    split2(v[0], v[2], hw[0], lw[0]);  // the order the weights' nibble pairs come in
    split2(v[1], v[3], hw[1], lw[1]);
    split2(v[4], v[6], hw[2], lw[2]);
    split2(v[5], v[7], hw[3], lw[3]);
    *(uint4*)hi = make_uint4(hw[0], hw[1], hw[2], hw[3]);
    *(uint4*)(hi + (size_t)bn * 128) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
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
        uint8_t* sums = xs + ((size_t)nt * image_tiles + 4 * units + (unit >> 3)) * 2 * (size_t)bn * 128;
        if ((lane & 7) == 0) {
            const int at = swizzled(r, unit & 7) + 4 * (lane >> 3);
            *(uint32_t*)(sums + at) = h;
            *(uint32_t*)(sums + (size_t)bn * 128 + at) = l;
        }
        if (unit == units - 1) {  // groups past the last superblock of the window count as zeros
            const int chunk = lane & 7;
            if (chunk > (unit & 7) && lane < 16) *(uint4*)(sums + (lane < 8 ? 0 : (size_t)bn * 128) + swizzled(r, chunk)) = make_uint4(0, 0, 0, 0);
        }
    }
}

// eight columns at two places of this warp's 32 lanes
__device__ __forceinline__ void tmem_ld8_pair(uint32_t a, uint32_t b, uint32_t (&u)[8], uint32_t (&v)[8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=&r"(u[0]), "=&r"(u[1]), "=&r"(u[2]), "=&r"(u[3]), "=&r"(u[4]), "=&r"(u[5]), "=&r"(u[6]), "=&r"(u[7]), "=&r"(v[0]), "=&r"(v[1]), "=&r"(v[2]), "=&r"(v[3]),
          "=&r"(v[4]), "=&r"(v[5]), "=&r"(v[6]), "=&r"(v[7])
        : "r"(a), "r"(b));
}

// A ring position: slot index and the parity of its current use.
struct Ring {
    int slot, n;
    uint32_t phase;
    __device__ __forceinline__ explicit Ring(int n_) : slot(0), n(n_), phase(0) {}
    __device__ __forceinline__ void next() { if (++slot == n) { slot = 0; phase ^= 1; } }
};

template <int TYPE, int MH>
__global__ void __launch_bounds__(tc_threads<MH>(), 1) rq_tc_kernel(const __grid_constant__ TcParams p) {
    using F = Format<TYPE>;
    constexpr int kGroups = Shape<MH>::groups, kStageFirst = kDrainWarps, kMiscFirst = kDrainWarps + 4 * kGroups, kCols = Shape<MH>::cols;
    constexpr int kHalves = F::halves, kMinSlices = TYPE == RQ_Q4_K ? 2 : 0;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // swizzled tiles want 1024-byte alignment
    // A STEP is one sum that leaves tensor memory: (slice, row half, half slice), numbered in issue order. Its one commit arrives on
    // done[step % kDone]: the drain warps wait for it (the sum is complete), the staging warps for the last step that read their
    // operand slot, the activation copies for the last step that read theirs. Indexing by step keeps every parity wait within one
    // phase: the issuing thread is never kDone steps ahead of anyone (slots x steps per slot < kDone).
    __shared__ __align__(8) uint64_t done[kDone], raw_full[kMaxRaw], raw_empty[kMaxRaw], b_full[kMaxB], a_full[kMaxA], acc_empty[kMaxAcc];
    __shared__ uint32_t tmem_base_slot;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // visibly the same for the whole warp: the compiler budgets registers by role only then
    const int bn = p.bn, b_bytes = bn * 256, a_slots = p.a_slots, accs = p.accs;
    const int acc_cols = MH == 1 ? 2 * bn : bn;
    uint8_t* raw = smem + (size_t)p.b_slots * b_bytes;

    if (tid == 0) {
        for (int s = 0; s < kDone; ++s) mbar_init(&done[s], 1);
        for (int s = 0; s < kMaxRaw; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_empty[s], 4 * F::raw_slices); }
        for (int s = 0; s < kMaxB; ++s) mbar_init(&b_full[s], 1);
        for (int s = 0; s < kMaxA; ++s) mbar_init(&a_full[s], 4);
        for (int s = 0; s < kMaxAcc; ++s) mbar_init(&acc_empty[s], kDrainWarps);
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
    const uint32_t tmem_base = tmem_base_slot, a_ring = tmem_base + 512u - (uint32_t)(a_slots * F::a_cols);
    Walk walk(p.whole, p.rest_tiles, p.units);
    int tile, u0, u1;

    if (warp < kDrainWarps) {
        // ------------------------------------------------------------ drain warps
        // launched with 96 registers a thread (MH = 2: 640 x 96 = 61440 in all): drain 256 x 152 + staging 256 x 64 + the rest 128 x 48
        // = 61440 as well
        if (MH == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
        // warp w may read accumulator rows 32 (w % 4) ..; warps 0-3 take the first half of the tile's tokens, warps 4-7 the second
        const int quarter = warp & 3, tokens_here = bn >> 1, col0 = (warp >> 2) * tokens_here;
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        int step = 0;
        Ring acc_at(accs);
        bool dead = false;
        while (walk.next(tile, u0, u1)) {
            const int mt = tile % p.tiles_m, nt = tile / p.tiles_m;
            float sum[MH][kCols];
            // this lane's row of half m, kept inside the weight for the scale loads (at most 2^31 rows)
            auto row_of = [&](int m) -> int64_t { return min((uint32_t)(mt * MH + m) * 128u + (uint32_t)(quarter * 32 + lane), (uint32_t)(p.rows - 1)); };
#pragma unroll
            for (int m = 0; m < MH; ++m) {
#pragma unroll
                for (int i = 0; i < kCols; ++i) sum[m][i] = 0.f;
            }
            auto drain = [&](int m, float d) {
                if (!dead && !mbar_wait_warp(&done[step % kDone], (step / kDone) & 1, p.wait_ns)) { atomicExch(p.error_flag, 14); dead = true; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t at = tmem_base + lane_base + (uint32_t)(acc_at.slot * acc_cols + col0);
                if (MH == 1) {
#pragma unroll
                    for (int c = 0; c < kCols; c += 8) {
                        if (c < tokens_here) {
                            uint32_t h[8], l[8];
                            tmem_ld8_pair(at + c, at + bn + c, h, l);
#pragma unroll
                            for (int j = 0; j < 8; ++j) sum[m][c + j] = fmaf(d, __uint_as_float(h[j]) + __uint_as_float(l[j]), sum[m][c + j]);
                        }
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < kCols; c += 16) {
                        if (c < tokens_here) {
                            uint32_t t[16];
                            tmem_ld16(at + c, t);
#pragma unroll
                            for (int j = 0; j < 16; ++j) sum[m][c + j] = fmaf(d, __uint_as_float(t[j]), sum[m][c + j]);
                        }
                    }
                }
                // this warp has read the accumulator: the tensor core may overwrite it
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[acc_at.slot]);
                ++step;
                acc_at.next();
            };
            if constexpr (F::kquant) {
                auto d_of = [&](int m, int u) -> float {
                    if (TYPE == RQ_Q4_K) return rq_h2f(__ldg((const uint16_t*)(p.main + (row_of(m) * p.units + u) * 144)));
                    return rq_h2f(__ldg(p.scale + row_of(m) * p.units + u));
                };
                float d[MH], d_next[MH];
#pragma unroll
                for (int m = 0; m < MH; ++m) d_next[m] = d_of(m, u0);
                for (int u = u0; u < u1; ++u) {
#pragma unroll
                    for (int m = 0; m < MH; ++m) { d[m] = d_next[m]; if (u + 1 < u1) d_next[m] = d_of(m, u + 1); }  // the next unit's scale is on its way
#pragma unroll 1
                    for (int sl = 0; sl < 4; ++sl)
#pragma unroll
                        for (int m = 0; m < MH; ++m) drain(m, d[m]);
                }
                if (kMinSlices) {
                    const int extra = kMinSlices * (((u1 - 1) >> 3) - (u0 >> 3) + 1);
#pragma unroll 1
                    for (int e = 0; e < extra; ++e)
#pragma unroll
                        for (int m = 0; m < MH; ++m) drain(m, -kMinUnscale);
                }
            } else {
                // eight fp16 scales per unit; one word (two blocks: a slice) at a time, the next on its way
                auto d_of = [&](int m, int b) -> uint32_t {  // b: an even block; rows of an odd number of blocks are only 2-byte aligned
                    const uint16_t* at = p.scale + row_of(m) * p.blocks32;
                    const uint32_t lo = b < p.blocks32 ? __ldg(at + b) : 0u, hi = b + 1 < p.blocks32 ? __ldg(at + b + 1) : 0u;
                    return lo | (hi << 16);
                };
                uint32_t d[MH], d_next[MH];
#pragma unroll
                for (int m = 0; m < MH; ++m) d_next[m] = d_of(m, 8 * u0);
#pragma unroll 1
                for (int s = 4 * u0; s < 4 * u1; ++s) {
#pragma unroll
                    for (int m = 0; m < MH; ++m) { d[m] = d_next[m]; if (s + 1 < 4 * u1) d_next[m] = d_of(m, 2 * s + 2); }
#pragma unroll
                    for (int m = 0; m < MH; ++m)
#pragma unroll
                        for (int h = 0; h < kHalves; ++h) drain(m, rq_h2f((uint16_t)(h ? d[m] >> 16 : d[m] & 0xffff)));
                }
            }
            const bool whole = u0 == 0 && u1 == p.units;
            float* part = p.partial + (size_t)(2 * blockIdx.x + (u0 == 0 ? 1 : 0)) * bn * 128 * MH;
#pragma unroll
            for (int m = 0; m < MH; ++m) {
                const int r = m * 128 + quarter * 32 + lane;
                const int64_t out_row = (int64_t)mt * MH * 128 + r;
#pragma unroll
                for (int j = 0; j < kCols; ++j) {
                    const int token = nt * bn + col0 + j;
                    if (j < tokens_here && token < p.tokens && out_row < p.rows && !dead) {
                        if (whole) p.y[out_row * p.yn + (int64_t)token * p.yt] = sum[m][j];
                        else part[(size_t)(col0 + j) * 128 * MH + r] = sum[m][j];
                    }
                }
            }
        }
    } else if (warp < kMiscFirst) {
        // ------------------------------------------------------------ staging groups: stored bytes -> integer operands in tensor memory
        if (MH == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
        const int group = (warp - kStageFirst) >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        int a_base = 0, raw_base = 0;  // operand tiles and raw tiles of the segments before this one
        bool dead = false;
        while (walk.next(tile, u0, u1)) {
            const int mt = tile % p.tiles_m;
            const int main_slices = 4 * (u1 - u0), extra = kMinSlices ? kMinSlices * (((u1 - 1) >> 3) - (u0 >> 3) + 1) : 0;
            const int tiles = (main_slices + extra) * MH;
            int first = group - a_base % kGroups;
            if (first < 0) first += kGroups;
#pragma unroll 1
            for (int i = first; i < tiles; i += kGroups) {
                const int ks = i / MH, m = i % MH, a = a_base + i;
                const uint32_t at = a_ring + lane_base + (uint32_t)((a % a_slots) * F::a_cols);
                const int freed = (a - a_slots) * kHalves + kHalves - 1;  // the last step that read the slot
                bool free_slot = a < a_slots;
                auto wait_slot = [&]() {
                    if (!free_slot) {
                        if (!dead && !mbar_wait_warp(&done[freed % kDone], (freed / kDone) & 1, p.wait_ns)) { atomicExch(p.error_flag, 11); dead = true; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        free_slot = true;
                    }
                };
                if (ks < main_slices) {
                    const int rt = raw_base + (ks / F::raw_slices) * MH + m, rslot = rt % p.raw_slots;
                    if (!dead && !mbar_wait_warp(&raw_full[rslot], (rt / p.raw_slots) & 1, p.wait_ns)) { atomicExch(p.error_flag, 18); dead = true; }
                    const uint8_t* src = raw + (size_t)rslot * F::raw_bytes;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t o[16], res[16];
                        unpack32<TYPE>(src, r, u0 + (ks >> 2), ks & 3, half, p.permuted != 0, o, res);
                        wait_slot();
                        tmem_st16(at + 16 * half, o);
                        if (F::residual) tmem_st16(at + 32 + 16 * half, res);
                    }
                    // this warp has read its rows of the slice
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&raw_empty[rslot]);
                } else if (TYPE == RQ_Q4_K) {
                    // the minimum terms of one window's superblocks, hi or lo: chunk j of the operand is superblock 8 w + j (zeros outside u0 .. u1)
                    const int e = ks - main_slices, window = (u0 >> 3) + (e >> 1);
                    const int64_t rr = ((int64_t)mt * MH + m) * 128 + r;
                    const uint8_t* base = p.main + (rr < p.rows ? rr : p.rows - 1) * p.units * 144;
                    wait_slot();
#pragma unroll 1
                    for (int q = 0; q < 2; ++q) {
                        uint32_t o[16];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int u = 8 * window + 4 * q + j;
                            const bool in = u >= u0 && u < u1;
                            const uint4 hdr = in ? __ldg((const uint4*)(base + (int64_t)u * 144)) : make_uint4(0, 0, 0, 0);
                            minimum_terms(hdr, (e & 1) != 0, o + 4 * j);
                        }
                        tmem_st16(at + 16 * q, o);
                    }
                }
                tmem_st_wait();
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&a_full[a % a_slots]);  // one arrival per warp (an arrival is an atomic on the barrier)
            }
            a_base += tiles;
            raw_base += main_slices / F::raw_slices * MH;
        }
    } else {
        if (MH == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
        if (warp == kMiscFirst && elect_one()) {
            // ------------------------------------------------------------ the issuing thread
            const uint32_t idesc = instr_desc(bn), idesc2 = instr_desc(MH == 1 ? 2 * bn : bn);
            Ring a_at(a_slots), b_at(p.b_slots), acc_at(accs);
            int step = 0;
            bool dead = false;
            while (walk.next(tile, u0, u1)) {
                const int slices = 4 * (u1 - u0) + (kMinSlices ? kMinSlices * (((u1 - 1) >> 3) - (u0 >> 3) + 1) : 0);
#pragma unroll 1
                for (int ks = 0; ks < slices; ++ks) {
                    if (!dead && !mbar_wait(&b_full[b_at.slot], b_at.phase, p.wait_ns)) { atomicExch(p.error_flag, 17); dead = true; }
                    const uint32_t bbase = smem_u32(smem + (size_t)b_at.slot * b_bytes);
                    const uint64_t b_hi = smem_desc(bbase), b_lo = smem_desc(bbase + bn * 128);
#pragma unroll 1
                    for (int m = 0; m < MH; ++m) {
                        if (!dead && !mbar_wait(&a_full[a_at.slot], a_at.phase, p.wait_ns)) { atomicExch(p.error_flag, 13); dead = true; }
                        const uint32_t a_hi = a_ring + (uint32_t)(a_at.slot * F::a_cols), a_res = a_hi + 32;
#pragma unroll
                        for (int h = 0; h < kHalves; ++h) {
                            if (step >= accs && !dead && !mbar_wait(&acc_empty[acc_at.slot], acc_at.phase ^ 1, p.wait_ns)) { atomicExch(p.error_flag, 15); dead = true; }
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            if (!dead) {
                                const uint32_t acc = tmem_base + (uint32_t)(acc_at.slot * acc_cols);
                                constexpr int kk_n = 4 / kHalves;
                                // kk: 16-wide steps, 32 bytes along K (in 16-byte units of the descriptor's start address), eight columns of A
                                if (MH == 1) {
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
                                // one commit: the sum is complete and, after the last step that reads them, the operand and activation slots are free
                                mma_commit(&done[step % kDone]);
                            }
                            ++step;
                            acc_at.next();
                        }
                        a_at.next();
                    }
                    b_at.next();
                }
            }
            // nothing may be in flight when tensor memory is freed: the drain warps have waited for every step by then
        } else if (warp == kMiscFirst + 1 && elect_one()) {
            // ------------------------------------------------------------ activation copies (the images were written by the kernel before this one)
            asm volatile("griddepcontrol.wait;" ::: "memory");
            Ring b_at(p.b_slots);
            int ks_all = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const uint8_t* src = p.xs + (size_t)(tile / p.tiles_m) * p.image_tiles * b_bytes;
                const int main_slices = 4 * (u1 - u0), extra = kMinSlices ? kMinSlices * (((u1 - 1) >> 3) - (u0 >> 3) + 1) : 0;
                for (int ks = 0; ks < main_slices + extra; ++ks, ++ks_all) {
                    const int freed = (ks_all - p.b_slots + 1) * MH * kHalves - 1;  // the last step that read the slot
                    if (ks_all >= p.b_slots && !mbar_wait(&done[freed % kDone], (freed / kDone) & 1, p.wait_ns)) { atomicExch(p.error_flag, 16); dead = true; break; }
                    const int image = ks < main_slices ? 4 * u0 + ks : 4 * p.units + (u0 >> 3) + ((ks - main_slices) >> 1);
                    mbar_expect_tx(&b_full[b_at.slot], (uint32_t)b_bytes);
                    bulk_g2s(smem + (size_t)b_at.slot * b_bytes, src + (size_t)image * b_bytes, (uint32_t)b_bytes, &b_full[b_at.slot]);
                    b_at.next();
                }
            }
        } else if (warp == kMiscFirst + 2 && elect_one()) {
            // ------------------------------------------------------------ stored bytes: constants of the model, nothing to wait for before the first fetches
            Ring at(p.raw_slots);
            int n = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const int mt = tile % p.tiles_m;
                constexpr int kPer = 4 / F::raw_slices;  // TMA tiles per unit and row half
                for (int t = u0 * kPer; t < u1 * kPer && !dead; ++t)
                    for (int m = 0; m < MH; ++m, ++n) {
                        if (n >= p.raw_slots && !mbar_wait(&raw_empty[at.slot], at.phase ^ 1, p.wait_ns)) { atomicExch(p.error_flag, 19); dead = true; break; }
                        mbar_expect_tx(&raw_full[at.slot], F::raw_bytes);
                        tma_load_2d(raw + (size_t)at.slot * F::raw_bytes, &p.tile_map, t * F::box_bytes, (mt * MH + m) * 128, &raw_full[at.slot]);
                        at.next();
                    }
            }
        }
        __syncwarp();
    }
    // free the tensor memory: everyone is past its use
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMiscFirst) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

// Adds up the tiles that several CTAs share, in unit order. grid (token lanes, shared tiles): a thread takes one row of a tile and
// every gridDim.x-th token of it.
template <int MH>
__global__ void __launch_bounds__(128 * MH) rq_tc_sum_kernel(const float* __restrict__ partial, int ctas, int first_tile, int rest_tiles, int units, int tiles_m, int bn, int tokens, int64_t rows,
                                                              float* __restrict__ y, int64_t yn, int64_t yt) {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int t = blockIdx.y, tile = first_tile + t, mt = tile % tiles_m, nt = tile / tiles_m;
    const int64_t total = (int64_t)rest_tiles * units, begin = (int64_t)t * units, end = begin + units;
    int c0 = (int)(begin * ctas / total);
    while (c0 > 0 && c0 * total / ctas > begin) --c0;
    while ((c0 + 1) * total / ctas <= begin) ++c0;
    if ((c0 + 1) * total / ctas >= end && c0 * total / ctas <= begin) return;  // one CTA had the whole tile and wrote it
    const int64_t out_row = (int64_t)mt * 128 * MH + threadIdx.x;
    if (out_row >= rows) return;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    for (int j = blockIdx.x; j < bn && nt * bn + j < tokens; j += gridDim.x) {
        float s = 0.f;
        for (int c = c0; c < ctas; ++c) {
            const int64_t lo = c * total / ctas, hi = (c + 1) * total / ctas;
            if (lo >= end) break;
            if (hi <= begin || hi == lo) continue;
            const int slot = 2 * c + (lo > begin ? 0 : 1);
            s += __ldcg(partial + ((size_t)slot * bn + j) * 128 * MH + threadIdx.x);
        }
        y[out_row * yn + (int64_t)(nt * bn + j) * yt] = s;
    }
}

template <int TYPE, int MH>
int launch_tc(const TcParams& p, int ctas, size_t smem, cudaStream_t s) {
    auto kernel = rq_tc_kernel<TYPE, MH>;
    static bool configured[64] = {};
    int dev = 0;
    RQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        RQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 225 * 1024));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(tc_threads<MH>());
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
int launch_tc(const TcParams& p, int mh, int ctas, size_t smem, cudaStream_t s) {
    return mh == 1 ? launch_tc<TYPE, 1>(p, ctas, smem, s) : launch_tc<TYPE, 2>(p, ctas, smem, s);
}

// How a call is cut: row halves and tokens per tile, CTAs, ring depths, shared memory and scratch.
struct TcCut {
    int mh, bn, n_tiles, tiles_m, units, image_tiles, windows, ctas, whole, rest_tiles;
    int raw_slots, b_slots, a_slots, accs;
    size_t smem, xs_bytes, partial_bytes;
};
struct FormatSizes { int raw_bytes, a_cols, raw_per_unit; };
FormatSizes format_sizes(int type) {
    switch (type) {
        case RQ_Q4_K: return {Format<RQ_Q4_K>::raw_bytes, Format<RQ_Q4_K>::a_cols, 1};
        case RQ_Q6_K: return {Format<RQ_Q6_K>::raw_bytes, Format<RQ_Q6_K>::a_cols, 1};
        case RQ_Q8_0: return {Format<RQ_Q8_0>::raw_bytes, Format<RQ_Q8_0>::a_cols, 2};
        default: return {Format<RQ_Q4_0>::raw_bytes, Format<RQ_Q4_0>::a_cols, 1};
    }
}
TcCut tc_cut(int type, int sm_count, int64_t rows, int64_t cols, int tokens) {
    TcCut c;
    const FormatSizes f = format_sizes(type);
    c.mh = tokens <= 64 ? 1 : 2;
    const int widest = 2 * (c.mh == 1 ? Shape<1>::cols : Shape<2>::cols), grain = c.mh == 1 ? 16 : 32;
    c.n_tiles = (tokens + widest - 1) / widest;
    c.bn = ((tokens + c.n_tiles - 1) / c.n_tiles + grain - 1) / grain * grain;
    c.tiles_m = (int)((rows + 128 * c.mh - 1) / (128 * c.mh));
    c.units = (int)((cols + 255) / 256);
    c.windows = type == RQ_Q4_K ? (c.units + 7) / 8 : 0;
    c.image_tiles = 4 * c.units + c.windows;
    const int64_t tiles = (int64_t)c.tiles_m * c.n_tiles, work = tiles * c.units;
    c.ctas = work < sm_count ? (int)work : sm_count;
    c.whole = (int)(tiles / c.ctas);
    c.rest_tiles = (int)(tiles - (int64_t)c.whole * c.ctas);
    // tensor memory, 512 columns: operand slots, the rest accumulators
    c.a_slots = type == RQ_Q6_K ? (c.mh == 1 ? 4 : 2) : 4;
    const int acc_cols = c.mh == 1 ? 2 * c.bn : c.bn;
    c.accs = (512 - c.a_slots * f.a_cols) / acc_cols;
    if (c.accs > kMaxAcc) c.accs = kMaxAcc;
    // shared memory: activation slots, then as many slots of stored bytes as fit
    const int budget = 220 * 1024, b_bytes = c.bn * 256;
    c.b_slots = c.mh == 1 ? 4 : 3;
    c.raw_slots = (budget - c.b_slots * b_bytes) / f.raw_bytes;
    const int raw_max = c.mh * 2 * f.raw_per_unit < kMaxRaw ? 6 : kMaxRaw;
    if (c.raw_slots > raw_max) c.raw_slots = raw_max;
    while (c.b_slots < 6 && (c.b_slots + 1) * b_bytes + c.raw_slots * f.raw_bytes <= budget) ++c.b_slots;
    c.smem = (size_t)c.b_slots * b_bytes + (size_t)c.raw_slots * f.raw_bytes + 1024;
    c.xs_bytes = (size_t)c.n_tiles * c.image_tiles * b_bytes;
    c.partial_bytes = c.rest_tiles ? (size_t)2 * c.ctas * c.bn * 128 * c.mh * 4 : 0;
    return c;
}

}  // namespace

// Enough for every call of up to this many rows, inputs and tokens, of any format: token tiles are padded by less than 32 rows
// each, and the shared tiles' sums are two tiles a CTA.
size_t rq_matmul_scratch_bytes(const rq_ctx* ctx, int64_t rows, int64_t cols, int tokens) {
    const int64_t units = (cols + 255) / 256, tiles_n = (tokens + 95) / 96;
    const size_t image = (size_t)(tokens + 32 * tiles_n + 32) * 256 * (size_t)(4 * units + (units + 7) / 8);
    const int64_t work = ((rows + 127) / 128) * units * (tiles_n < 1 ? 1 : tiles_n);
    const size_t ctas = (size_t)(work < ctx->sm_count ? work : ctx->sm_count);
    return image + 256 + 2 * ctas * (tokens > 64 ? 96 * 256 : 64 * 128) * 4;
}

// RQ_ERR_UNSUPPORTED (no error text) = not one of the four formats. act_mode FLOAT or INT8 (step 32 / 256).
int rq_launch_matmul(rq_ctx* ctx, const rq_weight* w, const float* x, int64_t sk, int64_t st, int tokens, float* y, int64_t yn, int64_t yt, int act_mode, int step, cudaStream_t s) {
    if (!w->has_tile_map || !rq_type_has_fast_path(w->type)) return RQ_ERR_UNSUPPORTED;
    const TcCut cut = tc_cut(w->type, ctx->sm_count, w->rows, w->cols, tokens);
    int rc = rq_ensure_act_scratch(ctx, cut.xs_bytes + cut.partial_bytes, s);
    if (rc) return rc;
    ctx->act_cols = 0;  // whatever int8 records the scratch held for INT8_CACHED calls are gone
    uint8_t* xs = ctx->act_scratch;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    {
        const int padded = cut.n_tiles * cut.bn;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)cut.units, (unsigned)((padded + 7) / 8));
        cfg.blockDim = dim3(256);
        cfg.stream = s;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        auto prep = act_mode == RQ_ACT_FLOAT ? rq_tc_prep_kernel<0> : (step == 256 ? rq_tc_prep_kernel<256> : rq_tc_prep_kernel<32>);
        RQ_CUDA(cudaLaunchKernelEx(&cfg, prep, x, sk, st, (int)w->cols, cut.units, tokens, cut.bn, padded, cut.image_tiles, cut.windows, xs));
    }
    TcParams p;
    p.tile_map = w->tile_map;
    p.main = w->main; p.scale = w->scale; p.rows = w->rows;
    p.blocks32 = (int)(w->cols / 32); p.units = cut.units; p.permuted = rq_plane_permuted(w->type, w->cols) ? 1 : 0;
    p.xs = xs; p.image_tiles = cut.image_tiles; p.bn = cut.bn; p.tokens = tokens; p.y = y; p.yn = yn; p.yt = yt;
    p.tiles_m = cut.tiles_m; p.whole = cut.whole; p.rest_tiles = cut.rest_tiles;
    p.partial = (float*)(xs + cut.xs_bytes);
    p.raw_slots = cut.raw_slots; p.b_slots = cut.b_slots; p.a_slots = cut.a_slots; p.accs = cut.accs;
    p.error_flag = ctx->error_flag; p.wait_ns = ctx->wait_limit_ns;
    switch (w->type) {
        case RQ_Q4_K: rc = launch_tc<RQ_Q4_K>(p, cut.mh, cut.ctas, cut.smem, s); break;
        case RQ_Q6_K: rc = launch_tc<RQ_Q6_K>(p, cut.mh, cut.ctas, cut.smem, s); break;
        case RQ_Q8_0: rc = launch_tc<RQ_Q8_0>(p, cut.mh, cut.ctas, cut.smem, s); break;
        default: rc = launch_tc<RQ_Q4_0>(p, cut.mh, cut.ctas, cut.smem, s); break;
    }
    if (rc || !cut.rest_tiles) return rc;
    cudaLaunchConfig_t cfg = {};
    const int lanes = cut.bn < 32 ? cut.bn : 32;
    cfg.gridDim = dim3((unsigned)lanes, (unsigned)cut.rest_tiles);
    cfg.blockDim = dim3((unsigned)(128 * cut.mh));
    cfg.stream = s;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RQ_CUDA(cudaLaunchKernelEx(&cfg, cut.mh == 1 ? rq_tc_sum_kernel<1> : rq_tc_sum_kernel<2>, (const float*)p.partial, cut.ctas, cut.whole * cut.ctas, cut.rest_tiles, cut.units, cut.tiles_m,
                               cut.bn, tokens, w->rows, y, yn, yt));
    return RQ_OK;
}
