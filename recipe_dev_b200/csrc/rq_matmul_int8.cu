// Batched product of int8 activations over Q8_0 and Q4_0, more than 64 tokens: the codes of both sides meet in the 5th-generation tensor
// cores' 8-bit integer products.
//
//   Y[t][n] = sum_g d[n][g] * s[t][g] * (sum over the group's 32 inputs of code[n][k] * code[t][k])
//
// A group of 32 inputs is one tcgen05.mma (kind::i8, K = 32): its sum is an exact 32-bit integer that both scales meet on its way out
// of tensor memory. Q8_0's stored bytes ARE the operand: the tile that TMA lands with the 128-byte swizzle is the K-major operand that the
// product reads, in the stored order of its 16-byte chunks (a permutation that the activations' image repeats). Q4_0's nibbles become bytes by
// one or two logic operations a word (in the high half of a byte, less eight by turning its top bit: sixteen times the code, which d / 16 undoes).
// So no warp unpacks Q8_0 and little is unpacked of Q4_0, and the kernel is what its drain warps need for a sum:
// a conversion, and a product of the two scales and a multiply-add, two sums an instruction.
//
// One CTA per SM, persistent, over tiles of 256 rows x 64 tokens, dealt as in rq_matmul_tc.cu (rq_matmul_cut.cuh). Roles: three copying warps
// (stored bytes; activations and their steps; stored scales), one issuing warp, Q4_0: four staging warps (nibbles -> operands in shared memory),
// sixteen drain warps. A drain thread holds two rows (one of each row half) of sixteen tokens: a step read from shared memory, 128 bytes a cycle
// like everything from there, serves two sums. All of tensor memory is accumulators: two stages of a 64-wide slice (two groups x two row
// halves x 64 columns), one filled while the other is drained. The scales come through shared memory because a drain thread that loads them
// ahead into registers waits for them where the branch for ragged widths ends (a fifth of the time).
//
// What bounds it: instructions and the fp32 pipe. A sum is a conversion (the ALU, half rate), half a product of scales and half a multiply-add (two
// sums an instruction, two cycles each); a warp alone with another one on its scheduler takes 39 cycles for sixteen of them, 35 where four share it, and of
// 1500 cycles a slice and scheduler that is 560; the rest is totals (180), barriers, scales and the instructions that find their place, issued in 65 % of the cycles. Measured
// on one B200, calls back to back, the form before (codes as fp16, unpacked into tensor memory by eight warps) and now: Q8_0 4096 x 14336
// 509 tokens 279 -> 198 us, 14336 x 4096 65 tokens 88.5 -> 64.6, 2000 x 1536 128 tokens 22.4 -> 18.2; Q4_0 277 -> 230, 87.3 -> 75.0, 22.2 -> 20.5; 72 calls
// of 65 to 509 tokens 0.70 to 0.94. Not kept: eight drain warps (205 us for 198), accumulators that start as 1.5 * 2^23 so that a subtraction
// of two numbers does for the conversions (265 where conversions took 228: the stores to tensor memory), scalar multiply-adds (278 for 222).
//
// Every wait is bounded, and before the CTA frees its tensor memory and exits the issuing and copying warps wait once more, within the
// same limit, for the products and copies that they have under way.
#include "rq_internal.cuh"
#include "rq_matmul_cut.cuh"
#include "rq_matmul_int8.cuh"
#include "rq_mma.cuh"
#include "rq_pairs.cuh"

using namespace rqmma;
using namespace rqcut;

namespace {

constexpr int kTokens = kInt8Tokens, kTile = 128 * 128;  // tokens of a tile; bytes of 128 rows x 128 inputs
constexpr int kDrainWarps = kInt8DrainWarps, kStages = kInt8Stages;
template <int TYPE> __host__ __device__ constexpr int staging_warps() { return TYPE == RQ_Q4_0 ? 4 : 0; }
template <int TYPE> __host__ __device__ constexpr int int8_threads() { return (kDrainWarps + staging_warps<TYPE>() + 4) * 32; }
template <int TYPE> struct Regs;  // of the launch's 640 x 96 and 768 x 80 (the kernels spill 68 and 166 bytes a thread)
template <> struct Regs<RQ_Q8_0> { static constexpr int drain = 112, other = 32; };
template <> struct Regs<RQ_Q4_0> { static constexpr int drain = 96, other = 40; };

// kind::i8, signed x signed -> 32-bit integers, both operands K-major, M = 128, N = 64
__device__ __forceinline__ uint32_t instr_desc_i8() { return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTokens >> 3) << 17) | ((uint32_t)(BM >> 4) << 24); }
// D[tensor memory] = A[shared memory] x B[shared memory], 32 bytes along K
__device__ __forceinline__ void mma_i8_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(0u)
        : "memory");
}
// Sixteen columns of this warp's 32 lanes, asked for; two such are there behind tmem_landed (which has them as operands so that nothing that uses
// them moves ahead of it).
__device__ __forceinline__ void tmem_ask(uint32_t a, uint32_t (&v)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]),
                   "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(a));
}
__device__ __forceinline__ void tmem_landed(uint32_t (&u)[16], uint32_t (&v)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]), "+r"(u[8]), "+r"(u[9]), "+r"(u[10]), "+r"(u[11]), "+r"(u[12]),
                   "+r"(u[13]), "+r"(u[14]), "+r"(u[15]), "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7]), "+r"(v[8]), "+r"(v[9]),
                   "+r"(v[10]), "+r"(v[11]), "+r"(v[12]), "+r"(v[13]), "+r"(v[14]), "+r"(v[15]));
}

template <int TYPE>
__global__ void __launch_bounds__(int8_threads<TYPE>(), 1) rq_tc_int8_kernel(const __grid_constant__ RqInt8Params p) {
    using R = Int8Rings<TYPE>;
    constexpr bool kStaged = TYPE == RQ_Q4_0;
    constexpr int kRaw = kStaged ? R::raw_slots : 1, kScaleSlot = R::scale_bytes;
    static_assert(R::half_bytes == kTile && R::b_bytes == kTokens * 128, "the rings' slots are what the copies fill");
    constexpr int kStaging = staging_warps<TYPE>(), kMiscFirst = kDrainWarps + kStaging;
    static_assert(32 * kDrainWarps * Regs<TYPE>::drain + 32 * (kStaging + 4) * Regs<TYPE>::other <= int8_threads<TYPE>() * (65536 / int8_threads<TYPE>() / 8 * 8), "more registers than the launch has: the increase would wait forever");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);  // swizzled tiles want 1024-byte alignment
    uint8_t* const b_ring = smem;                                      // [slot][64 tokens x 128 inputs]
    uint8_t* const a_ring = b_ring + R::b_slots * (kTokens * 128);     // [slot][row half][128 rows x 128 inputs]
    uint8_t* const raw = a_ring + R::a_slots * 2 * kTile;              // Q4_0: [slot][128 rows x 256 inputs]
    const int tid = threadIdx.x, lane = tid & 31;
    // [slot]: what scales a unit's sums, steps [8 groups][64 tokens], then the weight's eight fp16 scales [256 rows]
    uint8_t* const scales = raw + R::raw_slots * kTile;
    ulonglong2* const totals = (ulonglong2*)(scales + R::scale_slots * kScaleSlot) + tid;  // a drain thread's own: [row half][four tokens][256 threads]
    // stages: done = a slice's products are complete, drained = the drain warps have read them. a: operands (Q8_0: as landed), b: activations,
    // freed by the commit behind the last slice that reads them.
    __shared__ __align__(8) uint64_t done[kStages], drained[kStages], a_full[R::a_slots], a_free[R::a_slots], b_full[R::b_slots], b_free[R::b_slots];
    __shared__ __align__(8) uint64_t raw_full[kRaw], raw_free[kRaw], scales_full[R::scale_slots], scales_free[R::scale_slots], ended;
    __shared__ uint32_t tmem_base_slot;
    __shared__ int last_piece;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // visibly the same for the whole warp: the compiler budgets registers by role only then

    if (tid == 0) {
        for (int s = 0; s < kStages; ++s) { mbar_init(&done[s], 1); mbar_init(&drained[s], kDrainWarps); }
        for (int s = 0; s < R::a_slots; ++s) { mbar_init(&a_full[s], kStaged ? 2 * kStaging : 1); mbar_init(&a_free[s], 1); }
        for (int s = 0; s < R::b_slots; ++s) { mbar_init(&b_full[s], 1); mbar_init(&b_free[s], 1); }
        for (int s = 0; s < kRaw; ++s) { mbar_init(&raw_full[s], 1); mbar_init(&raw_free[s], 4); }
        for (int s = 0; s < R::scale_slots; ++s) { mbar_init(&scales_full[s], 33); mbar_init(&scales_free[s], kDrainWarps); }
        mbar_init(&ended, 1);
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
    const uint32_t tmem_base = tmem_base_slot;
    Walk walk(p.whole, p.rest_tiles, p.units, p.share, (int)gridDim.x, (int)blockIdx.x);
    int tile, u0, u1;

    if (warp < kDrainWarps) {
        // ------------------------------------------------------------ drain warps
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Regs<TYPE>::drain));
        constexpr int kMine = kTokens / 4;
        const int quarter = warp & 3, col0 = (warp >> 2) * kMine, r0 = quarter * 32 + lane;
        const uint32_t acc0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)col0;
        Ring scale_at(R::scale_slots);
        uint32_t phase = 0;  // of the stages, one half unit after another
        bool dead = false;
        while (walk.next(tile, u0, u1)) {
            const int mt = tile % p.tiles_m, nt = tile / p.tiles_m;
            const bool whole = u0 == 0 && u1 == p.units;
            const int t = tile - p.whole * (int)gridDim.x;
            int c0 = 0, c1 = 0;
            if (!whole) {
                const Deal deal(p.share, p.rest_tiles, p.units);
                c0 = deal.first(t);
                c1 = deal.last(t, (int)blockIdx.x);
            }
            // The products are exact, so what a sum loses it loses where its terms (a group each) are added up. After every unit (half a unit where there
            // are few) the sums go into totals, and what that addition rounds off stays behind as the start of the next run. Error
            // against 64 bits, random terms of 448 groups: 3.8e-7 in one chain, 1.3e-7 with plain totals, 0.66e-7 so, the matvec kernel's tree 0.86e-7.
            Pair sum[2][kMine / 2];
            bool flushed = false;
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int i = 0; i < kMine / 2; ++i) sum[m][i] = 0;
            const bool often = u1 - u0 <= 16;
            const Pair minus = pair_of(-1.0f, -1.0f);
            auto flush = [&]() {
                Pair lost = 0;
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int i = 0; i < kMine / 2; i += 2) {
                        ulonglong2& at = totals[(m * (kMine / 4) + i / 2) * (32 * kDrainWarps)];
                        const ulonglong2 total = flushed ? at : make_ulonglong2(0, 0);
                        const Pair next[2] = {pair_add(total.x, sum[m][i]), pair_add(total.y, sum[m][i + 1])};
                        at = make_ulonglong2(next[0], next[1]);
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            sum[m][i + k] = pair_fma(minus, pair_fma(minus, k ? total.y : total.x, next[k]), sum[m][i + k]);
                            lost = pair_add(lost, sum[m][i + k]);
                        }
                    }
                flushed = true;
                // an infinite total has no rounding error to carry on
                if (!(fabsf(pair_at(lost, 0) + pair_at(lost, 1)) <= 3.402823466e38f)) {
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int i = 0; i < kMine / 2; ++i) {
                            const float e0 = pair_at(sum[m][i], 0), e1 = pair_at(sum[m][i], 1);
                            sum[m][i] = pair_of(fabsf(e0) <= 3.402823466e38f ? e0 : 0.f, fabsf(e1) <= 3.402823466e38f ? e1 : 0.f);
                        }
                }
            };
#pragma unroll 1
            for (int u = u0; u < u1; ++u, scale_at.next()) {
                if (!mbar_wait_warp(&scales_full[scale_at.slot], scale_at.phase, p.wait_ns, dead)) atomicExch(p.error_flag, 26);
                const uint8_t* const mine = scales + scale_at.slot * kScaleSlot;
                const float* const steps = (const float*)mine + col0;
                const uint32_t* const d = (const uint32_t*)(mine + R::step_bytes) + 4 * r0;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int sl = 0; sl < 2; ++sl) {
                        static_assert(kStages == 2, "a half unit's slices take the stages in turn");
                        const uint32_t w[2] = {d[2 * h + sl], d[512 + 2 * h + sl]};
                        // a group's sixteen columns of both rows at a time; the first group's steps are asked for before the wait
                        constexpr int kItems = 2 * kMine / 16;
                        const uint32_t acc = acc0 + (uint32_t)(sl * 256);
                        const float* const st = steps + (4 * h + 2 * sl) * kTokens;
                        uint32_t v[2][16];
                        float4 s4[4];
                        auto steps_of = [&](int i) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) s4[k] = *(const float4*)(st + i * kTokens + 4 * k);
                        };
                        steps_of(0);
                        if (!mbar_wait_warp(&done[sl], phase, p.wait_ns, dead)) atomicExch(p.error_flag, 14);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                        for (int i = 0; i < kItems; ++i) {
                            tmem_ask(acc + (uint32_t)(i * 128), v[0]);
                            tmem_ask(acc + (uint32_t)(i * 128) + kTokens, v[1]);
                            if (i) steps_of(i);
                            tmem_landed(v[0], v[1]);
                            if (i + 1 == kItems) {  // the slice is in registers: its stage may be filled again
                                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                                __syncwarp();
                                if (lane == 0) mbar_arrive(&drained[sl]);
                            }
                            const float k = kStaged ? 0.0625f : 1.0f, d0 = k * rq_h2f((uint16_t)(w[0] >> (16 * i))), d1 = k * rq_h2f((uint16_t)(w[1] >> (16 * i)));
                            const Pair scale[2] = {pair_of(d0, d0), pair_of(d1, d1)};
#pragma unroll
                            for (int j = 0; j < 16; j += 4) {
                                const float4 sj = s4[j / 4];
                                const Pair sv[2] = {pair_of(sj.x, sj.y), pair_of(sj.z, sj.w)};
#pragma unroll
                                for (int m = 0; m < 2; ++m)
#pragma unroll
                                    for (int q = 0; q < 2; ++q) {
                                        const uint32_t* t = v[m] + j + 2 * q;
                                        Pair& to = sum[m][j / 2 + q];
                                        to = pair_fma(pair_mul(sv[q], scale[m]), pair_of((float)(int)t[0], (float)(int)t[1]), to);
                                    }
                            }
                        }
                    }
                    phase ^= 1;
                    if (h || often) flush();
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&scales_free[scale_at.slot]);
            }
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int i = 0; i < kMine / 2; i += 2) {
                    const ulonglong2 total = totals[(m * (kMine / 4) + i / 2) * (32 * kDrainWarps)];
                    sum[m][i] = pair_add(total.x, sum[m][i]);
                    sum[m][i + 1] = pair_add(total.y, sum[m][i + 1]);
                }
            const int tokens_here = dead ? 0 : min(kMine, p.tokens - nt * kTokens - col0);
            auto live = [&](int m) { return (int64_t)(mt * 2 + m) * 128 + r0 < p.rows ? tokens_here : 0; };
            auto out = [&](int m) { return p.y + ((int64_t)(mt * 2 + m) * 128 + r0) * p.yn + (int64_t)(nt * kTokens + col0) * p.yt; };
            if (whole) {
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int n = live(m);
                    float* at = out(m);
#pragma unroll
                    for (int j = 0; j < kMine; ++j) {
                        if (j < n) *at = pair_at(sum[m][j / 2], j & 1);
                        at += p.yt;
                    }
                }
            } else {
                // pieces of a shared tile: [token][256 rows]; the last CTA to leave one adds them in unit order (the same bits on every run)
                auto piece_of = [&](int c) { return p.partial + (size_t)Deal::place(c, c0) * (kTokens * 256) + (size_t)col0 * 256 + r0; };
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const int n = live(m);
                    float* at = piece_of((int)blockIdx.x) + 128 * m;
#pragma unroll
                    for (int j = 0; j < kMine; ++j)
                        if (j < n) at[j * 256] = pair_at(sum[m][j / 2], j & 1);
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
                    // two pieces at a time, 64 loads in flight (the padding tokens' places exist and hold nothing that is used)
#pragma unroll 1
                    for (int m = 0; m < 2; ++m) {
                        const int n = live(m);
                        if (n <= 0) continue;
                        Pair all[kMine / 2];
#pragma unroll
                        for (int q = 0; q < kMine / 2; ++q) all[q] = 0;
#pragma unroll 1
                        for (int c = c0; c <= c1; c += 2) {
                            const bool two = c < c1;
                            const float *piece = piece_of(c) + 128 * m, *other = two ? piece_of(c + 1) + 128 * m : piece;
                            float v[kMine], w[kMine];
#pragma unroll
                            for (int q = 0; q < kMine; ++q) {
                                v[q] = __ldcg(piece + q * 256);
                                w[q] = __ldcg(other + q * 256);
                            }
#pragma unroll
                            for (int q = 0; q < kMine; q += 2)
                                all[q / 2] = pair_add(all[q / 2], two ? pair_add(pair_of(v[q], v[q + 1]), pair_of(w[q], w[q + 1])) : pair_of(v[q], v[q + 1]));
                        }
                        float* at = out(m);
#pragma unroll
                        for (int q = 0; q < kMine; ++q) {
                            if (q < n) *at = pair_at(all[q / 2], q & 1);
                            at += p.yt;
                        }
                    }
                }
            }
        }
    } else if (kStaged && warp < kMiscFirst) {
        // ------------------------------------------------------------ Q4_0: stored nibbles -> bytes of sixteen times (code - 8), in operand order
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<TYPE>::other));
        const int r = (warp & 3) * 32 + lane;
        int tiles = 0, halves = 0;
        bool dead = false;
        while (walk.next(tile, u0, u1)) {
#pragma unroll 1
            for (int u = u0; u < u1; ++u, halves += 2, tiles += 2) {
                const int x = p.permuted ? u & 7 : 0;
#pragma unroll 1
                for (int h = 0; h < 2; ++h) {
                    const int half = halves + h, slot = half % R::a_slots;
                    if (half >= R::a_slots && !mbar_wait_warp(&a_free[slot], (half / R::a_slots - 1) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 11);
#pragma unroll 1
                    for (int m = 0; m < 2; ++m) {
                        const int at = (tiles + m) % kRaw;
                        if (!mbar_wait_warp(&raw_full[at], ((tiles + m) / kRaw) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 18);
                        const uint8_t* src = raw + at * kTile;
                        uint8_t* dst = a_ring + (slot * 2 + m) * kTile;
                        uint4 v[4];
#pragma unroll
                        for (int b = 0; b < 4; ++b) v[b] = *(const uint4*)(src + swizzled(r, (4 * h + b) ^ x));
#pragma unroll
                        for (int b = 0; b < 4; ++b) {
                            constexpr uint32_t kHigh = 0xF0F0F0F0u, kTop = 0x80808080u;
                            *(uint4*)(dst + swizzled(r, 2 * b)) = make_uint4(((v[b].x << 4) & kHigh) ^ kTop, ((v[b].y << 4) & kHigh) ^ kTop, ((v[b].z << 4) & kHigh) ^ kTop, ((v[b].w << 4) & kHigh) ^ kTop);
                            *(uint4*)(dst + swizzled(r, 2 * b + 1)) = make_uint4((v[b].x & kHigh) ^ kTop, (v[b].y & kHigh) ^ kTop, (v[b].z & kHigh) ^ kTop, (v[b].w & kHigh) ^ kTop);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the products read what was written here
                        __syncwarp();
                        if (lane == 0) {
                            mbar_arrive(&a_full[slot]);
                            if (h) mbar_arrive(&raw_free[at]);
                        }
                    }
                }
            }
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Regs<TYPE>::other));
        // (these warps wait as a whole and one lane acts: rq_matmul_tc.cu)
        const bool leader = elect_one();
        auto landed = [&](uint64_t* full, int slots, int n) {
            bool dead = false;
            for (int i = max(0, n - slots); i < n && !dead; ++i)
                if (!mbar_wait_warp(&full[i % slots], (i / slots) & 1, p.wait_ns, dead)) atomicExch(p.error_flag, 24);
        };
        if (warp == kMiscFirst) {
            // ------------------------------------------------------------ the issuing warp
            const uint32_t idesc = instr_desc_i8();
            Ring b_at(R::b_slots), a_at(R::a_slots);
            uint32_t phase = 0;
            bool dead = false, first = true;
            while (walk.next(tile, u0, u1)) {
#pragma unroll 1
                for (int u = u0; u < u1; ++u) {
                    const int x = TYPE == RQ_Q8_0 && p.permuted ? (u & 7) >> 1 : 0;  // a group's two chunks lie side by side (in either order, on both sides)
#pragma unroll 1
                    for (int h = 0; h < 2; ++h, b_at.next(), a_at.next(), phase ^= 1, first = false) {
                        if (!mbar_wait_warp(&b_full[b_at.slot], b_at.phase, p.wait_ns, dead)) atomicExch(p.error_flag, 17);
                        if (!mbar_wait_warp(&a_full[a_at.slot], a_at.phase, p.wait_ns, dead)) atomicExch(p.error_flag, 13);
                        const uint64_t b = smem_desc(smem_u32(b_ring + b_at.slot * (kTokens * 128))), a = smem_desc(smem_u32(a_ring + a_at.slot * 2 * kTile));
#pragma unroll
                        for (int sl = 0; sl < 2; ++sl) {
                            if (!first && !mbar_wait_warp(&drained[sl], phase ^ 1, p.wait_ns, dead)) atomicExch(p.error_flag, 15);
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            if (leader && !dead) {
#pragma unroll
                                for (int g = 0; g < 2; ++g) {
                                    const uint32_t at = 2 * ((2 * sl + g) ^ x);  // 32 bytes along K, in the descriptor's units of sixteen
#pragma unroll
                                    for (int m = 0; m < 2; ++m) mma_i8_ss(tmem_base + (uint32_t)(sl * 256 + g * 128 + m * 64), a + m * (kTile >> 4) + at, b + at, idesc);
                                }
                                mma_commit(&done[sl]);
                                if (sl) { mma_commit(&a_free[a_at.slot]); mma_commit(&b_free[b_at.slot]); }
                            }
                            __syncwarp();
                        }
                    }
                }
            }
            // nothing may be in flight when tensor memory is freed
            if (leader) mma_commit(&ended);
            __syncwarp();
            dead = false;
            if (!mbar_wait_warp(&ended, 0, p.wait_ns, dead)) atomicExch(p.error_flag, 23);
        } else if (warp == kMiscFirst + 1) {
            // ------------------------------------------------------------ activation copies (written by the kernel before this one)
            asm volatile("griddepcontrol.wait;" ::: "memory");
            Ring b_at(R::b_slots), scale_at(R::scale_slots);
            int n = 0, units = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const size_t first = (size_t)(tile / p.tiles_m) * p.units;
                for (int u = u0; u < u1 && !dead; ++u) {
                    for (int h = 0; h < 2; ++h) {
                        if (n >= R::b_slots && !mbar_wait_warp(&b_free[b_at.slot], b_at.phase ^ 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 16); break; }
                        if (leader) {
                            mbar_expect_tx(&b_full[b_at.slot], kTokens * 128);
                            bulk_g2s(b_ring + b_at.slot * (kTokens * 128), p.xs + ((first + u) * 2 + h) * (kTokens * 128), kTokens * 128, &b_full[b_at.slot]);
                        }
                        b_at.next();
                        ++n;
                    }
                    if (dead) break;
                    if (units >= R::scale_slots && !mbar_wait_warp(&scales_free[scale_at.slot], scale_at.phase ^ 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 25); break; }
                    if (leader) {
                        mbar_expect_tx(&scales_full[scale_at.slot], R::step_bytes);
                        bulk_g2s(scales + scale_at.slot * kScaleSlot, p.steps + (first + u) * (8 * kTokens), R::step_bytes, &scales_full[scale_at.slot]);
                    }
                    scale_at.next();
                    ++units;
                }
            }
            landed(b_full, R::b_slots, n);
            landed(scales_full, R::scale_slots, units);
        } else if (warp == kMiscFirst + 2) {
            // ------------------------------------------------------------ stored bytes: constants of the model, nothing to wait for before the first fetches
            uint64_t *const full = kStaged ? raw_full : a_full, *const freed = kStaged ? raw_free : a_free;
            constexpr int kSlots = kStaged ? kRaw : R::a_slots, kHalves = kStaged ? 1 : 2;  // Q4_0: a unit of one row half a slot; Q8_0: half a unit of both
            uint8_t* const ring = kStaged ? raw : a_ring;
            Ring at(kSlots);
            int n = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const int row = (tile % p.tiles_m) * 256;
                for (int i = 2 * u0; i < 2 * u1; ++i, ++n, at.next()) {
                    if (n >= kSlots && !mbar_wait_warp(&freed[at.slot], at.phase ^ 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 19); break; }
                    if (leader) {
                        mbar_expect_tx(&full[at.slot], kHalves * kTile);
#pragma unroll
                        for (int m = 0; m < kHalves; ++m)
                            tma_load_2d(ring + (at.slot * kHalves + m) * kTile, &p.tile_map, (kStaged ? i >> 1 : i) * 128, row + (kStaged ? i & 1 : m) * 128, &full[at.slot]);
                    }
                    __syncwarp();
                }
            }
            landed(full, kSlots, n);
        } else {
            // ------------------------------------------------------------ the stored scales: a unit's eight of each row (constants as well)
            const bool wide = (p.blocks32 & 7) == 0 && ((uintptr_t)p.scale & 15) == 0;
            Ring at(R::scale_slots);
            int n = 0;
            bool dead = false;
            while (!dead && walk.next(tile, u0, u1)) {
                const int64_t row0 = (int64_t)(tile % p.tiles_m) * 256 + lane;
                for (int u = u0; u < u1; ++u, ++n, at.next()) {
                    if (n >= R::scale_slots && !mbar_wait_warp(&scales_free[at.slot], at.phase ^ 1, p.wait_ns, dead)) { atomicExch(p.error_flag, 25); break; }
                    uint4* const to = (uint4*)(scales + at.slot * kScaleSlot + R::step_bytes) + lane;
#pragma unroll 1
                    for (int i = 0; i < 256; i += 32) {
                        // (Kept inside the weight. Copies for rows past its last are of no bytes: with the last row's scales in their place every CTA asked for the same
                        // line of L2 all the time. Q4_0 with 2000 tokens, us: 16 x 4096 76.5 -> 47.0, 300 x 4096 80.8 -> 62.4; Q8_0 72.4 -> 41.7, 76.3 -> 54.8. The loads
                        // below find it in L1.)
                        const uint16_t* from = p.scale + min(row0 + i, p.rows - 1) * p.blocks32 + 8 * u;
                        if (wide) {  // rows of whole units
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(to + i)), "l"(from), "r"(row0 + i < p.rows ? 16 : 0) : "memory");
                        } else {
                            uint32_t w[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int b = 8 * u + 2 * k;
                                w[k] = (b < p.blocks32 ? (uint32_t)__ldg(from + 2 * k) : 0u) | (b + 1 < p.blocks32 ? (uint32_t)__ldg(from + 2 * k + 1) << 16 : 0u);
                            }
                            to[i] = make_uint4(w[0], w[1], w[2], w[3]);
                        }
                    }
                    // each lane arrives once its copies (stores: this is behind them) are there
                    if (wide) asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(&scales_full[at.slot])) : "memory");
                    else mbar_arrive(&scales_full[at.slot]);
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
        }
        __syncwarp();
    }
    // free the tensor memory: everyone is past its use
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == kMiscFirst) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
}

template <int TYPE>
int launch_int8(const RqInt8Params& p, int ctas, cudaStream_t s) {
    auto kernel = rq_tc_int8_kernel<TYPE>;
    constexpr size_t smem = Int8Rings<TYPE>::bytes;
    static bool configured[64] = {};
    int dev = 0;
    RQ_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev]) {
        RQ_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        if (dev >= 0 && dev < 64) configured[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(int8_threads<TYPE>());
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

}  // namespace

int rq_launch_tc_int8(int type, const RqInt8Params& p, int ctas, cudaStream_t s) {
    return type == RQ_Q8_0 ? launch_int8<RQ_Q8_0>(p, ctas, s) : launch_int8<RQ_Q4_0>(p, ctas, s);
}
