// How a batched product is cut: row halves and tokens per tile, CTAs, ring depths, shared memory and scratch, and the deal of the tiles
// that several CTAs share. Arithmetic only and no CUDA in it, so that a host test can walk the work of a call over many shapes.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "rq.h"
#include "rq_act_layout.cuh"

namespace rqcut {

constexpr int kMaxRaw = 8, kMaxB = 12, kMaxA = 8, kMaxAcc = 8;
constexpr int kStashBytes = 4 * 128 * 16;  // Q4_K, a row half: the headers of a window's superblocks

// drain_warps; groups: staging groups of four warps; cols: tokens per tile at most; registers of the drain, staging and other
// warps, which together may not exceed the launch's (threads x the registers a thread is compiled for: 896 x 72, 640 x 96).
// CODES: int8 activations over the 32-value formats, up to 64 tokens (beyond: rq_matmul_int8.cu).
template <int MH, bool CODES> struct Shape;
template <> struct Shape<1, false> { static constexpr int drain_warps = 8, groups = 4, cols = 64, drain_regs = 120, stage_regs = 56, other_regs = 40, launch_regs = 72; };
template <> struct Shape<2, false> { static constexpr int drain_warps = 8, groups = 2, cols = 128, drain_regs = 168, stage_regs = 56, other_regs = 32, launch_regs = 96; };
template <> struct Shape<1, true> { static constexpr int drain_warps = 8, groups = 4, cols = 64, drain_regs = 128, stage_regs = 48, other_regs = 40, launch_regs = 72; };
// The kernel of int8 activations over Q8_0 / Q4_0 beyond that (rq_matmul_int8.cu): a tile is 128 * 2 rows x kInt8Tokens, a drain thread has two rows of a
// quarter of the tokens; accumulators are stages of a 64-wide slice (two groups x two row halves).
constexpr int kInt8Tokens = 64, kInt8DrainWarps = 16, kInt8Stages = 2, kInt8AccColumns = kInt8Stages * 2 * 2 * kInt8Tokens;
static_assert(kInt8AccColumns == 512, "all of tensor memory, and no more");

template <int TYPE> struct Format {
    static constexpr bool kquant = TYPE == RQ_Q4_K || TYPE == RQ_Q6_K;
    static constexpr bool residual = TYPE == RQ_Q6_K;            // a second operand tile
    static constexpr int halves = kquant ? 1 : 2;                // sums that leave tensor memory per 64-wide slice
    static constexpr int box_bytes = TYPE == RQ_Q4_K ? 144 : (TYPE == RQ_Q6_K ? 208 : 128);  // stored bytes of a row in one TMA tile
    static constexpr int raw_slices = TYPE == RQ_Q8_0 ? 2 : 4;   // slices in one TMA tile
    static constexpr int raw_bytes = 128 * box_bytes;
    static constexpr int a_cols = residual ? 64 : 32;            // tensor-memory columns of an operand slot
};

// The kernel of bytes' shared memory (of a TcCut it takes the tiles, the deal and the scratch), in half units: activations, operands of both row halves (Q8_0: the stored bytes as
// they land), Q4_0's stored bytes (slots of a unit of 128 rows), the steps and the stored scales of a unit; behind them the drain threads' totals, and room to align.
template <int TYPE> struct Int8Rings {
    static constexpr int b_slots = TYPE == RQ_Q8_0 ? 4 : 3, a_slots = TYPE == RQ_Q8_0 ? 3 : 2, raw_slots = TYPE == RQ_Q8_0 ? 0 : 3, scale_slots = 3;
    static constexpr int b_bytes = kInt8Tokens * 128, half_bytes = 128 * 128, step_bytes = 8 * kInt8Tokens * 4, scale_bytes = step_bytes + 256 * 16;
    static constexpr int totals_bytes = 32 * kInt8DrainWarps * 2 * (kInt8Tokens / 4) * 4;
    static constexpr size_t bytes = b_slots * b_bytes + a_slots * 2 * half_bytes + raw_slots * half_bytes + scale_slots * scale_bytes + totals_bytes + 1024;
    static_assert(bytes + 512 <= 227 * 1024, "the barriers want room too");
};

// The slices of a segment (units u0 .. u1 - 1 of a tile) in the order every role takes them: four a unit and, over Q4_K, behind the last unit of every
// aligned window of four (or the segment's last) one more for the window's minimum terms.
template <int TYPE> struct Slices {
    static constexpr bool minimum = TYPE == RQ_Q4_K;
    static RQ_HOST_DEVICE int count(int u0, int u1) { return 4 * (u1 - u0) + (minimum ? ((u1 - 1) >> 2) - (u0 >> 2) + 1 : 0); }
    static RQ_HOST_DEVICE bool closes(int u, int u1) { return minimum && ((u & 3) == 3 || u == u1 - 1); }
};

// The deal of the shared tiles: their units, numbered tile after tile, are cut into `share` ranges of equal length (to one unit), CTA c
// of the launch takes range c and the CTAs from `share` on take none. No range is empty (share <= the units) and none is longer
// than a tile, so the pieces of a tile are exactly the ranges first(t) .. last(t), and a CTA has at most two pieces: the end of one
// tile and the start of the next. (Fewer than 148 tiles of at most 65536 units among 148 CTAs: the products fit 32 bits.)
struct Deal {
    uint32_t total;
    int share, units;
    RQ_HOST_DEVICE Deal(int share_, int rest_tiles, int units_) : total((uint32_t)rest_tiles * (uint32_t)units_), share(share_), units(units_) {}
    RQ_HOST_DEVICE uint32_t begin(int c) const { return (uint32_t)c * total / (uint32_t)share; }
    RQ_HOST_DEVICE int first(int t) const {
        const uint32_t at = (uint32_t)t * (uint32_t)units;
        int c = (int)(at * (uint32_t)share / total);
        while (c > 0 && begin(c) > at) --c;
        while (begin(c + 1) <= at) ++c;
        return c;
    }
    RQ_HOST_DEVICE int last(int t, int c) const {  // c: a CTA that has a piece of the tile
        const uint32_t end = (uint32_t)(t + 1) * (uint32_t)units;
        while (c + 1 < share && begin(c + 1) < end) ++c;
        return c;
    }
    // where CTA c leaves its sums of a tile whose pieces begin at CTA `first`: the tile's first CTA began in an earlier tile or where this
    // one does and uses its second place, the others began in this tile and use their first
    static RQ_HOST_DEVICE int place(int c, int first) { return 2 * c + (c == first ? 1 : 0); }
};

// The tiles and unit ranges of one CTA, in the order every role walks them.
struct Walk {
    const int whole, units, ctas, cta;
    int i, at, end;  // whole tiles taken; position among the shared units
    RQ_HOST_DEVICE Walk(int whole_, int rest_tiles, int units_, int share, int ctas_, int cta_) : whole(whole_), units(units_), ctas(ctas_), cta(cta_), i(0), at(0), end(0) {
        if (cta < share) {
            const Deal deal(share, rest_tiles, units);
            at = (int)deal.begin(cta);
            end = (int)deal.begin(cta + 1);
        }
    }
    RQ_HOST_DEVICE bool next(int& tile, int& u0, int& u1) {
        if (i < whole) { tile = i * ctas + cta; u0 = 0; u1 = units; ++i; return true; }
        if (at >= end) return false;
        const int t = at / units;
        tile = whole * ctas + t;
        u0 = at - t * units;
        u1 = units < u0 + end - at ? units : u0 + end - at;
        at += u1 - u0;
        return true;
    }
};

struct TcCut {
    int mh, bn, n_tiles, tiles_m, units, image_tiles, windows, ctas, whole, rest_tiles, share;
    int raw_slots, b_slots, a_slots, accs;
    size_t smem, records_bytes, xs_bytes, steps_bytes, partial_bytes;
};
struct FormatSizes { int raw_bytes, a_cols, raw_per_unit; };
inline FormatSizes format_sizes(int type) {
    switch (type) {
        case RQ_Q4_K: return {Format<RQ_Q4_K>::raw_bytes, Format<RQ_Q4_K>::a_cols, 1};
        case RQ_Q6_K: return {Format<RQ_Q6_K>::raw_bytes, Format<RQ_Q6_K>::a_cols, 1};
        case RQ_Q8_0: return {Format<RQ_Q8_0>::raw_bytes, Format<RQ_Q8_0>::a_cols, 2};
        default: return {Format<RQ_Q4_0>::raw_bytes, Format<RQ_Q4_0>::a_cols, 1};
    }
}
// Tokens per tile and token tiles, of tiles of at most `widest` tokens in steps of `grain`.
struct TokenTiles { int n, bn; };
inline TokenTiles token_tiles(int tokens, int widest, int grain) {
    TokenTiles t;
    t.n = (tokens + widest - 1) / widest;
    t.bn = ((tokens + t.n - 1) / t.n + grain - 1) / grain * grain;
    return t;
}
// Whole tiles per CTA, and the tiles that are left with the number of CTAs that share them out. Few tiles to share: more CTAs to a tile shorten its
// products (some two microseconds a unit) and lengthen the last one's sum (most of a microsecond a piece, a trip to L2 each), so about
// the square root of twice its units share one, at most (never more than it has).
struct TileShare { int ctas, whole, rest_tiles, share; };
inline TileShare share_out(int64_t tiles, int units, int sm_count) {
    TileShare s;
    s.ctas = tiles * units < sm_count ? (int)(tiles * units) : sm_count;
    int pieces = 1;
    while ((pieces + 1) * (pieces + 1) <= 2 * units) ++pieces;
    if (tiles * pieces < s.ctas) s.ctas = (int)(tiles * pieces);
    s.whole = (int)(tiles / s.ctas);
    s.rest_tiles = (int)(tiles - (int64_t)s.whole * s.ctas);
    s.share = (int64_t)s.rest_tiles * pieces < s.ctas ? s.rest_tiles * pieces : s.ctas;
    return s;
}
// What the CTA with the most to do needs for a K-quant call of two row halves, roughly (one is some five nanoseconds): its units, each three hundred columns' worth of
// staging and hand-offs besides its columns, and a shared tile's way out (two of them where the ranges do not end with the
// tiles) with the sum over its pieces, both by the column. 312 calls (both K-quants, thirteen shapes, 65 to 509 tokens) timed with tiles of up to 96 and of up to 128
// tokens: the lower estimate is the faster one, or within 7 % of it; where 128 had replaced 96 for every call, the few tiles of small weights and short rows took up to
// 1.38 times as long (Q6_K, us, 96 / 128: 2000 x 1536 with 128 tokens 18.6 / 25.7, 12000 x 1024 with 256 35.1 / 44.5; 14336 x 4096 with 509 180 / 150).
inline int64_t call_cost(int64_t row_tiles, int units, int tokens, int widest, int grain, int sm_count) {
    const TokenTiles t = token_tiles(tokens, widest, grain);
    const TileShare s = share_out(row_tiles * t.n, units, sm_count);
    int64_t own = (int64_t)s.whole * units, ways = 0, pieces = 0;
    if (s.share) {
        const int64_t shared = (int64_t)s.rest_tiles * units;
        own += (shared + s.share - 1) / s.share;
        if (s.share % s.rest_tiles) {
            const int64_t least = shared / s.share;
            ways = 2;
            pieces = (units + least - 1) / least + 1;
        } else if (s.share > s.rest_tiles) {
            ways = 1;
            pieces = s.share / s.rest_tiles;
        }
    }
    return 2 * own * (300 + t.bn) + t.bn * (10 * ways + pieces);
}
inline TcCut tc_cut(int type, bool codes, int sm_count, int64_t rows, int64_t cols, int tokens) {
    TcCut c;
    const FormatSizes f = format_sizes(type);
    const bool kquant = type == RQ_Q4_K || type == RQ_Q6_K;
    // (fp32 activations over the 32-value formats: two accumulators a slice, of hi and lo columns each, twice; 48 tokens fit, 96 of two row halves)
    const int widest_1 = !codes && !kquant ? 48 : Shape<1, false>::cols;
    c.mh = tokens <= widest_1 ? 1 : 2;
    c.tiles_m = (int)((rows + 128 * c.mh - 1) / (128 * c.mh));
    c.units = (int)((cols + 255) / 256);
    const int grain = c.mh == 2 ? 32 : 16;
    int widest = c.mh == 1 ? widest_1 : (codes ? kInt8Tokens : 96);
    if (c.mh == 2 && kquant && call_cost(c.tiles_m, c.units, tokens, Shape<2, false>::cols, grain, sm_count) <= call_cost(c.tiles_m, c.units, tokens, widest, grain, sm_count)) widest = Shape<2, false>::cols;
    const TokenTiles t = token_tiles(tokens, widest, grain);
    c.n_tiles = t.n;
    c.bn = t.bn;
    c.windows = type == RQ_Q4_K ? (c.units + 3) / 4 : 0;
    c.image_tiles = codes && c.mh == 2 ? 2 * c.units : 4 * c.units + c.windows;  // (of 64 inputs a row; codes of two row halves: bytes, of 128)
    const TileShare sh = share_out((int64_t)c.tiles_m * c.n_tiles, c.units, sm_count);
    c.ctas = sh.ctas; c.whole = sh.whole; c.rest_tiles = sh.rest_tiles; c.share = sh.share;
    const int b_bytes = c.bn * (codes ? 128 : 256);
    c.records_bytes = codes ? (rq_act_token_bytes(cols) * (size_t)tokens + 255) & ~(size_t)255 : 0;
    c.xs_bytes = (size_t)c.n_tiles * c.image_tiles * b_bytes;
    c.steps_bytes = codes ? (size_t)c.n_tiles * c.units * 8 * c.bn * 4 : 0;
    c.partial_bytes = (size_t)2 * c.share * c.bn * 128 * c.mh * 4;
    if (codes && c.mh == 2) {  // rq_matmul_int8.cu: its rings are known beforehand
        c.raw_slots = c.b_slots = c.a_slots = c.accs = 0;
        c.smem = type == RQ_Q8_0 ? Int8Rings<RQ_Q8_0>::bytes : Int8Rings<RQ_Q4_0>::bytes;
        return c;
    }
    // A parity wait says no more than odd or even, so whoever waits on a slot must have seen its previous use: MH = 1, the issuing warps
    // take alternate activation slots, and Q8_0's staging groups every second tile of stored bytes; MH = 2, a staging group every second
    // tile: even numbers of each. (The steps' own barriers are indexed by the step.)
    // tensor memory, 512 columns: operand slots (a power of two; eight where two steps' accumulators still fit beside them), totals
    // (codes, one row half), and accumulators of as many steps as are left room for: a step's are drained while the next ones are filled
    const int halves = kquant ? 1 : 2, acc_cols = c.mh == 1 && !codes ? 2 * c.bn : c.bn, step_cols = halves * acc_cols, totals = codes && c.mh == 1 ? 2 * c.bn : 0;
    c.a_slots = type == RQ_Q6_K ? (c.mh == 1 ? 4 : 2) : (c.mh == 1 && 512 - 8 * f.a_cols - totals >= 2 * step_cols ? 8 : 4);
    int steps = (512 - c.a_slots * f.a_cols - totals) / step_cols;
    if (steps > kMaxAcc / halves) steps = kMaxAcc / halves;
    c.accs = steps * halves;
    // shared memory: activation slots, then as many slots of stored bytes as fit (MH = 1: and the odd slices' sums; Q4_K: and the headers of a window)
    const int kept = (c.mh == 1 ? c.bn * 128 * 4 : 0) + (type == RQ_Q4_K ? kStashBytes * c.mh : 0), budget = (codes ? 212 : 220) * 1024 - kept;
    c.b_slots = c.mh == 1 ? 4 : 3;
    c.raw_slots = (budget - c.b_slots * b_bytes) / f.raw_bytes;
    const int raw_max = c.mh * 2 * f.raw_per_unit < kMaxRaw ? 6 : kMaxRaw, raw_grain = c.mh == 2 || f.raw_per_unit == 2 ? 2 : 1;
    c.raw_slots = (c.raw_slots < raw_max ? c.raw_slots : raw_max) / raw_grain * raw_grain;
    const int b_max = c.mh == 1 ? kMaxB : 6, b_more = c.mh == 1 ? 2 : 1;  // a slot is refilled over one trip to L2, some 1500 cycles, a few slices' worth of time
    while (c.b_slots + b_more <= b_max && (c.b_slots + b_more) * b_bytes + c.raw_slots * f.raw_bytes <= budget) c.b_slots += b_more;
    c.smem = (size_t)c.b_slots * b_bytes + (size_t)c.raw_slots * f.raw_bytes + kept + 1024;
    return c;
}
// Work area of a call: the records (where INT8_CACHED calls look for them), the image, its steps, the shared tiles' sums and a counter
// for each of them.
inline size_t scratch_bytes(const TcCut& c) { return c.records_bytes + c.xs_bytes + c.steps_bytes + c.partial_bytes + (size_t)c.rest_tiles * 4; }

// Enough for every call of up to this many rows, inputs and tokens, of any format and activation mode. Tokens are padded by less than
// 32 to a token tile (four bytes an input: the codes' image, steps and records are less); the shared tiles' sums are two tiles a CTA: 64 x 128 numbers of one row half, of two row halves (from 49
// tokens on for fp32 activations over the 32-value formats) 64 x 256, from 65 tokens on 128 x 256.
inline size_t scratch_bound(int sm_count, int64_t rows, int64_t cols, int tokens) {
    const int64_t units = (cols + 255) / 256, tiles_n = (tokens + 95) / 96;
    const size_t image = (size_t)(tokens + 32 * tiles_n + 32) * 256 * (size_t)(4 * units + (units + 3) / 4);
    const int64_t work = ((rows + 127) / 128) * units * tiles_n;
    const size_t ctas = (size_t)(work < sm_count ? work : sm_count);
    return image + 256 + 4 * ctas + 2 * ctas * (size_t)(tokens > 64 ? 128 * 256 : (tokens > 48 ? 64 * 256 : 64 * 128)) * 4;
}

}  // namespace rqcut
