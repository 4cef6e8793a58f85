// The cut of a batched product (recipe_dev_b200/csrc/rq_matmul_cut.cuh) walked on the host: every unit of every output tile is taken
// exactly once, the rings fit, every shared tile is added up by exactly one of its CTAs, and a work area sized ahead of time holds the call's. Built and run by tests/test_matmul_cut.py. Prints "ok".
#include <cstdio>
#include <vector>

#include "rq_matmul_cut.cuh"

using namespace rqcut;

static int fail(const char* what, int type, bool codes, int sms, long long rows, long long cols, int tokens) {
    std::printf("%s: type %d codes %d, %d SMs, %lld x %lld, %d tokens\n", what, type, (int)codes, sms, rows, cols, tokens);
    return 1;
}

static int walk_call(int type, bool codes, int sms, int64_t rows, int64_t cols, int tokens) {
    const TcCut c = tc_cut(type, codes, sms, rows, cols, tokens);
    const int64_t tiles = (int64_t)c.tiles_m * c.n_tiles;
    if (c.tiles_m * 128LL * c.mh < rows || (int64_t)c.n_tiles * c.bn < tokens) return fail("outputs outside every tile", type, codes, sms, rows, cols, tokens);
    const bool k = type == RQ_Q4_K || type == RQ_Q6_K;
    if (codes && c.mh == 2) {
        // the kernel of bytes: its own rings (how they fit is asserted where they are laid out), and every part of its shared memory in them
        const bool q8 = type == RQ_Q8_0;
        const int b = q8 ? 4 : 3, a = q8 ? 3 : 2, raw = q8 ? 0 : 3, scales = 3;
        const size_t parts = (size_t)b * (64 * 128) + (size_t)a * (256 * 128) + (size_t)raw * (128 * 128) + (size_t)scales * (8 * 64 * 4 + 256 * 16) + 256 * 64 * 4;
        if (c.smem != parts + 1024 || c.smem > 220 * 1024) return fail("shared memory of the kernel of bytes", type, codes, sms, rows, cols, tokens);
        if (c.accs || c.a_slots || c.b_slots || c.raw_slots) return fail("rings that nobody reads", type, codes, sms, rows, cols, tokens);
        if (c.xs_bytes != (size_t)c.n_tiles * c.units * 2 * (64 * 128) || c.steps_bytes != (size_t)c.n_tiles * c.units * 8 * 64 * 4 || c.partial_bytes != (size_t)2 * c.share * 64 * 256 * 4)
            return fail("scratch of the kernel of bytes", type, codes, sms, rows, cols, tokens);
    } else {
        // tensor memory, 512 columns: accumulators of at least two steps, (codes, one row half) two sets of totals, operand slots, found by a mask
        const int acc_cols = c.mh == 1 && !codes ? 2 * c.bn : c.bn, totals = codes ? 2 * c.bn : 0;
        if (c.accs * acc_cols + totals + c.a_slots * format_sizes(type).a_cols > 512 || c.accs < (k ? 2 : 4) || c.accs > kMaxAcc || c.accs % (k ? 1 : 2) || c.a_slots < 2 || c.a_slots > kMaxA ||
            (c.a_slots & (c.a_slots - 1)))
            return fail("tensor memory", type, codes, sms, rows, cols, tokens);
        // rings whose slots keep their waiters, and nobody as many steps ahead as there are step barriers (32)
        const bool even_raw = c.mh == 2 || type == RQ_Q8_0;
        if (c.b_slots < 2 || c.b_slots > kMaxB || (c.mh == 1 && c.b_slots % 2) || c.raw_slots < 2 || c.raw_slots > kMaxRaw || (even_raw && c.raw_slots % 2) || c.b_slots * c.mh * (k ? 1 : 2) >= 32)
            return fail("rings", type, codes, sms, rows, cols, tokens);
        // shared memory: the rings, what the drain and staging warps keep behind them, and room to align
        const size_t b_bytes = (size_t)c.bn * (codes ? 128 : 256), kept = (c.mh == 1 ? c.bn * 512 : 0) + (type == RQ_Q4_K ? kStashBytes * c.mh : 0);
        if (c.b_slots * b_bytes + (size_t)c.raw_slots * format_sizes(type).raw_bytes + kept + 1024 > c.smem || c.smem > (size_t)(codes ? 218 : 225) * 1024)
            return fail("shared memory", type, codes, sms, rows, cols, tokens);
    }
    // token tiles of a width that the drain loops are instantiated for
    const bool width = c.mh == 1 ? c.bn == 16 || c.bn == 32 || c.bn == 48 || c.bn == 64 : (codes ? c.bn == kInt8Tokens : c.bn == 64 || c.bn == 96 || (k && c.bn == 128));
    if (!width) return fail("a tile of another width", type, codes, sms, rows, cols, tokens);
    std::vector<int> next_unit(tiles, 0), arrivals(c.rest_tiles, 0), summed(c.rest_tiles, 0);
    std::vector<char> place_used((size_t)2 * c.share, 0);
    for (int cta = 0; cta < c.ctas; ++cta) {  // in CTA order, a tile's pieces come in unit order
        Walk walk(c.whole, c.rest_tiles, c.units, c.share, c.ctas, cta);
        int tile, u0, u1, segments = 0;
        while (walk.next(tile, u0, u1)) {
            ++segments;
            if (tile < 0 || tile >= tiles || u0 < 0 || u0 >= u1 || u1 > c.units) return fail("a segment outside the work", type, codes, sms, rows, cols, tokens);
            if (next_unit[tile] != u0) return fail("a unit missed or taken twice", type, codes, sms, rows, cols, tokens);
            next_unit[tile] = u1;
            if (u0 == 0 && u1 == c.units) continue;  // written by the CTA itself
            const int t = (int)(tile - (int64_t)c.whole * c.ctas);
            if (t < 0 || t >= c.rest_tiles) return fail("a whole tile cut in pieces", type, codes, sms, rows, cols, tokens);
            const Deal deal(c.share, c.rest_tiles, c.units);
            const int first = deal.first(t), last = deal.last(t, cta), place = Deal::place(cta, first);
            if (cta < first || cta > last || place < 0 || place >= 2 * c.share || place_used[place]) return fail("a piece's place", type, codes, sms, rows, cols, tokens);
            place_used[place] = 1;
            if (arrivals[t]++ == last - first) {  // the last one to arrive adds the pieces first .. last
                ++summed[t];
                for (int p = first; p <= last; ++p)
                    if (!place_used[Deal::place(p, first)]) return fail("a sum over a piece nobody left", type, codes, sms, rows, cols, tokens);
            }
        }
        if (segments > c.whole + 2) return fail("more than two pieces", type, codes, sms, rows, cols, tokens);
    }
    for (int64_t t = 0; t < tiles; ++t)
        if (next_unit[t] != c.units) return fail("a tile not finished", type, codes, sms, rows, cols, tokens);
    for (int t = 0; t < c.rest_tiles; ++t)
        if (arrivals[t] ? summed[t] != 1 : 0) return fail("a shared tile nobody adds up", type, codes, sms, rows, cols, tokens);
    return 0;
}

int main() {
    const int types[4] = {RQ_Q4_K, RQ_Q6_K, RQ_Q8_0, RQ_Q4_0};
    const int64_t named[][3] = {{14336, 4096, 673}, {14336, 4096, 700}, {14336, 4096, 768}, {28672, 8192, 300}, {151936, 4096, 1}, {151936, 2560, 16}, {152064, 3584, 16}, {11008, 4096, 600},
                                {8192, 2048, 400}, {25600, 5120, 200}, {19072, 512, 16}, {19200, 4096, 16}, {19072, 4096, 100}, {1, 256, 12}, {300, 16777216, 9}};
    // how wide a K-quant's token tile is: where there are tiles enough a wide one, where few are shared by many CTAs a narrower one
    const int64_t widths[][4] = {{14336, 4096, 509, 128}, {4096, 14336, 256, 128}, {8192, 1024, 256, 128}, {14336, 4096, 80, 96}, {12000, 1024, 256, 96}, {8192, 1024, 300, 96}, {2000, 1536, 128, 64}, {512, 14336, 128, 64}};
    for (int type : {RQ_Q4_K, RQ_Q6_K})
        for (const auto& w : widths)
            if (tc_cut(type, false, 148, w[0], w[1], (int)w[2]).bn != w[3]) return fail("another tile width than the measured one", type, false, 148, w[0], w[1], (int)w[2]);
    for (int type : types)
        for (int codes = 0; codes < (type == RQ_Q8_0 || type == RQ_Q4_0 ? 2 : 1); ++codes) {
            for (const auto& n : named)
                if (walk_call(type, codes, 148, n[0], n[1], (int)n[2])) return 1;
            uint64_t state = 88172645463325252ull + type;
            auto pick = [&](int64_t lo, int64_t hi) { state ^= state << 13; state ^= state >> 7; state ^= state << 17; return lo + (int64_t)(state % (uint64_t)(hi - lo + 1)); };
            for (int i = 0; i < 20000; ++i) {
                const int sms = i % 4 ? 148 : (int)pick(1, 160);
                const int64_t rows = pick(1, i % 2 ? 30000 : 160000), units = pick(1, i % 3 ? 20 : 64), tokens = pick(1, i % 5 ? 200 : 1200);
                if (walk_call(type, codes, sms, rows, units * 256, (int)tokens)) return 1;
                // reserved for this shape and for a larger one
                const size_t need = scratch_bytes(tc_cut(type, codes, sms, rows, units * 256, (int)tokens));
                if (scratch_bound(sms, rows, units * 256, (int)tokens) < need) return fail("reserved too little", type, codes, sms, rows, units * 256, (int)tokens);
                if (scratch_bound(sms, rows + pick(0, 5000), 256 * (units + pick(0, 8)), (int)(tokens + pick(0, 100))) < need) return fail("a larger shape reserved too little", type, codes, sms, rows, units * 256, (int)tokens);
            }
        }
    std::printf("ok\n");
    return 0;
}
