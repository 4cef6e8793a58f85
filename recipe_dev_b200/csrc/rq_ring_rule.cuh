// Which of its two kernels the decode-only formats' matvec takes (rq_gemv_generic.cu): with a ring of rows in shared memory, or without.
// Arithmetic only and no CUDA in it, so that a host test can ask.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include "rq.h"

namespace rqring {

constexpr int kWarps = 8;                     // per CTA, of both kernels
constexpr int kChunkGroups = 256;             // 32-value groups of x in shared memory at a time: 8192 inputs
constexpr int kGroupFloats = 36;              // a group's 32 inputs, padded: 144 bytes, so that eight lanes on adjacent groups read eight bank groups
constexpr int kRows = 4, kMaxStages = 4;      // rows a slot, slots a warp at most
constexpr int kCtas = 2;                      // CTAs an SM of the kernel with the ring
constexpr size_t kSmem = 112 * 1024;          // of one of them

constexpr int block_values(int t) { return t == RQ_Q5_K || t == RQ_Q2_K || t == RQ_Q3_K || t == RQ_Q8_K || t == RQ_IQ4_XS ? 256 : 32; }
constexpr int block_bytes(int t) {
    return t == RQ_Q4_1 ? 20 : t == RQ_Q5_0 ? 22 : t == RQ_Q5_1 ? 24 : t == RQ_IQ4_NL ? 18 : t == RQ_Q8_1 ? 36 : t == RQ_Q5_K ? 176 : t == RQ_Q2_K ? 84 : t == RQ_Q3_K ? 110 : t == RQ_Q8_K ? 292 : 136;
}
constexpr int chunk_bytes(int t) { return 1024 / block_values(t) * block_bytes(t); }  // 32 groups
// Bulk copies are whole 16-byte lines: 32 groups of Q3_K are 440 bytes, so it never has a ring.
constexpr bool whole_lines(int t) { return chunk_bytes(t) % 16 == 0; }

// CTAs an SM that the registers of the kernel without a ring are cut for, four rows a warp: two for the formats of many words a group.
constexpr bool many_words(int t) { return t == RQ_Q5_K || t == RQ_Q3_K || t == RQ_Q8_1 || t == RQ_Q8_K || t == RQ_IQ4_XS; }

// Whether the ring is the faster one. It gives every warp an equal share of the rows, to one row, and hides memory behind its own
// copies; the other kernel has up to 24 warps an SM instead of 16 where the format's words fit the registers of three CTAs, but its CTAs of 32 rows come
// in whole numbers to an SM. Measured over 987 weights (nine formats, 9472 to 152064 rows, 384 to 8192 inputs; us without / with the ring):
//   * many words a group: always, from the first row past four a warp on (Q5_K 14336 x 4096 26.5 / 21.0, Q8_K 17.4 of 23.2; one round of
//     exactly four rows 2048 wide 6.9 / 7.3). IQ4_XS, whose sixteen bytes need the least of them, from ten rows a warp on, below where the fullest
//     SM has a fifth more CTAs than the average (14336 rows 26.0 / 22.4, 13000 rows 1024 wide 1.08 times as long with it).
//   * the others where a first full round of CTAs leaves a second one: Q4_1 from 2048 inputs, Q2_K from 3072 (14336 x 4096 20.1 / 16.7 and 19.3 / 16.8, 12000 x 2048
//     1.09 and 1.06 times as long); the 18, 22 and 24 byte blocks, whose words straddle the ring's banks, where the second round is a quarter full or less, from
//     3072 inputs (Q5_0 14336 x 4096 24.5 / 20.3; 28416 rows 1.03 times as long, IQ4_NL 1.09);
//   * and where two CTAs an SM and little more would be dealt as three to some and one to others: four to 4.25 rows a warp, from 4096 inputs
//     (9472 x 4096, Q4_1 0.80, Q5_1 0.76 of the time; IQ4_NL 1.09).
constexpr bool faster(int t, int sm_count, int64_t rows, int64_t cols) {
    const int64_t ctas = (rows + 4 * kWarps - 1) / (4 * kWarps), full = 3 * (int64_t)sm_count, share = (int64_t)sm_count * kCtas * kWarps;  // share: rows at one a warp
    const bool one_round = rows >= 4 * share && 4 * rows <= 17 * share && cols >= 4096;
    if (t == RQ_IQ4_XS) return rows > 10 * share || (rows > 4 * share && cols >= 1024 && 5 * ((ctas + sm_count - 1) / sm_count * sm_count) >= 6 * ctas);
    if (many_words(t)) return rows > 4 * share || one_round;
    if (t == RQ_IQ4_NL) return cols >= 3072 && ctas > full && 4 * ctas <= 5 * full;
    if (one_round) return true;
    if (t == RQ_Q4_1) return cols >= 2048 && ctas > full;
    if (t == RQ_Q2_K) return cols >= 3072 && ctas > full;
    return cols >= 3072 && ctas > full && 4 * ctas <= 5 * full;
}

inline size_t input_bytes(int64_t cols) { return ((size_t)(cols / 32) * kGroupFloats * 4 + 127) & ~(size_t)127; }
// Slots of each warp's ring; 0: the kernel without one. One token (several have warps enough to hide each other's waits: Q4_1, four tokens of 9000 x 3072,
// 24.9 us without / 30.6 with), rows of whole lines (the plane itself starts on one: the caller's check), inputs that lie in
// shared memory at once, and two CTAs an SM with as many slots as fit half of its shared memory beside the inputs.
inline int stages(int t, int sm_count, int64_t rows, int64_t cols, int tokens) {
    if (tokens > 1 || !whole_lines(t) || cols / block_values(t) * block_bytes(t) % 16 || cols > 32 * kChunkGroups || !faster(t, sm_count, rows, cols)) return 0;
    const int n = (int)((kSmem - input_bytes(cols)) / ((size_t)kWarps * kRows * chunk_bytes(t)));
    return n < 2 ? 0 : (n < kMaxStages ? n : kMaxStages);
}

}  // namespace rqring
