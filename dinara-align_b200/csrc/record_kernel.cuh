// Whole-matrix recording of two pairs a lane group in 16-bit halves.
#pragma once

#include "affine_kernel.cuh"

namespace dinara {
namespace sweep {

// The recording sweeps' halves' maximum and flags (halves in [0, 0x8000)): the DPX maximum floored at zero; and
// adding to a plane `acc` (pair A's 16 places in the low half, pair B's in the high) place k's flags, set where a
// half of `v` has bit 15 clear. `v` = b - a + 0x8000 in each half (nothing crosses between them) has bit 15 set
// exactly where b >= a, so a clear bit records a > b. The flags move from bits 15 and 31 down to k and 16 + k by the
// high word of a product, added in the same instruction (the FMA pipe's, leaving the ALU to the cells).
__device__ __forceinline__ uint32_t max_halves(uint32_t a, uint32_t b) { return __vimax_s16x2_relu(a, b); }
__device__ __forceinline__ uint32_t gather_flag(uint32_t acc, uint32_t v, int k) {
    const uint32_t flags = ~v & 0x80008000u;
    return k == 15 ? acc + flags : __umulhi(flags, 1u << (17 + k)) + acc;
}
// b - a + c (the halves' sums in [0, 0x10000), so none crosses into the other) by two multiply-adds,
// which the multiply-add pipe takes, leaving the ALU pipe, the recording sweeps' bound, to the cells.
__device__ __forceinline__ uint32_t difference_mad(uint32_t b, uint32_t a, uint32_t c) {
    uint32_t biased, out;
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(biased) : "r"(b), "r"(1u), "r"(c));
    asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(out) : "r"(a), "r"(0xFFFFFFFFu), "r"(biased));
    return out;
}

// What a recorded cell is held above its value: every half, a gap's opening or an entry (a byte) below a real cell
// among them, stays at zero or more.
__host__ __device__ inline int32_t record_bias(int32_t open, int32_t extend) { return -4 * (open + extend) + 130; }

// Scores and decisions of two pairs a group of G lanes of 16 columns: affine_pairs_kernel's cells, and gotoh.mojo:173-186
// decide's flags for each, a bit a place in planes of both pairs (the deletion beats the diagonal; the insertion beats
// both; each run extends only where extending beats opening; local, the cell is above the floor). A row's
// planes leave as a 64-bit word a pair: deleting, inserting, deletion runs, insertion runs, 16 places each, with both
// deleting and inserting where a local path stops (the walk's layouts 6 and 7). Strips as the 32-bit
// recording sweep's, a lane's rows together: word (strip * G + lane) * rows_pad + row - 1, two rows a store.
//
// Local pairs are hits' rows (affine_pairs_kernel<..., TRACK>), so their score is known and they end on their last
// row, in its first column of that score; no cell is compared with a best. The 32-bit form takes some
// 60 instructions a local cell, most of them for the best's place; 5,000 hits of 575 by 750 letters: 6.5 ms.
template <int G, bool LOCAL, int BITS>
__global__ void __launch_bounds__(kBlock, 2) record_pairs_kernel(KernelArgs p, TableArgs t, const int32_t *__restrict__ table32) {
    constexpr int C = 16;
    constexpr int W = G * C;
    constexpr int GPW = 32 / G;
    constexpr bool PROFILE = BITS == 8;
    __shared__ uint32_t rows8[4];
    __shared__ int8_t table8[PROFILE ? 32 * 32 : 1];
    if (threadIdx.x < 4) rows8[threadIdx.x] = t.rows8[threadIdx.x];
    if (PROFILE) load_table8(table8, table32, LOCAL ? p.extend : 0);
    __syncthreads();

    const int lane = threadIdx.x & 31;
    const int member = lane % G;
    const int group = lane / G;
    const int warp = int((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
    const int warps = int((int64_t(gridDim.x) * blockDim.x) >> 5);
    // This lane's part of its group's two profiles, letter a's of half h at [(h * t.size + a) * G].
    ProfileRow<C> *profile = reinterpret_cast<ProfileRow<C> *>(sweep_profiles) +
                             int64_t((threadIdx.x >> 5) * GPW + group) * 2 * t.size * G + member;
    const int32_t open = p.open, extend = p.extend;
    const int32_t opening = open - extend;
    const int32_t first_gap = open + extend;
    const int32_t bias = record_bias(open, extend);
    const int64_t slot = int64_t(warp) * GPW + group;
    const uint32_t opening2 = halves(opening, opening), extend2 = halves(extend, extend);
    const uint32_t open_both = uint32_t(open) + (uint32_t(open) << 16);  // of two halves, each left at zero or more
    const uint32_t at_least = 0x80008000u;                               // b - a + this: bit 15 where b >= a
    const uint32_t at_least_open = halves(0x8000 + opening, 0x8000 + opening);  // where b + opening >= a
    const int32_t top = bias + (LOCAL ? 0 : opening);

    for (uint32_t base = p.begin + uint32_t(warp) * 2 * GPW; base < p.end; base += uint32_t(warps) * 2 * GPW) {
        const uint32_t item = base + 2 * group;
        bool live[2];
        uint32_t pair[2] = {0, 0};
        PairShape sh[2] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        int rows[2], cols[2], strips[2];
        uint64_t *words[2] = {nullptr, nullptr};
        int32_t known[2] = {0, 0}, reported[2] = {0, 0};
        int end_column[2] = {INT32_MAX, INT32_MAX};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            live[h] = item + h < p.end;
            if (live[h]) {
                pair[h] = p.order[item + h];
                sh[h] = p.shapes[pair[h]];
                words[h] = p.decisions + p.decision_offsets[pair[h] - p.first_pair];
                if (LOCAL) known[h] = p.scores[pair[h]];
            }
            rows[h] = int(sh[h].rows);
            cols[h] = int(sh[h].columns);
            strips[h] = live[h] && rows[h] > 0 && cols[h] > 0 ? (cols[h] + W - 1) / W : 0;
        }
        const int warp_strips = warp_max(max(strips[0], strips[1]));

        for (int s = 0; s < warp_strips; ++s) {
            const int first_col = s * W + member * C;
            uint32_t sel[PROFILE ? 1 : C];
            if (PROFILE) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    fill_profile<C>(profile + h * t.size * G, G, t.size, table8,
                                    s < strips[h] ? min(max(cols[h] - first_col, 0), C) : 0, [&](int k) {
                                        return letter_at<8>(p.tape, sh[h].second_word, uint32_t(first_col + k));
                                    });
            }
#pragma unroll
            for (int k = 0; k < (PROFILE ? 0 : C); ++k) {
                const int col = first_col + k;
                const uint32_t a = s < strips[0] && col < cols[0]
                                       ? half_selector_a(letter_at<2>(p.tape, sh[0].second_word, uint32_t(col)))
                                       : kPadHalf;
                const uint32_t b = s < strips[1] && col < cols[1]
                                       ? half_selector_b(letter_at<2>(p.tape, sh[1].second_word, uint32_t(col)))
                                       : kPadHalf;
                sel[k] = pair_selector(a, b);
            }
            const uint32_t top2 = halves(top, top), top_gap2 = halves(top + first_gap, top + first_gap);
            uint32_t H[C], D[C];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                H[k] = top2;
                D[k] = top_gap2;
            }
            uint32_t edgeH = top2, edgeI = top_gap2;
            const int32_t corner = bias + (LOCAL || first_col == 0 ? 0 : opening);
            uint32_t above_left = halves(corner, corner);
            uint2 held[2] = {{0, 0}, {0, 0}};  // an odd row's word, until the next row's joins it
            uint64_t *lane_words[2];
            int group_rows = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                lane_words[h] = words[h] + int64_t(s * G + member) * ((rows[h] + 3) & ~3);
                group_rows = max(group_rows, s < strips[h] ? rows[h] : 0);
            }
            const int steps = group_rows > 0 ? group_rows + G : 0;
            const int warp_steps = warp_max(steps);
            uint32_t codes[2] = {0, 0};

            for (int step = 1; step <= warp_steps; ++step) {
                const int row = step - member;
                if (!PROFILE && (step & 15) == 1) {
#pragma unroll
                    for (int h = 0; h < 2; ++h)
                        codes[h] = sixteen_letters(p.tape, sh[h].first_word, s < strips[h] ? rows[h] : 0, row - 1);
                }
                const uint32_t here[2] = {codes[0] & 3u, codes[1] & 3u};
                codes[0] >>= 2;
                codes[1] >>= 2;
                // Local: the floor of this row's cells, held less row x extend.
                const int32_t floor_h = LOCAL ? bias - max(row, 0) * extend : 0;
                const uint32_t floor2 = halves(floor_h, floor_h);
                uint32_t leftH = __shfl_up_sync(kFull, edgeH, 1, G);
                uint32_t leftI = __shfl_up_sync(kFull, edgeI, 1, G);
                if (member == 0) {
                    if (s == 0) {
                        leftH = LOCAL ? floor2 : top2;
                        leftI = LOCAL ? halves(floor_h + first_gap, floor_h + first_gap) : top_gap2;
                    } else {
                        const int r = min(max(row, 0), group_rows);
                        const int2 c = p.carry[slot * p.carry_stride + r];
                        leftH = uint32_t(c.x);
                        leftI = uint32_t(c.y);
                    }
                }
                uint32_t diag = above_left;
                above_left = leftH;
                if (row >= 1 && row <= group_rows) {
                    uint32_t tr[2] = {0, 0};
                    ProfileRow<C> entries[PROFILE ? 2 : 1];
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const bool inside = s < strips[h] && row <= rows[h];
                        if (PROFILE) {
                            const uint32_t letter =
                                inside ? letter_at<8>(p.tape, sh[h].first_word, uint32_t(row - 1)) : 0u;
                            entries[PROFILE ? h : 0] = profile[int(h * t.size + letter) * G];
                            if (!inside) entries[PROFILE ? h : 0] = ProfileRow<C>{};
                        } else {
                            tr[h] = inside ? rows8[here[h]] : 0u;
                        }
                    }
                    uint32_t deleting = 0, inserting = 0, deletion_runs = 0, insertion_runs = 0, above_floor = 0;
                    uint32_t I = 0, Xprev = 0, Hprev = leftH, Iprev = leftI;
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const uint32_t sub = PROFILE ? profile_entry(entries[0], entries[PROFILE ? 1 : 0], k)
                                                     : uint32_t(prmt(tr[0], tr[1], sel[PROFILE ? 0 : k]));
                        const uint32_t Hup = H[k], Dup = D[k];
                        const uint32_t Dn = __viaddmax_s16x2(Hup, opening2, Dup);
                        const uint32_t Xd = __viaddmax_s16x2(diag, sub, 0u);  // never below zero
                        const uint32_t X = max_halves(Xd, Dn);
                        if (k == 0)
                            I = LOCAL ? __viaddmax_s16x2(leftI, extend2, leftH + open_both)
                                      : __viaddmax_s16x2(leftH, opening2, leftI);
                        else
                            I = LOCAL ? __viaddmax_s16x2(I, extend2, Xprev + open_both)
                                      : __viaddmax_s16x2(Xprev, opening2, I);
                        const uint32_t Hn = LOCAL ? __vimax3_s16x2(X, I, floor2) : max_halves(X, I);
                        deleting = gather_flag(deleting, difference_mad(Xd, Dn, at_least), k);                 // Dn > Xd
                        deletion_runs = gather_flag(deletion_runs, difference_mad(Hup, Dup, at_least_open), k);  // Dup > Hup + opening
                        inserting = gather_flag(inserting, difference_mad(X, I, at_least), k);                 // I > X
                        insertion_runs = gather_flag(insertion_runs, difference_mad(Hprev, Iprev, at_least_open), k);
                        if (LOCAL) above_floor = gather_flag(above_floor, difference_mad(floor2, Hn, at_least), k);
                        Xprev = X;
                        Hprev = Hn;
                        Iprev = I;
                        diag = Hup;
                        H[k] = Hn;
                        D[k] = Dn;
                    }
                    edgeH = H[C - 1];
                    edgeI = I;
                    if (member == G - 1 && s + 1 < warp_strips)
                        p.carry[slot * p.carry_stride + row] = make_int2(int32_t(edgeH), int32_t(edgeI));
                    // The insertion wins over the deletion; both where a local path stops.
                    deleting &= ~inserting;
                    if (LOCAL) {
                        deleting |= ~above_floor;
                        inserting |= ~above_floor;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const uint32_t pick = h == 0 ? 0x5410u : 0x7632u;
                        const uint2 word = make_uint2(uint32_t(prmt(deleting, inserting, pick)),
                                                      uint32_t(prmt(deletion_runs, insertion_runs, pick)));
                        const bool second = (row & 1) == 0;
                        if (s < strips[h] && row <= rows[h] && (second || row == rows[h])) {
                            const uint2 first = second ? held[h] : word;
                            *reinterpret_cast<uint4 *>(lane_words[h] + ((row - 1) & ~1)) =
                                make_uint4(first.x, first.y, word.x, word.y);
                        }
                        held[h] = word;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int owned = min(max(cols[h] - first_col, 0), C);
                        if (s >= strips[h] || row != rows[h] || owned <= 0) continue;
                        if (LOCAL) {
                            // The end: the last row's first column of the known score.
#pragma unroll
                            for (int k = C - 1; k >= 0; --k) {
                                const int32_t value = (h == 0 ? low_of(H[k]) : high_of(H[k])) - floor_h;
                                if (k < owned && value == known[h]) end_column[h] = min(end_column[h], first_col + k + 1);
                            }
                        } else if (first_col + owned == cols[h]) {
                            uint32_t value = 0;
#pragma unroll
                            for (int k = 0; k < C; ++k) value |= H[k] & (0u - uint32_t(k == owned - 1));
                            reported[h] = (h == 0 ? low_of(value) : high_of(value)) - bias;
                        }
                    }
                }
            }
            __syncwarp();
        }

#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int32_t value = reported[h];
            int column = end_column[h];
#pragma unroll
            for (int span = 1; span < G; span <<= 1) {
                value += __shfl_xor_sync(kFull, value, span, G);  // one lane holds the corner
                column = min(column, __shfl_xor_sync(kFull, column, span, G));
            }
            if (!live[h] || member != 0) continue;
            if (LOCAL)
                p.ends[pair[h] - p.first_pair] =
                    known[h] > 0 && column <= cols[h] ? (int64_t(rows[h]) << 32) | int64_t(column) : 0;
            else
                p.scores[pair[h]] = value + (rows[h] + cols[h]) * extend;
        }
    }
}

}  // namespace sweep
}  // namespace dinara
