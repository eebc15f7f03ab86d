// Free-end and extension scores of two pairs a lane group in 16-bit halves.
#pragma once

#include "affine_kernel.cuh"

namespace dinara {
namespace sweep {

// A row window: the letters of rows row0 .. row0 + 15, the first in the low bits, for a sequence read forwards,
// or (backwards) its last `length` letters' mirror, row r reading letter length - r.
__device__ __forceinline__ uint32_t sixteen_rows(const uint32_t *__restrict__ tape, uint32_t first_word, int length,
                                                 int row0, bool backwards) {
    if (!backwards) return sixteen_letters(tape, first_word, length, row0 - 1);
    uint32_t run = __brev(sixteen_letters(tape, first_word, length, length - row0 - 15));
    return ((run & 0x55555555u) << 1) | ((run >> 1) & 0x55555555u);  // each letter's two bits back in order
}

// Global scores with free ends (scored.mojo:69-240 FROM_EDGE) of two pairs a group of G lanes, pair A in every
// register's low half and pair B in its high half: the recurrence of affine_pairs_kernel, cells shifted by (row +
// column) * extend, from borders with free letters (free_edge). The schedule gives it pairs whose shifted values
// stay inside 16 bits. Each row's last column is picked out of the lane's registers by a mask a place (an
// instruction a place, a fifth of the sweep's; the last row's ends, once a pair, by a loop).
//
// Of equal ends the one furthest along the reference less the query is kept with p.free_highest, else the
// least so. With p.extents each pair is its prefixes of so many letters, read backwards; with p.known, each
// pair's score, it stops at the last row a path worth that can span (hit_first_row).
//
// 16 places a lane move 32 cells in 96 DPX, permute and logic instructions, where the 32-bit form takes 80 for
// 16 cells and a shared-memory read a cell.
template <int G, int C, int BITS = 2>
__global__ void __launch_bounds__(kBlock, 2) free_pairs_kernel(KernelArgs p, TableArgs t, const int32_t *__restrict__ table32) {
    constexpr int W = G * C;
    constexpr int GPW = 32 / G;
    constexpr bool PROFILE = BITS == 8;
    __shared__ uint32_t rows8[4];
    __shared__ int8_t table8[PROFILE ? 32 * 32 : 1];
    if (threadIdx.x < 4) rows8[threadIdx.x] = t.rows8[threadIdx.x];
    if (PROFILE) load_table8(table8, table32, 0);
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
    const int64_t slot = int64_t(warp) * GPW + group;
    const uint32_t opening2 = halves(opening, opening);
    const bool backwards = p.extents != nullptr;
    const bool highest = p.free_highest != 0;

    for (uint32_t item0 = p.begin + uint32_t(warp) * 2 * GPW; item0 < p.end; item0 += uint32_t(warps) * 2 * GPW) {
        const uint32_t item = item0 + 2 * group;
        bool live[2];
        uint32_t pair[2] = {0, 0};
        PairShape sh[2] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        int rows[2], cols[2], strips[2], swept[2], first_end[2], free_rs[2];
        int32_t best[2];
        int best_row[2] = {0, 0}, best_col[2] = {0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            live[h] = item + h < p.end;
            if (live[h]) {
                pair[h] = p.order[item + h];
                sh[h] = p.shapes[pair[h]];
            }
            rows[h] = int(sh[h].rows);
            cols[h] = int(sh[h].columns);
            if (backwards && live[h]) {
                const int64_t extent = p.extents[pair[h] - p.first_pair];
                rows[h] = int(extent >> 32);
                cols[h] = int(extent & 0xffffffff);
            }
            const bool work = live[h] && rows[h] > 0 && cols[h] > 0;
            strips[h] = work ? (cols[h] + W - 1) / W : 0;
            free_rs[h] = min(p.free_reference_start, rows[h]);
            swept[h] = work ? rows[h] : 0;
            if (work && p.known)
                swept[h] = rows[h] - hit_first_row(rows[h], cols[h], p.known[pair[h]], p.best_entry, open, extend);
            // The first row whose last column is an end.
            first_end[h] = max(rows[h] - min(p.free_reference_end, rows[h]), 1);
            best[h] = -(1 << 30);
        }
        const int warp_strips = warp_max(max(strips[0], strips[1]));
        auto offer = [&](int h, int32_t value, int r, int c) {
            const int key = r - c, best_key = best_row[h] - best_col[h];
            if (value > best[h] || (value == best[h] && (highest ? key > best_key : key < best_key))) {
                best[h] = value;
                best_row[h] = r;
                best_col[h] = c;
            }
        };

        for (int s = 0; s < warp_strips; ++s) {
            const int first = s * W + member * C;
            uint32_t sel[PROFILE ? 1 : C], last[C];
            if (PROFILE) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    fill_profile<C>(profile + h * t.size * G, G, t.size, table8,
                                    s < strips[h] ? min(max(cols[h] - first, 0), C) : 0, [&](int k) {
                                        const int col = first + k;
                                        return letter_at<8>(p.tape, sh[h].second_word,
                                                            uint32_t(backwards ? cols[h] - 1 - col : col));
                                    });
            }
#pragma unroll
            for (int k = 0; k < C; ++k) {
                uint32_t half_sel[2] = {kPadHalf, kPadHalf}, half_last[2] = {0, 0};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = first + k;
                    if (s < strips[h] && col < cols[h]) {
                        if (!PROFILE) {
                            const uint32_t y =
                                letter_at<2>(p.tape, sh[h].second_word, uint32_t(backwards ? cols[h] - 1 - col : col));
                            half_sel[h] = h == 0 ? half_selector_a(y) : half_selector_b(y);
                        }
                        if (col == cols[h] - 1) half_last[h] = 0xFFFFu;
                    }
                }
                if (!PROFILE) sel[PROFILE ? 0 : k] = pair_selector(half_sel[0], half_sel[1]);
                last[k] = half_last[0] | (half_last[1] << 16);
            }
            bool holds_last[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) holds_last[h] = s < strips[h] && cols[h] > first && cols[h] <= first + C;
            // The first row, shifted: each column's border.
            auto top = [&](int h, int column) {
                return free_edge(column, min(p.free_query_start, cols[h]), open, extend) - column * extend;
            };
            uint32_t H[C], D[C];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const int32_t a = top(0, first + k + 1), b = top(1, first + k + 1);
                H[k] = halves(a, b);
                D[k] = halves(a + first_gap, b + first_gap);
            }
            uint32_t edgeH = H[C - 1], edgeI = D[C - 1];
            uint32_t above_left = first == 0 ? 0u : halves(top(0, first), top(1, first));
            int group_rows = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) group_rows = max(group_rows, s < strips[h] ? swept[h] : 0);
            const int steps = group_rows > 0 ? group_rows + G : 0;
            const int warp_steps = warp_max(steps);

            for (int step0 = 1; step0 <= warp_steps; step0 += 16) {
                uint32_t codes[2] = {0, 0};
#pragma unroll
                for (int h = 0; h < (PROFILE ? 0 : 2); ++h)
                    codes[h] = sixteen_rows(p.tape, sh[h].first_word, live[h] ? rows[h] : 0, step0 - member, backwards);
#pragma unroll 2
                for (int u = 0; u < 16; ++u) {
                    const int row = step0 + u - member;
                    uint32_t leftH = __shfl_up_sync(kFull, edgeH, 1, G);
                    uint32_t leftI = __shfl_up_sync(kFull, edgeI, 1, G);
                    uint32_t trA = 0, trB = 0;
                    ProfileRow<C> entries[PROFILE ? 2 : 1];
                    if (PROFILE) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            // A row outside the pair reads its nearest letter: no cell that counts uses it.
                            const int r = min(max(row, 1), max(rows[h], 1));
                            const uint32_t letter =
                                s < strips[h] ? letter_at<8>(p.tape, sh[h].first_word, uint32_t(backwards ? rows[h] - r : r - 1))
                                              : 0u;
                            entries[PROFILE ? h : 0] = profile[int(h * t.size + letter) * G];
                        }
                    } else {
                        trA = rows8[codes[0] & 3u];
                        trB = rows8[codes[1] & 3u];
                        codes[0] >>= 2;
                        codes[1] >>= 2;
                    }
                    if (member == 0) {
                        if (s == 0) {
                            const int r = max(row, 0);
                            const int32_t a = free_edge(r, free_rs[0], open, extend) - r * extend;
                            const int32_t b = free_edge(r, free_rs[1], open, extend) - r * extend;
                            leftH = halves(a, b);
                            leftI = halves(a + first_gap, b + first_gap);
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
                        uint32_t I = leftI, left = leftH, last_column = 0;
#pragma unroll
                        for (int k = 0; k < C; ++k) {
                            const uint32_t sub = PROFILE ? profile_entry(entries[0], entries[PROFILE ? 1 : 0], k)
                                                         : uint32_t(prmt(trA, trB, sel[PROFILE ? 0 : k]));
                            const uint32_t Hup = H[k];
                            const uint32_t Dn = __viaddmax_s16x2(Hup, opening2, D[k]);
                            const uint32_t X = __viaddmax_s16x2(diag, sub, Dn);
                            I = __viaddmax_s16x2(left, opening2, I);
                            left = X;
                            diag = Hup;
                            H[k] = __vimax3_s16x2(X, I, X);
                            D[k] = Dn;
                            last_column |= H[k] & last[k];
                        }
                        edgeH = H[C - 1];
                        edgeI = I;
                        if (member == G - 1 && s + 1 < warp_strips)
                            p.carry[slot * p.carry_stride + row] = make_int2(int32_t(edgeH), int32_t(edgeI));
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            if (holds_last[h] && row >= first_end[h] && row <= rows[h])
                                offer(h, (h == 0 ? low_of(last_column) : high_of(last_column)) + (row + cols[h]) * extend,
                                      row, cols[h]);
                        if (p.free_query_end > 0) {
#pragma unroll
                            for (int h = 0; h < 2; ++h)
                                if (s < strips[h] && row == rows[h]) {
#pragma unroll
                                    for (int k = 0; k < C; ++k) {
                                        const int column = first + k + 1;
                                        if (column <= cols[h] && column >= cols[h] - min(p.free_query_end, cols[h]))
                                            offer(h, (h == 0 ? low_of(H[k]) : high_of(H[k])) + (row + column) * extend,
                                                  row, column);
                                    }
                                }
                        }
                    }
                }
            }
            __syncwarp();
        }

        // The best end of the group's lanes, then the borders' own ends (a free end reaching them).
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int span = 1; span < G; span <<= 1) {
                const int32_t their_value = __shfl_xor_sync(kFull, best[h], span, G);
                const int their_row = __shfl_xor_sync(kFull, best_row[h], span, G);
                const int their_col = __shfl_xor_sync(kFull, best_col[h], span, G);
                offer(h, their_value, their_row, their_col);
            }
            if (live[h] && member == 0) {
                if (rows[h] == 0 || cols[h] == 0) {
                    // A prefix swept back may have an empty side.
                    int64_t at = 0;
                    empty_side_end(rows[h], cols[h], free_rs[h], min(p.free_reference_end, rows[h]),
                                   min(p.free_query_start, cols[h]), min(p.free_query_end, cols[h]), highest, open,
                                   extend, best[h], at);
                    best_row[h] = int(at >> 32);
                    best_col[h] = int(at & 0xffffffff);
                } else {
                    if (cols[h] <= p.free_query_end)
                        offer(h, free_edge(rows[h], free_rs[h], open, extend), rows[h], 0);
                    if (rows[h] <= p.free_reference_end)
                        offer(h, free_edge(cols[h], min(p.free_query_start, cols[h]), open, extend), 0, cols[h]);
                }
                p.scores[pair[h]] = best[h];
                if (p.free_ends_out)
                    p.free_ends_out[pair[h] - p.first_pair] = (int64_t(best_row[h]) << 32) | int64_t(best_col[h]);
            }
        }
    }
}

// An extension's stop (scored.mojo:69-100 and 272-300, FROM_ORIGIN: the best cell anywhere above zero, of equal ones
// the furthest along both sequences together, then along the reference) of two pairs a group of G lanes, in 16-bit
// halves, no letter free. Each place's cells of a row join a key a pair, its value over its row, that moves one
// place left a row with its anti-diagonal (row + column), from a lane's place 0 on to the place before: the lane
// that starts the group then holds the strip's whole part of one anti-diagonal a row, where later rows win ties,
// and it alone takes it further. With p.diagonals it goes to that anti-diagonal's word by an atomic maximum (a
// Z-drop reads them in order); without, to the lane's best, later anti-diagonals winning ties. After the last row
// each lane takes the keys it holds further itself. (A compare and an atomic a cell in 32 bits held 10,000 pairs
// of 450 letters for 17.8 ms; an atomic a lane a row made their call 9.9 ms against 9.3.)
//
// A row's key is bits 16-31 the cell, shifted as held, bits 0-15 the row; on one anti-diagonal every cell's
// shift is the same. Columns past a pair's end join with a weight below every real key. Eight places a lane
// keep both pairs' keys and weights in registers.
template <int G, int C, int BITS = 2>
__global__ void __launch_bounds__(kBlock, 2) extension_pairs_kernel(KernelArgs p, TableArgs t,
                                                                   const int32_t *__restrict__ table32) {
    constexpr int W = G * C;
    constexpr int GPW = 32 / G;
    // A real cell, held shifted, lies within two openings (4,000) below zero and 15,000 above, so real keys are at
    // least kLeast; a key past a pair's columns (kPast added) or rows (kBelow in place of its cell) lies below
    // that, and both together above INT32_MIN.
    constexpr int32_t kNoKey = INT32_MIN, kLeast = -4576 * 65536, kPast = -1400000000;
    constexpr uint32_t kBelow = 0xE0000000u;
    constexpr bool PROFILE = BITS == 8;
    __shared__ uint32_t rows8[4];
    __shared__ int8_t table8[PROFILE ? 32 * 32 : 1];
    if (threadIdx.x < 4) rows8[threadIdx.x] = t.rows8[threadIdx.x];
    if (PROFILE) load_table8(table8, table32, 0);
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
    const int64_t slot = int64_t(warp) * GPW + group;
    const uint32_t opening2 = halves(opening, opening), top_gap2 = halves(opening + first_gap, opening + first_gap);
    const bool backwards = p.extents != nullptr;

    for (uint32_t item0 = p.begin + uint32_t(warp) * 2 * GPW; item0 < p.end; item0 += uint32_t(warps) * 2 * GPW) {
        const uint32_t item = item0 + 2 * group;
        bool live[2];
        uint32_t pair[2] = {0, 0};
        PairShape sh[2] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        int rows[2], cols[2], strips[2];
        int64_t words[2] = {0, 0};
        // Each half's best so far: a true score, its anti-diagonal and its row.
        int32_t best[2] = {0, 0};
        int best_along[2] = {0, 0}, best_row[2] = {0, 0};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            live[h] = item + h < p.end;
            if (live[h]) {
                pair[h] = p.order[item + h];
                sh[h] = p.shapes[pair[h]];
                if (p.diagonals) words[h] = p.diagonal_offsets[pair[h] - p.first_pair];
            }
            rows[h] = int(sh[h].rows);
            cols[h] = int(sh[h].columns);
            strips[h] = live[h] && rows[h] > 0 && cols[h] > 0 ? (cols[h] + W - 1) / W : 0;
        }
        const int warp_strips = warp_max(max(strips[0], strips[1]));
        auto offer = [&](int h, int32_t value, int along, int row) {
            if (value > best[h] || (value == best[h] && value > 0 &&
                                    (along > best_along[h] || (along == best_along[h] && row > best_row[h])))) {
                best[h] = value;
                best_along[h] = along;
                best_row[h] = row;
            }
        };

        for (int s = 0; s < warp_strips; ++s) {
            const int first = s * W + member * C;
            uint32_t sel[PROFILE ? 1 : C];
            int32_t weight[2][C], key[2][C];
            if (PROFILE) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                    fill_profile<C>(profile + h * t.size * G, G, t.size, table8,
                                    s < strips[h] ? min(max(cols[h] - first, 0), C) : 0, [&](int k) {
                                        const int col = first + k;
                                        return letter_at<8>(p.tape, sh[h].second_word,
                                                            uint32_t(backwards ? cols[h] - 1 - col : col));
                                    });
            }
#pragma unroll
            for (int k = 0; k < C; ++k) {
                uint32_t half_sel[2] = {kPadHalf, kPadHalf};
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int col = first + k;
                    const bool inside = s < strips[h] && col < cols[h];
                    if (inside && !PROFILE) {
                        const uint32_t y =
                            letter_at<2>(p.tape, sh[h].second_word, uint32_t(backwards ? cols[h] - 1 - col : col));
                        half_sel[h] = h == 0 ? half_selector_a(y) : half_selector_b(y);
                    }
                    weight[h][k] = inside ? 0 : kPast;
                    key[h][k] = kNoKey;
                }
                if (!PROFILE) sel[PROFILE ? 0 : k] = pair_selector(half_sel[0], half_sel[1]);
            }
            uint32_t H[C], D[C];
#pragma unroll
            for (int k = 0; k < C; ++k) {
                H[k] = opening2;
                D[k] = top_gap2;
            }
            uint32_t edgeH = opening2, edgeI = top_gap2;
            uint32_t above_left = first == 0 ? 0u : opening2;
            int group_rows = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) group_rows = max(group_rows, s < strips[h] ? rows[h] : 0);
            const int steps = group_rows > 0 ? group_rows - 1 + G : 0;
            const int warp_steps = warp_max(steps);
            // A key of pair h's anti-diagonal `along`, taken further.
            auto send = [&](int h, int32_t whole, int along) {
                if (whole < kLeast) return;
                if (p.diagonals)
                    atomicMax(reinterpret_cast<uint32_t *>(p.diagonals + words[h] + along), uint32_t(whole) ^ 0x80000000u);
                else
                    offer(h, (whole >> 16) + along * extend, along, whole & 0xFFFF);
            };

            for (int step0 = 1; step0 <= warp_steps; step0 += 16) {
                uint32_t codes[2] = {0, 0};
#pragma unroll
                for (int h = 0; h < (PROFILE ? 0 : 2); ++h)
                    codes[h] = sixteen_rows(p.tape, sh[h].first_word, live[h] ? rows[h] : 0, step0 - member, backwards);
#pragma unroll 2
                for (int u = 0; u < 16; ++u) {
                    const int row = step0 + u - member;
                    // The next lane's place 0 one row up, on the anti-diagonal of this lane's last place there.
                    const int32_t further_a = __shfl_down_sync(kFull, key[0][0], 1, G);
                    const int32_t further_b = __shfl_down_sync(kFull, key[1][0], 1, G);
                    uint32_t leftH = __shfl_up_sync(kFull, edgeH, 1, G);
                    uint32_t leftI = __shfl_up_sync(kFull, edgeI, 1, G);
                    uint32_t trA = 0, trB = 0;
                    ProfileRow<C> entries[PROFILE ? 2 : 1];
                    if (PROFILE) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            // A row outside the pair reads its nearest letter: no cell that counts uses it.
                            const int r = min(max(row, 1), max(rows[h], 1));
                            const uint32_t letter =
                                s < strips[h] ? letter_at<8>(p.tape, sh[h].first_word, uint32_t(backwards ? rows[h] - r : r - 1))
                                              : 0u;
                            entries[PROFILE ? h : 0] = profile[int(h * t.size + letter) * G];
                        }
                    } else {
                        trA = rows8[codes[0] & 3u];
                        trB = rows8[codes[1] & 3u];
                        codes[0] >>= 2;
                        codes[1] >>= 2;
                    }
                    if (member == 0) {
                        if (s == 0) {
                            leftH = opening2;
                            leftI = top_gap2;
                        } else {
                            const int r = min(max(row, 0), group_rows);
                            const int2 c = p.carry[slot * p.carry_stride + r];
                            leftH = uint32_t(c.x);
                            leftI = uint32_t(c.y);
                        }
                    }
                    uint32_t diag = above_left;
                    above_left = leftH;
                    // Every lane of the group goes on until its last has swept the last row: its keys move with them.
                    if (row >= 1 && row + member <= steps) {
                        if (member < G - 1) {
                            key[0][C - 1] = max(key[0][C - 1], further_a);
                            key[1][C - 1] = max(key[1][C - 1], further_b);
                        }
                        const uint32_t stamp = uint32_t(row) | kBelow;
                        const uint32_t key_a = row <= rows[0] ? 0x1054u : 0x7654u;
                        const uint32_t key_b = row <= rows[1] ? 0x3254u : 0x7654u;
                        uint32_t I = leftI, left = leftH;
#pragma unroll
                        for (int k = 0; k < C; ++k) {
                            const uint32_t sub = PROFILE ? profile_entry(entries[0], entries[PROFILE ? 1 : 0], k)
                                                         : uint32_t(prmt(trA, trB, sel[PROFILE ? 0 : k]));
                            const uint32_t Hup = H[k];
                            const uint32_t Dn = __viaddmax_s16x2(Hup, opening2, D[k]);
                            const uint32_t X = __viaddmax_s16x2(diag, sub, Dn);
                            I = __viaddmax_s16x2(left, opening2, I);
                            left = X;
                            diag = Hup;
                            H[k] = __vimax3_s16x2(X, I, X);
                            D[k] = Dn;
                            const int32_t later_a = k + 1 < C ? key[0][k + 1] : kNoKey;
                            const int32_t later_b = k + 1 < C ? key[1][k + 1] : kNoKey;
                            key[0][k] = __viaddmax_s32(prmt(H[k], stamp, key_a), weight[0][k], later_a);
                            key[1][k] = __viaddmax_s32(prmt(H[k], stamp, key_b), weight[1][k], later_b);
                        }
                        edgeH = H[C - 1];
                        edgeI = I;
                        if (member == G - 1 && s + 1 < warp_strips && row <= group_rows)
                            p.carry[slot * p.carry_stride + row] = make_int2(int32_t(edgeH), int32_t(edgeI));
                        if (member == 0) {
                            send(0, key[0][0], row + first + 1);
                            send(1, key[1][0], row + first + 1);
                        }
                    }
                }
            }
            if (steps > 0) {
#pragma unroll
                for (int k = 0; k < C; ++k) {
                    send(0, key[0][k], steps - member + first + k + 1);
                    send(1, key[1][k], steps - member + first + k + 1);
                }
            }
            __syncwarp();
        }

#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
            for (int span = 1; span < G; span <<= 1) {
                const int32_t their_value = __shfl_xor_sync(kFull, best[h], span, G);
                const int their_along = __shfl_xor_sync(kFull, best_along[h], span, G);
                const int their_row = __shfl_xor_sync(kFull, best_row[h], span, G);
                offer(h, their_value, their_along, their_row);
            }
            if (live[h] && member == 0) {
                p.scores[pair[h]] = best[h];
                p.free_ends_out[pair[h] - p.first_pair] =
                    (int64_t(best_row[h]) << 32) | int64_t(best_along[h] - best_row[h]);
            }
        }
    }
}

}  // namespace sweep
}  // namespace dinara
