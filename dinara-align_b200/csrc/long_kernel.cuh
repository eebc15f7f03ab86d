// Scores of one long pair a block, or a cluster of blocks, by warps that each sweep a strip of columns in 16-bit
// halves.
#pragma once

#include "affine_kernel.cuh"

namespace dinara {
namespace sweep {

// A strip is 64 virtual lanes of C columns (16, or 8 for a batch of few pairs): a lane's low halves hold C columns and
// its high halves the next C, one row behind, so each DPX instruction on 16-bit pairs moves two cells of the one
// pair.
constexpr int kLongStrip = 1024;
constexpr int kLongWarps = 8;     // most warps a block without clusters; a launch may take fewer
constexpr int kLongChunk = 32;    // steps of a chunk: a strip's letters and left column are read, and its base moved, once
constexpr int kLongChunks = 2;    // chunks between barriers
constexpr int kLongCluster = 8;   // blocks a cluster
__host__ __device__ constexpr int long_cluster_warps(int C) { return C == 8 ? 4 : 2; }  // and each one's warps

// A lane's halves hold its cells less its base, a true 32-bit value that follows them: at each chunk the
// lane's own middle cell becomes the base. Within a lane's 32 columns two reached cells of a row differ
// by at most 31 steps K (K: the largest shifted entry plus a gap's opening, in size), a cell's value
// moves at most K a row, and a lane whose base was last set when its strip began is at most 64 rows from
// its first row, so every reached half lies within (32 + 33 + 64) K of zero: within 12,900 for K up to
// kLongStep. An unreached half is at least kLongFloor and below every true value of its cell, since a true
// value lies no further than that below its base; kLongFloor less the largest change of base stays above
// -32,768. So no half overflows.
constexpr int32_t kLongStep = 100;
constexpr int32_t kLongFloor = -18000;

struct LongArgs {
    const uint32_t *tape;
    const PairShape *shapes;
    const uint32_t *order;       // the pairs, longest first
    const int32_t *band_widths;  // by item; null: whole matrices
    uint32_t count;
    int32_t open, extend;
    uint32_t rows8[4];           // the shifted table, a byte an entry
    int32_t *scores;
    int2 *carry;                 // a column of (score, insertion) a pair in flight
    int64_t carry_stride;
};

// Every thread of a cluster's blocks meets here; what each wrote before, the others read after.
__device__ __forceinline__ void cluster_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// A strip's rows: those its columns share with the band [low, high] of diagonals (column less row).
template <int STRIP>
__device__ __forceinline__ int long_first_row(int s, int high) {
    return max(1, s * STRIP + 1 - high);
}
template <int STRIP>
__device__ __forceinline__ int long_last_row(int s, int rows, int columns, int low) {
    return min(rows, min((s + 1) * STRIP, columns) - low);
}

// Stores `value` at `place` in this block's shared memory, or in block `rank` of its cluster's.
template <bool CLUSTER>
__device__ __forceinline__ void leave_word(int *place, int rank, int value) {
    if (CLUSTER) {
        uint32_t remote;
        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                     : "=r"(remote)
                     : "r"(uint32_t(__cvta_generic_to_shared(place))), "r"(rank));
        asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(value) : "memory");
    } else {
        *reinterpret_cast<volatile int *>(place) = value;
    }
}

// The whole or banded score of one pair a block, or with CLUSTER a cluster of eight blocks (score_groups.mojo's
// recurrence, cells shifted by (row + column) * extend). Warp w of them sweeps strips w, w + warps, ...: a strip's
// virtual lane v runs one row behind lane v - 1, whose last column reaches it from the lane's own low half or by one
// shuffle, and the column left of a strip comes from the strip before through `carry`, a chunk of 32 rows at a time.
// Warps meet at one barrier every two chunks and leave how far they are with the warp of the next strip; a warp
// takes a chunk when the strip before had, by the last barrier, left every row it reads, else waits for the next.
// Strips of a band start lower one after another, so about (width + 64 C) / (64 C + 100) of them run at once.
//
// Each step is C x 5 instructions of the DPX and permute pipe for 32 x 2 C cells a warp (16-bit pairs run at the
// 32-bit rate), so an SM's bound is 25.6 cells a cycle against 12.8 in 32 bits; a barrier a row (the block-wide
// 32-bit sweep, affine_wide_kernel) and its strips of 4,096 columns, which sweep 4,096 rows beyond a band's width,
// are what this one does without.
//
// Eight warps on one SM share its four issue ports, and a pair of 50,000 letters keeps them all for each of its
// rows; a batch too small to fill the GPU with pairs takes a cluster a pair instead, neighbouring strips on
// different SMs, a warp or less a port. Its warps meet at a cluster barrier, whose release and acquire order the
// column in global memory and the words left in one another's shared memory. A batch smaller still, whose ports wait
// for a row's chain of insertions through a lane's C columns, takes C = 8 and twice the warps (sweep_long).
//
// A banded strip sweeps its rows alone, every cell above or left of them unreached; the score is then the best over
// paths within the swept rows, the whole matrix's when the band proves it (band_proves_width).
template <bool CLUSTER, int C>
__global__ void __launch_bounds__(32 * (CLUSTER ? long_cluster_warps(C) : kLongWarps),
                                  CLUSTER ? 16 / long_cluster_warps(C) : 2) affine_long_kernel(LongArgs p) {
    constexpr int STRIP = 64 * C;
    __shared__ uint32_t rows8[4];
    // By round parity: for each of the block's warps, the strip and steps of the warp before it; and whether the
    // last strip is done.
    __shared__ int left_by[2][CLUSTER ? long_cluster_warps(C) : kLongWarps][2], finished[2];
    if (threadIdx.x < 4) rows8[threadIdx.x] = p.rows8[threadIdx.x];

    const int lane = threadIdx.x & 31;
    const uint32_t first_item = CLUSTER ? blockIdx.x / kLongCluster : blockIdx.x;
    const uint32_t items_apart = CLUSTER ? gridDim.x / kLongCluster : gridDim.x;
    const int rank = CLUSTER ? int(blockIdx.x % kLongCluster) : 0;  // clusters are consecutive blocks
    const int warps = int(blockDim.x >> 5) * (CLUSTER ? kLongCluster : 1);
    const int warp = CLUSTER ? int(threadIdx.x >> 5) * kLongCluster + rank : int(threadIdx.x >> 5);
    const int own = int(threadIdx.x >> 5);  // the warp's place in its block, and the next strip's warp's
    const int next_warp = (warp + 1) % warps;
    const int next_own = CLUSTER ? next_warp / kLongCluster : next_warp, next_rank = CLUSTER ? next_warp % kLongCluster : 0;
    auto meet = [&] {
        if (CLUSTER)
            cluster_barrier();
        else
            __syncthreads();
    };
    const int32_t opening = p.open - p.extend;
    const int32_t first_gap = p.open + p.extend;
    const uint32_t opening2 = halves(opening, opening), floor2 = halves(kLongFloor, kLongFloor);
    int2 *carry = p.carry + int64_t(first_item) * p.carry_stride;

    for (uint32_t item = first_item; item < p.count; item += items_apart) {
        const uint32_t pair = p.order[item];
        const PairShape sh = p.shapes[pair];
        const int rows = int(sh.rows), cols = int(sh.columns);
        const int strips = (cols + STRIP - 1) / STRIP;
        // The band's diagonals; a pair whose band cannot hold both ends is swept whole.
        int low = -rows, high = cols;
        if (p.band_widths) {
            const int32_t width = p.band_widths[item];
            const int32_t from = band_low_for_width(rows, cols, width);
            if (from != INT32_MIN) {
                low = from;
                high = from + width - 1;
            }
        }
        meet();  // the last pair's words and column are read
        if (lane < 2) {
            left_by[lane][own][0] = -1;
            left_by[lane][own][1] = 0;
            finished[lane] = 0;
        }
        meet();

        // The strip under this warp: its rows, its state and the steps it has done.
        int strip = warp, done = 0;
        int first_row = 0, last_row = 0, previous_last = 0, total = 0;
        uint32_t sel[C], H[C], D[C];
        uint32_t edgeH = 0, edgeI = 0, above_left = 0, send = 0, before = 0;
        int32_t base = 0;
        // Every round some strip's chunk is ready (the first unfinished strip's always is), so the rounds
        // end within the sum of all strips' chunks: when the last strip is done, which every warp reads as of the
        // same barrier.
        for (int round = 0;; ++round) {
            const int before_round = (round + 1) & 1;
            if (*const_cast<volatile int *>(&finished[before_round])) break;
            const int their_strip = *const_cast<volatile int *>(&left_by[before_round][own][0]);
            const int their_done = *const_cast<volatile int *>(&left_by[before_round][own][1]);
            for (int chunk = 0; chunk < kLongChunks; ++chunk) {
                bool ready = strip < strips;
                if (ready && done == 0) {
                    first_row = long_first_row<STRIP>(strip, high);
                    last_row = long_last_row<STRIP>(strip, rows, cols, low);
                    previous_last = strip > 0 ? long_last_row<STRIP>(strip - 1, rows, cols, low) : rows;
                    total = last_row - first_row + 1 + 63;
                }
                if (ready && strip > 0) {
                    // The strip before has left every row of this chunk (its virtual lane 63 leaves row r at its
                    // step r - its first row + 64) by the last barrier.
                    const int last_read = min(first_row - 1 + done + kLongChunk, previous_last);
                    const int needed = last_read - long_first_row<STRIP>(strip - 1, high) + 64;
                    ready = their_strip > strip - 1 || (their_strip == strip - 1 && their_done >= needed);
                }
                if (!ready) break;
                const bool from_top = first_row == 1;
                const int t0 = done + 1;
                if (done == 0) {
                    // A new strip: its columns' selectors, and every lane's base the value its cells start near.
                    static_assert(C == 16 || C == 8, "a lane's letters are two words or one");
                    const int word = strip * (STRIP / 16) + (C / 8) * lane;
                    const int last_word = (cols - 1) >> 4;
                    const uint32_t a = __ldg(p.tape + sh.second_word + min(word, last_word));
                    const uint32_t b = C == 16 ? __ldg(p.tape + sh.second_word + min(word + 1, last_word)) : a >> 16;
#pragma unroll
                    for (int k = 0; k < C; ++k)
                        sel[k] = pair_selector(half_selector_a((a >> (2 * k)) & 3u), half_selector_b((b >> (2 * k)) & 3u));
                    base = from_top ? 0 : carry[first_row - 1].x;
                    send = floor2;
                } else if (done >= 1 + 2 * lane) {
                    // The lane's middle cell becomes its base.
                    const int32_t moved = low_of(H[C - 1]);
                    const uint32_t less = halves(-moved, -moved);
                    base += moved;
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        H[k] = __viaddmax_s16x2(H[k], less, floor2);
                        D[k] = __viaddmax_s16x2(D[k], less, floor2);
                    }
                    edgeH = __viaddmax_s16x2(edgeH, less, floor2);
                    edgeI = __viaddmax_s16x2(edgeI, less, floor2);
                    above_left = __viaddmax_s16x2(above_left, less, floor2);
                    send = __viaddmax_s16x2(send, less, floor2);
                }
                // A value held against this lane's base.
                auto held = [&](int32_t value) { return min(max(value - base, kLongFloor), -kLongFloor); };
                // The lane before's halves, moved to this lane's base.
                const int32_t apart = __shfl_up_sync(kFull, base, 1) - base;
                const uint32_t apart2 = halves(apart, apart);
                // The chunk's rows' letters, and the column left of the strip on its 32 rows (lane i's row for
                // step t0 + i of virtual lane 0).
                uint32_t codes[2];
                {
                    const int start = first_row - 2 + t0 - 2 * lane;  // the first step's row's letter
                    const int word = start >> 4, last_word = (rows - 1) >> 4;
                    uint32_t words[3];
#pragma unroll
                    for (int i = 0; i < 3; ++i)
                        words[i] = __ldg(p.tape + sh.first_word + min(max(word + i, 0), last_word));
                    const uint32_t shift = uint32_t(start & 15) * 2u;
                    codes[0] = __funnelshift_r(words[0], words[1], shift);
                    codes[1] = __funnelshift_r(words[1], words[2], shift);
                }
                uint32_t left_column;
                {
                    const int row = first_row - 1 + t0 + lane;
                    const int32_t lane0_base = __shfl_sync(kFull, base, 0);
                    int2 c = make_int2(opening, opening + first_gap);
                    bool reached = true;
                    if (strip > 0) {
                        reached = row <= previous_last && row <= last_row;
                        if (reached) c = carry[row];
                    }
                    const int32_t h = min(max(c.x - lane0_base, kLongFloor), -kLongFloor);
                    const int32_t i = min(max(c.y - lane0_base, kLongFloor), -kLongFloor);
                    left_column = reached ? halves(h, i) : floor2;
                }
                const bool starting = t0 <= 64;
                const bool leaves = strip + 1 < strips;
                // The corner: its virtual lane reaches the last row at this step.
                const int corner = cols - 1 - strip * STRIP;
                const int corner_step = strip + 1 == strips ? rows - first_row + 1 + corner / C : -1;
                const int32_t top_h = held(opening), top_d = held(opening + first_gap);
#pragma unroll 2
                for (int u = 0; u < kLongChunk; ++u) {
                    const int step = t0 + u;
                    const uint32_t code = codes[0] & 3u;
                    codes[0] = __funnelshift_r(codes[0], codes[1], 2);
                    codes[1] >>= 2;
                    const uint32_t here = rows8[code];
                    const uint32_t from_lane = __viaddmax_s16x2(__shfl_up_sync(kFull, send, 1), apart2, floor2);
                    const uint32_t from_column = __shfl_sync(kFull, left_column, u);
                    const uint32_t received = lane == 0 ? from_column : from_lane;
                    const uint32_t leftH = uint32_t(prmt(received, edgeH, 0x5410u));
                    const uint32_t leftI = uint32_t(prmt(received, edgeI, 0x5432u));
                    if (starting) {
                        if (step == 1 + 2 * lane) {
                            // The low halves' first row: the matrix's top border, or unreached cells above it.
                            const int32_t h = from_top ? top_h : kLongFloor, d = from_top ? top_d : kLongFloor;
                            int32_t corner_value = h;
                            if (lane == 0 && from_top && strip == 0) corner_value = held(0);
                            if (lane == 0 && !from_top) corner_value = held(carry[first_row - 1].x);
#pragma unroll
                            for (int k = 0; k < C; ++k) {
                                H[k] = halves(h, h);
                                D[k] = halves(d, d);
                            }
                            above_left = halves(corner_value, corner_value);
                        } else if (step == 2 + 2 * lane) {
                            // The high halves', a step later.
                            const int32_t h = from_top ? top_h : kLongFloor, d = from_top ? top_d : kLongFloor;
#pragma unroll
                            for (int k = 0; k < C; ++k) {
                                H[k] = (H[k] & 0xFFFFu) | (uint32_t(h) << 16);
                                D[k] = (D[k] & 0xFFFFu) | (uint32_t(d) << 16);
                            }
                            above_left = (above_left & 0xFFFFu) | (uint32_t(h) << 16);
                        }
                    }
                    uint32_t diag = above_left;
                    above_left = leftH;
                    uint32_t I = 0, Xprev = 0;
#pragma unroll
                    for (int k = 0; k < C; ++k) {
                        const uint32_t sub = uint32_t(prmt(here, before, sel[k]));
                        const uint32_t Hup = H[k];
                        const uint32_t Dn = __viaddmax_s16x2(Hup, opening2, D[k]);
                        const uint32_t X = __viaddmax_s16x2(diag, sub, Dn);
                        I = k == 0 ? __viaddmax_s16x2(leftH, opening2, leftI) : __viaddmax_s16x2(Xprev, opening2, I);
                        Xprev = X;
                        diag = Hup;
                        H[k] = __vimax3_s16x2(X, I, X);
                        D[k] = Dn;
                    }
                    before = here;
                    edgeH = H[C - 1];
                    edgeI = I;
                    send = uint32_t(prmt(edgeH, edgeI, 0x7632u));
                    if (leaves && lane == 31) {
                        const int row = first_row - 1 + step - 63;
                        if (row >= first_row && row <= last_row)
                            carry[row] = make_int2(base + low_of(send), base + high_of(send));
                    }
                    if (step == corner_step && lane == corner / (2 * C)) {
                        uint32_t value = 0;
#pragma unroll
                        for (int k = 0; k < C; ++k) value |= H[k] & (0u - uint32_t(k == corner % C));
                        p.scores[pair] = base + ((corner & C) ? high_of(value) : low_of(value)) + (rows + cols) * p.extend;
                    }
                }
                done += kLongChunk;
                if (done < total) continue;
                // The strip is done.
                if (strip + 1 == strips && lane < (CLUSTER ? kLongCluster : 1))
                    leave_word<CLUSTER>(&finished[round & 1], lane, 1);
                strip += warps;
                done = 0;
                break;
            }
            if (lane < 2) leave_word<CLUSTER>(&left_by[round & 1][next_own][lane], next_rank, lane == 0 ? strip : done);
            meet();
        }
    }
}

}  // namespace sweep
}  // namespace dinara
