// Packing the caller's letters on the device, and the longest-first schedule of a batch.
#pragma once

#include "affine.cuh"

namespace dinara {

// Packs pairs [first_pair, first_pair + count) of the device ASCII tape (offsets: 2 entries a pair and
// one more, from the batch's first letter) into their places on the batch's `tape`, each letter through
// `codes` (256 entries, 255 for a byte outside the alphabet), `bits` a letter; writes each pair's shape
// and flags a pair holding an unknown byte. Packing a batch a range at a time gives the tape, shapes and
// flags packing it whole gives.
void pack_pairs(dinara_gpu *gpu, const uint8_t *letters_device, const int64_t *offsets_device, int64_t first_pair,
                int64_t count, const uint8_t *codes_device, int bits, uint32_t *tape, PairShape *shapes,
                uint8_t *unknown, const int64_t *spans = nullptr);

// A batch's sweep order: pairs by class, classes in descending order, then strips and rows descending.
// Classes: the whole-matrix shape classes 0-4 (affine_shape_for with `record`); with `band` the proven
// band, kBandClass, and of those the pairs whose rows and columns sum to at most `limits.band`,
// kBandPairsClass, for the 16-bit pair band sweep; the whole-matrix pairs the 16-bit pair score sweep
// takes, kWholePairsClass plus the shape class; long pairs one block sweeps, kWideClass; and, recording,
// pairs whose widening band proved a width (`limits.band_widths`), kBandRecordClass. `order` is valid on
// the device until the next call.
constexpr int kClasses = 18;
constexpr int kBandClass = 5;
constexpr int kBandPairsClass = 6;
constexpr int kWholePairsClass = 7;
constexpr int kWideClass = kWholePairsClass + kPairShapes;
constexpr int kBandRecordClass = kWideClass + 1;
static_assert(kBandRecordClass + 1 == kClasses && kClasses <= 32, "a class is five bits of a key");
// A context's counters on the device (class_counts): the launches' own in the first words, a schedule's classes
// from kScheduleCounts on.
constexpr int kClassCounters = 64, kScheduleCounts = 32;
// A pair a whole block sweeps (kWideClass), scoring without a CIGAR: at least this tall and this wide.
constexpr uint32_t kWideRows = 4096, kWideColumns = 2048;
// With the 16-bit strips: a pair of two strips or more, each way. (In 32 bits, a warp a pair, and in strips: 50 pairs of
// 1,100 letters 2.98 and 0.58 ms, 500 3.53 and 2.81, 5,000 7.45 and 4.61; of 2,500 letters 12.0 and 1.6, 12.6 and 9.3,
// 25.1 and 19.1.)
constexpr uint32_t kLongSide = 1024 + 1;
struct Schedule {
    const uint32_t *order;
    int64_t counts[kClasses];
    int skip = -1;  // a class the whole-matrix launches leave out
};

// Which pairs the 16-bit pair sweeps take: band pairs whose rows and columns sum to at most `band`; and,
// scoring without a CIGAR, non-empty whole-matrix pairs with best x swept columns + rows x row_step at
// most `whole` (local) or whose rows and swept columns are each at most half of it (global). Zero takes none. With `wide`,
// scoring without a CIGAR, whole-matrix pairs of at least kWideRows x kWideColumns go to kWideClass.
struct PairLimits {
    int32_t band = 0;
    int32_t whole = 0;
    int32_t local = 0;
    int32_t fine = 0;    // the score sweeps' own shapes past 320 columns too (pair_shape_for)
    int32_t record = 0;  // `whole` holds the recording sweep's pairs (else the score sweeps')
    int32_t hits = 0;    // recording: of hits' rows, so only pairs whose hits a score sweep has found
    int32_t columns = 0; // above 0: only pairs of at most so many columns
    int32_t wide = 0;
    // Scoring without a CIGAR, globally: the 16-bit strips of a long pair serve the batch's table. Then pairs of
    // at least kLongSide x kLongSide that no 16-bit pair sweep takes go to kWideClass too.
    int32_t long_strips = 0;
    // Local: a pair fits when best x swept columns + rows x row_step is at most `whole`.
    int32_t best = 1;
    int32_t row_step = 0;
    // Recording: each pair's proven band width by pair - band_first (0: none), when given; a pair with one
    // goes to kBandRecordClass.
    const int32_t *band_widths = nullptr;
    int64_t band_first = 0;
};

// Whether a pair takes the 16-bit pair sweep of shape `shape` (`record`: recording).
__host__ __device__ inline bool takes_pairs16(const PairLimits &limits, uint32_t rows, uint32_t columns, int shape,
                                              bool record) {
    if (limits.whole <= 0 || record != (limits.record != 0) || rows == 0 || columns == 0) return false;
    if (limits.columns > 0 && columns > uint32_t(limits.columns)) return false;
    // The score sweeps left a long pair (kWideClass) its whole shape and no hit.
    if (limits.hits && limits.wide && rows >= kWideRows && columns >= kWideColumns) return false;
    const uint32_t width = uint32_t(affine_lanes(shape) * affine_columns(shape));
    const int64_t swept = int64_t((columns + width - 1) / width) * width;
    return limits.local ? swept * limits.best + int64_t(rows) * limits.row_step <= limits.whole
                        : 2 * swept <= limits.whole && 2 * int64_t(rows) <= limits.whole;
}

// The order of pairs [first, first + count), or of the `count` pairs listed in `list` (device) when given.
Schedule schedule(dinara_gpu *gpu, const PairShape *shapes, const uint32_t *list, int64_t first, int64_t count,
                  bool record, bool band, PairLimits limits = PairLimits());

}  // namespace dinara
