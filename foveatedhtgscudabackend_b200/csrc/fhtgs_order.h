// The blend's work order: the words of its block items, the decision taken per tile and the place
// every item gets in the merged list.  No CUDA dependency, so that it can be compiled and
// exercised alone.
//
// One list of block items, longest estimated duration first, so that the serial walks of the
// long lists start early and the short ones fill the end:
//   full    a full-resolution tile, two pixels a thread
//   half    the upper or lower half of a full-resolution tile, one pixel a thread: the tiles
//           whose walk alone would outlast the frame's mean work per block
//   low     four periphery tiles, halves of them, or ring-mode quarter tiles with long lists, one
//           per warp
//   quarter sixteen other quarter tiles, four per warp
// An item word is kind << 29 | view << 21 | index into the view's work_full list, or kind << 29 |
// item number for the last two, whose tiles lie in a second list, the runs (the same word, with
// the index into work_low; kind kItemQuarter: a quarter tile that a warp blends alone), longest first:
// the entries of all views' low items, then those of the quarter items.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define FHTGS_HD __host__ __device__ __forceinline__
#else
#define FHTGS_HD inline
#endif

namespace fhtgs {

constexpr int kCostBuckets = 130;                // per tile class: estimated duration in quarter octaves
constexpr int kOrderBuckets = 3 * kCostBuckets;  // quarter (class 0), low (1), full-resolution (2)

constexpr uint32_t kItemFull = 0u, kItemHalf = 1u /* and 2 */, kItemLow = 3u, kItemQuarter = 4u;
constexpr int kItemKindShift = 29, kItemViewShift = 21;
constexpr uint32_t kItemIndexMask = (1u << kItemViewShift) - 1u;
constexpr uint32_t kItemNumberMask = (1u << kItemKindShift) - 1u;
FHTGS_HD int item_view(uint32_t packed) { return static_cast<int>((packed >> kItemViewShift) & 255u); }
FHTGS_HD uint32_t item_index(uint32_t packed) { return packed & kItemIndexMask; }
// Tiles (or halves) of a low / quarter item.
constexpr uint32_t kLowTiles = 4, kQuarterTiles = 16;

// Estimated duration of an item in list entries of a full item: per entry of its (longest) list,
// plus the item's fixed cost (about 5 us).  Measured per entry at 1 / 5 blocks per SM (K = 8): a full
// item 69-88 / 167-170 ns, a half item 30-49 / 47-91, a low item of whole tiles 137-196 / 303-339, of
// halves 72-95 / 134-136 (4 blocks), a quarter item 331-382 / 462-534, of quarter tiles alone 117-120 /
// 151 (3 blocks).  The factors are those ratios where the frames are fastest: half 0.6 (0.5: 6M with
// rings 14.26 -> 16.09 ms of blend, the stereo frame with rings 2.60 -> 2.77), low 1.6 (1.4: 14.82 and
// 2.62; 2.0: 15.62 and 2.77), quarter 4 (2.5: 64 mixed views with rings 9.47 instead of 7.45 ms), alone
// 1.2 (1.6: 16 mixed views 5.61 instead of 4.47 ms).
constexpr float kCostHalf = 0.6f, kCostLow = 1.6f, kCostQuarter = 4.0f, kCostAlone = 1.2f, kCostItem = 32.0f;
// A full-resolution tile becomes two half items when its list is longer than this share of the
// frame's instances per SM: its walk would then outlast the frame at five blocks per SM.  (Blend of
// the stereo frame in us at 0.06 / 0.1 / 0.13 / 0.16 / 0.2 / 0.26 / never: K = 8 3639 / 3507 / 3369 /
// 3256 / 3374 / 3450 / 3436, K = 16 4725 / 4633 / 4549 / 4448 / 4318 / 4284 / 4286, K = 32 7509 / 7492 /
// 7445 / 7374 / 7268 / 7241 / 7240; without halves the plain view takes 287 instead of 190, 300k at
// 1920x1080 593 instead of 430 at K = 8, 656 / 461 at K = 16, 996 / 625 at K = 32.  At K >= 16, where
// fewer blocks are resident, a larger share would be 2-4 % better on frames of many tiles.)
constexpr float kHalfShare = 0.16f;

// What the order decides about a tile: its bucket (class above duration bucket), and whether it
// becomes two half items or, a quarter tile, an entry of a low item.  Decided once, when the buckets
// are counted, and kept: the buckets' runs hold exactly the counted entries, whatever the
// estimate's rounding.
constexpr uint16_t kOrderSplit = 0xffffu;  // a tile of the split blend: no entry
FHTGS_HD uint16_t order_word(int bucket, bool halves, bool alone) {
    return static_cast<uint16_t>(bucket | (halves ? 0x8000 : 0) | (alone ? 0x4000 : 0));
}
FHTGS_HD int order_bucket(uint16_t word) { return word & 0x3fff; }
FHTGS_HD bool order_alone(uint16_t word) { return (word & 0x4000) != 0; }
FHTGS_HD uint32_t order_entries(uint16_t word) { return (word & 0x8000) ? 2u : 1u; }

// The frame's totals.  `base[b]`: entries in buckets above b (all classes, descending).
struct OrderTotals {
    const uint32_t* base;
    uint32_t all, full, low, quarter;  // entries

    FHTGS_HD OrderTotals(const uint32_t* base_, uint32_t all_) : base(base_), all(all_) {
        full = base[2 * kCostBuckets - 1];
        low = base[kCostBuckets - 1] - full;
        quarter = all - full - low;
    }
    FHTGS_HD uint32_t items() const {
        return full + (low + kLowTiles - 1) / kLowTiles + (quarter + kQuarterTiles - 1) / kQuarterTiles;
    }
    // entries of a class in duration buckets >= d (d = kCostBuckets: none)
    FHTGS_HD uint32_t at_least(int cls, int d) const {
        const uint32_t start = cls == 2 ? 0u : cls == 1 ? full : full + low;
        if (d >= kCostBuckets) return 0u;
        const int k = cls * kCostBuckets + d;
        return (k > 0 ? base[k - 1] : all) - start;
    }
    FHTGS_HD uint32_t low_items(int d) const { return (at_least(1, d) + kLowTiles - 1) / kLowTiles; }
    FHTGS_HD uint32_t quarter_items(int d) const { return (at_least(0, d) + kQuarterTiles - 1) / kQuarterTiles; }

    // Writes the entries of one tile.  `at`: its place among all entries, classes one after the
    // other.  The place of a block item in the merged list is its place in its own class plus the
    // items of the other classes in longer buckets (equal buckets: full, low, quarter).
    FHTGS_HD void put(uint16_t word, uint32_t at, uint32_t packed, uint32_t* out, uint32_t* runs) const {
        const int b = order_bucket(word), cls = b / kCostBuckets, d = b - cls * kCostBuckets;
        const bool halves = order_entries(word) == 2u;
        const uint32_t kind = halves ? kItemHalf : order_alone(word) ? kItemQuarter : kItemFull;
        uint32_t* list = cls == 2 ? out + low_items(d + 1) + quarter_items(d + 1) + at : runs + (at - full);
        list[0] = (kind << kItemKindShift) | packed;
        if (halves) list[1] = ((kind + 1u) << kItemKindShift) | packed;
        if (cls == 2) return;
        const uint32_t per = cls == 1 ? kLowTiles : kQuarterTiles, k = at - full - (cls == 1 ? 0u : low);
        const uint32_t first = (k + per - 1) / per * per;
        if (first < k + order_entries(word))  // the first tile (or half) of an item
            out[first / per + at_least(2, d) + (cls == 1 ? quarter_items(d + 1) : low_items(d))] =
                ((cls == 1 ? kItemLow : kItemQuarter) << kItemKindShift) | (first / per);
    }
};

}  // namespace fhtgs
