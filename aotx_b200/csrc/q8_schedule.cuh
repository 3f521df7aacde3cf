// The division of work of the kernels on tensor memory (q8_mid.cu, q8_pair.cu): which pieces - runs of segments of
// a tile - a block, or a pair of blocks, works on, and which others hold the rest of a tile that it finishes.
// On the host as well, for the check of tests/schedule_check.cu.
#pragma once

#include "q8_tile.cuh"

namespace q8 {

// A block's work: pieces of tiles, each the segments [s0, s1) of one tile.
struct MidWork {
    uint32_t tile, s0, s1;     // the piece
    uint32_t next_tile, next_seg, left, segs;
    uint32_t stride;           // from one tile of the block to the next
    uint32_t most;             // segments per piece, at most

    __host__ __device__ __forceinline__ bool next()
    {
        if (left == 0u) {
            return false;
        }
        tile = next_tile;
        s0 = next_seg;
        const uint32_t here = left < most ? left : most;
        s1 = segs - s0 < here ? segs : s0 + here;
        left -= s1 - s0;
        next_seg = s1;
        if (s1 == segs) {
            next_tile += stride;
            next_seg = 0u;
        }
        return true;
    }
};

// The work of block `block` of `grid`.  Clusters (csize above one): one tile each, a run of its segments per block, in
// pieces of at most run_segs (0: one piece).  Else whole tiles in `turns`, or (0) (tile, segment) units dealt evenly,
// the same arithmetic as the decode kernel's; decode_holder names the block that holds a unit.
__host__ __device__ __forceinline__ void mid_deal(MidWork *work, uint32_t block, uint32_t grid, uint32_t csize, uint32_t crank,
                                                  uint32_t tiles, uint32_t segs, uint32_t turns, uint32_t run_segs)
{
    work->segs = segs;
    work->stride = 1u;
    work->most = run_segs != 0u ? run_segs : segs;
    if (csize > 1u) {
        work->next_tile = block / csize;
        work->next_seg = crank * segs / csize;
        work->left = (crank + 1u) * segs / csize - work->next_seg;
        return;
    }
    if (turns != 0u) {
        // neighbouring blocks take neighbouring tiles, and where the last turn is not full its
        // blocks have memory to themselves
        work->next_tile = block;
        work->next_seg = 0u;
        work->stride = grid;
        work->left = block < tiles ? (tiles - block + grid - 1u) / grid * segs : 0u;
        return;
    }
    const uint32_t units = tiles * segs;
    const uint32_t blocks = units < grid ? units : grid;
    uint32_t begin = 0u, end = 0u;
    if (block < blocks) {
        decode_range(block, blocks, units, &begin, &end);
    }
    work->next_tile = begin / segs;
    work->next_seg = begin - work->next_tile * segs;
    work->left = end - begin;
}

// A pair's work: whole tiles `stride` apart, then a run of units of the tiles that are cut.
struct PairWork {
    uint32_t tile, s0, s1;                  // the piece
    uint32_t next_whole, whole_left, stride, segs;
    uint32_t next_tile, next_seg, left;
    uint32_t first_cut, units, sharers;     // the cut tiles: the first, their units, the pairs that share them
    uint32_t pieces;                        // per cut tile; 0: the units are dealt evenly, whatever the tile
    uint32_t each, more;                    // ... `each` units to every sharer and one more to the first `more`

    __host__ __device__ __forceinline__ bool next()
    {
        if (whole_left != 0u) {
            tile = next_whole;
            s0 = 0u;
            s1 = segs;
            next_whole += stride;
            whole_left -= 1u;
            return true;
        }
        if (left == 0u) {
            return false;
        }
        tile = next_tile;
        s0 = next_seg;
        s1 = segs - s0 < left ? segs : s0 + left;
        left -= s1 - s0;
        next_tile += 1u;
        next_seg = 0u;
        return true;
    }
    __host__ __device__ __forceinline__ bool last() const
    {
        return whole_left == 0u && left == 0u;
    }
};

// What cutting a tile costs, in units (256 weights deep): the hand-over of the partial sums and the stores at the
// end.  (21248 x 1024, 300 rows, tiles of 4 units: whole behind two turns 23.5 us, cut 28.5.  A line at 8 units is no
// different at the sizes of pair_split's last point.)
constexpr uint32_t kPairCutUnits = 5;
// A piece of a cut tile is worth this many units at least: every holder is a tile of sums more that is written and read
// back.  (20480 x 4096, 300 rows: 6 units 56.6 us, 4 units 54.4, 2 the same.)
constexpr uint32_t kPairMinPiece = 4;
// What pieces may be longer than evenly dealt units.  (21504 x 8192, 300 rows, 20 tiles of 32 units, three pieces of 11 or
// dealt in runs of 8 or 9: 106 us both.)
constexpr uint32_t kPairEvenUnits = 2;

// How the tiles are divided between all pairs; the divisions that need no pair's number, so that the host can do them.
struct PairSplit {
    uint32_t turns, first_cut, cut, units, sharers, pieces, each, more;
};

// As many turns of whole tiles as all pairs have; the tiles that are left:
//   * Fewer than two turns: their units are dealt evenly, because the error of a sum grows with the depth that goes into
//     one accumulator, and evenly dealt it is the smallest.  Pieces of at least four units are faster where the evenly
//     dealt ones are short and have many holders (256 x 16384, 150 rows, 13.5 us against 19.0; 5000 x 1024, 160 rows, 8.1
//     against 12.6; 300 x 16384, 700 rows, 19.6 against 27.4; 2560 x 2560, 300 rows, 14.1 against 14.6), not always (1000 x
//     2048, 200 rows, 14.8 against 11.6; 1024 x 4096, 300 rows, 14.4 against 13.8).
//   * Behind more whole tiles, whose depth gives the error, what is faster: whole as well where cutting costs more
//     than it evens out; else pieces of one size inside each tile, of kPairMinPiece units at least, as many as there
//     are pairs for; else evenly dealt units, where that makes the longest piece more than kPairEvenUnits
//     shorter (20480 x 4096, 300 rows, twelve tiles of 16 units behind two turns: four pieces each 55.4 us, dealt evenly
//     59.2; 19456 x 2560, four of 10: two pieces each 37.3, dealt evenly 36.2).
__host__ __device__ __forceinline__ PairSplit pair_split(uint32_t pairs, uint32_t tiles, uint32_t segs)
{
    PairSplit split;
    split.turns = tiles / pairs;
    split.first_cut = split.turns * pairs;
    split.cut = tiles - split.first_cut;
    split.units = split.cut * segs;
    split.sharers = split.units < pairs ? split.units : pairs;
    split.pieces = split.each = split.more = 0u;
    if (split.cut == 0u) {
        return split;
    }
    if (split.turns > 1u) {
        const uint32_t even = split.units / pairs;
        if (segs <= even + kPairCutUnits) {
            split.sharers = 0u;      // whole tiles as well
            return split;
        }
        const uint32_t places = pairs / split.cut;
        const uint32_t most = segs / kPairMinPiece > 1u ? segs / kPairMinPiece : 1u;
        const uint32_t pieces = most < places ? most : places;
        if (pieces > 1u && (most <= places || (segs + pieces - 1u) / pieces <= even + kPairEvenUnits)) {
            split.pieces = pieces;
            split.sharers = split.cut * pieces;
            return split;
        }
    }
    split.each = split.units / split.sharers;
    split.more = split.units - split.each * split.sharers;
    return split;
}

// The work of pair `id`.
__host__ __device__ __forceinline__ void pair_work(PairWork *work, const PairSplit &split, uint32_t id, uint32_t pairs, uint32_t segs)
{
    work->segs = segs;
    work->stride = pairs;
    work->next_whole = id;
    work->whole_left = split.turns + (split.sharers == 0u && id < split.cut ? 1u : 0u);
    work->next_tile = work->next_seg = work->left = 0u;
    work->first_cut = split.first_cut;
    work->units = split.units;
    work->sharers = split.sharers;
    work->pieces = split.pieces;
    work->each = split.each;
    work->more = split.more;
    if (id >= split.sharers) {
        return;
    }
    if (split.pieces != 0u) {
        const uint32_t tile = id / split.pieces;
        const uint32_t i = id - tile * split.pieces;
        work->next_tile = split.first_cut + tile;
        work->next_seg = i * segs / split.pieces;
        work->left = (i + 1u) * segs / split.pieces - work->next_seg;
        return;
    }
    const uint32_t begin = id * split.each + (id < split.more ? id : split.more);
    const uint32_t tile = begin / segs;
    work->next_tile = split.first_cut + tile;
    work->next_seg = begin - tile * segs;
    work->left = split.each + (id < split.more ? 1u : 0u);
}

__host__ __device__ __forceinline__ void pair_deal(PairWork *work, uint32_t id, uint32_t pairs, uint32_t tiles, uint32_t segs)
{
    pair_work(work, pair_split(pairs, tiles, segs), id, pairs, segs);
}

// The pair that holds a unit of the evenly dealt ones.
__host__ __device__ __forceinline__ uint32_t pair_holder(const PairWork &work, uint32_t unit)
{
    const uint32_t cut = work.more * (work.each + 1u);
    return unit < cut ? unit / (work.each + 1u) : work.more + (unit - cut) / work.each;
}

// The first of the pairs that hold pieces of the cut tile that `id` holds a piece of.
__host__ __device__ __forceinline__ uint32_t pair_first_holder(const PairWork &work, uint32_t id, uint32_t tile)
{
    if (work.pieces != 0u) {
        return id - id % work.pieces;
    }
    return pair_holder(work, (tile - work.first_cut) * work.segs);
}

// The last of the pairs right after `id` that hold later pieces of the cut tile whose first segment `id` holds.
__host__ __device__ __forceinline__ uint32_t pair_last_holder(const PairWork &work, uint32_t id, uint32_t tile)
{
    if (work.pieces != 0u) {
        return id + work.pieces - 1u;
    }
    return pair_holder(work, (tile - work.first_cut + 1u) * work.segs - 1u);
}

// A cut tile is finished by the pair that began it, or, where it has more holders than a pair has units by so many and
// all of them run (pair_undecided), by all its holders.  The one that began it reads as many tiles of sums as there are
// others, 0.8 us a round trip, but most of it before its own sums are there: the longer the runs, the more.  All together
// read one tile's worth each, and everybody waits for the last to publish.  (Units per pair, holders: beginner and all, us.  1, 8, 1000 x 2048, 200 rows:
// 19.1 and 11.7; 1, 64, 256 x 16384, 150 rows: 54.0 and 19.0; 1.7, 10, 1024 x 4096, 300 rows: 21.2 and 13.8; 2.7, 4 or 5,
// 2560 x 2560, 300 rows: 15.4 and 18.1, with the line between 4 and 5 14.6; 3.5, 10, 1024 x 8192, 300 rows: 20.8 and 18.7;
// 4.3, 15, 1280 x 16384, 150 rows: 26.1 and 22.2; 5.2, 13, 300 x 16384, 700 rows: 34.4 and 27.4; 6.9, 10, 2048 x 16384, 150
// rows: 25.5 and 25.1; 8.6, 8, 2560 x 16384, 150 rows: 27.1 and 27.7; 10.3, 4 or 5, 2560 x 9728, 300 rows: 23.4 and 27.1.)
constexpr uint32_t kPairShareMore = 3;

__host__ __device__ __forceinline__ uint32_t pair_share_from(const PairWork &work)
{
    return (work.pieces != 0u ? work.segs / work.pieces : work.each) + kPairShareMore;
}

// What such a tile's holders go by: a word that counts those that have begun, with kPairAlone set by the first that came
// to wait before all had.  Once all have begun, or the bit is set, it says the same for good.
constexpr uint32_t kPairAlone = 1u << 31;

__host__ __device__ __forceinline__ bool pair_undecided(uint32_t word, uint32_t holders)
{
    return word != holders && (word & kPairAlone) == 0u;
}

// The runs of rows [run, end) that holder `index` finishes.
__host__ __device__ __forceinline__ void pair_share(bool together, uint32_t index, uint32_t holders, uint32_t runs, uint32_t *run,
                                                    uint32_t *end)
{
    *run = together ? index * runs / holders : 0u;
    *end = together ? (index + 1u) * runs / holders : index == 0u ? runs : 0u;
}

} // namespace q8
