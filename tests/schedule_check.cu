// Host model of the streaming kernel's division of work, built on the kernel's own helpers
// (unit_range, WorkIter, last_holder from q8_tile.cuh).  For a sweep of shapes and grid sizes
// it checks the properties the device protocol rests on:
//
//   1. every (tile, segment) unit is computed exactly once;
//   2. a block holds at most one piece of a tile whose first segment it does not hold (it has
//      one slot for partial sums and one set of flags), and that piece is its first;
//   3. a piece that starts a tile without finishing it is its block's last piece, so a block
//      only ever waits after it has published its own partial sums: no cycle of waits;
//   4. last_holder() names exactly the blocks that hold the remaining segments of that tile,
//      and they are the blocks directly after the owner;
//   5. no block that takes part is without work;
//   6. the decode kernel's own 32-bit range arithmetic (decode_range, decode_holder in
//      q8_decode.cu) deals every unit once and names the block that holds a unit;
//   7. the division between pairs of SMs (PairWork, pair_deal, pair_last_holder in q8_schedule.cuh) has the properties
//      1 to 4, and where it cuts tiles into pieces of one size, each has kPairMinPiece segments at least;
//   8. the division between blocks and clusters (MidWork, mid_deal): every unit once, by the block that decode_holder
//      names where units are dealt, the pieces of a cluster's block within run_segs and in one tile;
//   9. launches of pairs that share the SMs (streams of one's own, in any order of steps) come to their end with as few
//      as one place more than there are launches, and every run of rows of a cut tile is finished once: pair_undecided,
//      pair_share.  With holders that wait whether or not all others run, some of the same orders have no end;
//  10. the router's tiles (route_plan in q8_route.cuh) take a ring as deep as one block of an SM has room for only where all
//      clusters run at the same time that way, with the fewest tokens to a group, and else groups of 8 where those run at the
//      same time in pairs.
//
// Prints "ok <cases>" and exits 0, or the first violated property and exits 1.
#include <cstdio>
#include <cstdlib>
#include <utility>
#include <vector>

#include "q8_route.cuh"
#include "q8_schedule.cuh"
#include "q8_tile.cuh"

using namespace q8;

struct Piece {
    uint32_t tile, s0, s1;
};

static int fail(const char *what, unsigned long long tiles, uint32_t segs, unsigned int grid, unsigned int b)
{
    std::printf("violated: %s (tiles %llu, segments %u, grid %u, block %u)\n", what, tiles, segs, grid, b);
    return 1;
}

// `dp_waves` whole waves of tiles dealt round-robin ahead of the cut tiles: 0 for the
// decode-regime kernel (everything is cut into units).
static int check(unsigned long long tiles, uint32_t segs, unsigned int grid, bool hybrid)
{
    const uint32_t waves = hybrid ? (uint32_t)(tiles / grid) : 0u;
    const uint32_t dp_tiles = waves * grid;
    const unsigned long long units = (tiles - dp_tiles) * segs;
    const unsigned int blocks = units < grid ? (unsigned int)units : grid;
    std::vector<unsigned int> seen((size_t)(tiles * segs), 0u);
    std::vector<std::vector<Piece>> work(grid);
    for (unsigned int b = 0; b < grid; ++b) {
        WorkIter it;
        it.segs = segs;
        it.u = 0;
        it.u_end = 0;
        if (b < blocks) {
            unit_range(b, blocks, units, &it.u, &it.u_end);
            if (it.u >= it.u_end) {
                return fail("a block in the schedule has no units", tiles, segs, grid, b);
            }
        }
        it.sk_tile0 = dp_tiles;
        it.dp_next = 0;
        it.dp_count = waves;
        it.dp_first = b;
        it.dp_stride = grid;
        Piece p;
        while (it.next(p.tile, p.s0, p.s1)) {
            if (p.tile >= tiles || p.s1 > segs || p.s0 >= p.s1) {
                return fail("piece out of range", tiles, segs, grid, b);
            }
            for (uint32_t s = p.s0; s < p.s1; ++s) {
                seen[(size_t)p.tile * segs + s] += 1u;
            }
            work[b].push_back(p);
        }
    }
    for (size_t i = 0; i < seen.size(); ++i) {
        if (seen[i] != 1u) {
            return fail("a unit is computed zero or several times", tiles, segs, grid, (unsigned int)(i / segs));
        }
    }
    for (unsigned int b = 0; b < grid; ++b) {
        const std::vector<Piece> &pieces = work[b];
        for (size_t i = 0; i < pieces.size(); ++i) {
            const Piece &p = pieces[i];
            const bool whole = p.s0 == 0u && p.s1 == segs;
            const bool owner = p.s0 == 0u;
            if (!owner && i != 0u) {
                return fail("a partial piece is not the block's first piece", tiles, segs, grid, b);
            }
            if (owner && !whole) {
                // In the hybrid order the cut tiles come first and whole tiles follow them, so
                // the waiting piece is the last of the cut pieces; every whole tile after it
                // needs nobody.  Nothing that is published may come after the wait.
                for (size_t later = i + 1; later < pieces.size(); ++later) {
                    if (pieces[later].s0 != 0u || pieces[later].s1 != segs) {
                        return fail("a block waits before it has published", tiles, segs, grid, b);
                    }
                }
                const unsigned long long cut_tile = p.tile - dp_tiles;
                const unsigned long long tile_end = (cut_tile + 1ull) * segs;
                const unsigned int last = last_holder(b, blocks, units, tile_end);
                uint32_t expect = p.s1;
                for (unsigned int cc = b + 1u; cc <= last; ++cc) {
                    if (cc >= blocks || work[cc].empty()) {
                        return fail("last_holder names a block without work", tiles, segs, grid, b);
                    }
                    const Piece &q = work[cc][0];
                    if (q.tile != p.tile || q.s0 != expect) {
                        return fail("a named holder does not continue the tile", tiles, segs, grid, b);
                    }
                    expect = q.s1;
                }
                if (expect != segs) {
                    return fail("the named holders do not finish the tile", tiles, segs, grid, b);
                }
            }
        }
    }
    return 0;
}

// The decode kernel's range arithmetic: the ranges of the blocks tile [0, units) in order, none
// is empty, and decode_holder names the block whose range holds a unit.
static int check_decode(uint32_t units, uint32_t blocks)
{
    uint32_t at = 0;
    for (uint32_t b = 0; b < blocks; ++b) {
        uint32_t begin, end;
        decode_range(b, blocks, units, &begin, &end);
        if (begin != at || end <= begin) {
            return fail("decode ranges do not tile the units", units, 0u, blocks, b);
        }
        for (uint32_t u = begin; u < end; ++u) {
            if (decode_holder(u, blocks, units) != b) {
                return fail("decode_holder names another block", units, u, blocks, b);
            }
        }
        at = end;
    }
    return at == units ? 0 : fail("decode ranges stop short", units, 0u, blocks, 0u);
}

static int check_pairs(uint32_t tiles, uint32_t segs, uint32_t pairs)
{
    std::vector<unsigned int> seen((size_t)tiles * segs, 0u);
    std::vector<std::vector<Piece>> pieces(pairs);
    std::vector<PairWork> work(pairs);
    for (uint32_t id = 0; id < pairs; ++id) {
        pair_deal(&work[id], id, pairs, tiles, segs);
        PairWork w = work[id];
        while (w.next()) {
            if (w.tile >= tiles || w.s0 >= w.s1 || w.s1 > segs) {
                return fail("a pair's piece out of range", tiles, segs, pairs, id);
            }
            if (w.pieces != 0u && w.tile >= w.first_cut && w.s1 - w.s0 < kPairMinPiece) {
                return fail("a piece shorter than the rule says", tiles, segs, pairs, id);
            }
            for (uint32_t s = w.s0; s < w.s1; ++s) {
                seen[(size_t)w.tile * segs + s] += 1u;
            }
            pieces[id].push_back({w.tile, w.s0, w.s1});
        }
        if (!w.last()) {
            return fail("a pair without pieces is not at its end", tiles, segs, pairs, id);
        }
    }
    for (unsigned int count : seen) {
        if (count != 1u) {
            return fail("pairs: a unit is computed zero or several times", tiles, segs, pairs, 0u);
        }
    }
    for (uint32_t id = 0; id < pairs; ++id) {
        uint32_t published = 0u;
        for (size_t i = 0; i < pieces[id].size(); ++i) {
            const Piece &p = pieces[id][i];
            if (p.s0 != 0u && ++published > 1u) {
                return fail("a pair publishes twice", tiles, segs, pairs, id);
            }
            if (p.s0 == 0u && p.s1 != segs) {
                if (i + 1u != pieces[id].size()) {
                    return fail("a pair waits before its last piece", tiles, segs, pairs, id);
                }
                uint32_t at = p.s1;
                for (uint32_t cc = id + 1u; cc <= pair_last_holder(work[id], id, p.tile); ++cc) {
                    bool holds = false;
                    for (const Piece &q : pieces[cc < pairs ? cc : id]) {
                        holds = holds || (q.tile == p.tile && q.s0 == at);
                        at = q.tile == p.tile && q.s0 == at ? q.s1 : at;
                    }
                    if (cc >= pairs || !holds) {
                        return fail("a named pair does not continue the tile", tiles, segs, pairs, id);
                    }
                }
                if (at != segs) {
                    return fail("the named pairs do not finish the tile", tiles, segs, pairs, id);
                }
            }
        }
    }
    return 0;
}

// Every holder of a cut tile names the same first pair, the one that has the tile's first segment.
static int check_first_holder(uint32_t tiles, uint32_t segs, uint32_t pairs)
{
    std::vector<uint32_t> first(tiles, pairs);
    for (uint32_t id = 0; id < pairs; ++id) {
        PairWork w;
        pair_deal(&w, id, pairs, tiles, segs);
        while (w.next()) {
            if (w.s0 == 0u) {
                first[w.tile] = id;
            }
            if ((w.s0 != 0u || w.s1 != segs) && pair_first_holder(w, id, w.tile) != first[w.tile]) {
                return fail("a holder names another pair as the tile's first", tiles, segs, pairs, id);
            }
        }
    }
    return 0;
}

// `way`: 0 units, 1 whole tiles in turns, 2 and 4 clusters of that size.
static int check_mid(uint32_t tiles, uint32_t segs, uint32_t grid, uint32_t way, uint32_t run_segs)
{
    const uint32_t csize = way >= 2u ? way : 1u;
    if (csize > 1u) {
        if (segs < csize) {
            return 0;
        }
        grid = tiles * csize;
    }
    const uint32_t units = tiles * segs;
    const uint32_t blocks = units < grid ? units : grid;
    std::vector<unsigned int> seen((size_t)units, 0u);
    for (uint32_t b = 0; b < grid; ++b) {
        MidWork w;
        mid_deal(&w, b, grid, csize, b % csize, tiles, segs, way == 1u ? (tiles + grid - 1u) / grid : 0u, csize > 1u ? run_segs : 0u);
        while (w.next()) {
            if (w.tile >= tiles || w.s0 >= w.s1 || w.s1 > segs) {
                return fail("a block's piece out of range", tiles, segs, grid, b);
            }
            if (csize > 1u && (w.tile != b / csize || (run_segs != 0u && w.s1 - w.s0 > run_segs))) {
                return fail("a cluster's piece in another tile or too long", tiles, segs, grid, b);
            }
            if (way == 1u && (w.s0 != 0u || w.s1 != segs)) {
                return fail("a cut tile in turns", tiles, segs, grid, b);
            }
            for (uint32_t s = w.s0; s < w.s1; ++s) {
                seen[(size_t)w.tile * segs + s] += 1u;
                if (way == 0u && decode_holder(w.tile * segs + s, blocks, units) != b) {
                    return fail("decode_holder names another block of the units", tiles, segs, grid, b);
                }
            }
        }
        if (w.left != 0u) {
            return fail("a block's work has no end", tiles, segs, grid, b);
        }
    }
    for (unsigned int count : seen) {
        if (count != 1u) {
            return fail("blocks: a unit is computed zero or several times", tiles, segs, grid, way);
        }
    }
    return 0;
}

// A launch of pairs, step by step as a pair goes through q8_pair.cu; a quarter of its blocks stands for all.
struct Launch {
    struct Cut {
        uint32_t first = 0, holders = 0, word = 0, published = 0;
        std::vector<unsigned int> finished;      // per run of rows
    };
    struct Pair {
        int at = -1;                             // -1: has no place yet
        std::vector<Piece> pieces;               // the cut ones, in order
        std::vector<int> together;               // per piece; -1: not decided
    };
    uint32_t runs, share_from, placed = 0, left = 0;
    std::vector<Cut> cuts;
    std::vector<Pair> pairs;
    bool always;

    Launch(uint32_t tiles, uint32_t segs, uint32_t count, uint32_t runs_, bool always_)
        : runs(runs_), cuts(tiles), pairs(tiles * segs < count ? tiles * segs : count), always(always_)
    {
        count = (uint32_t)pairs.size();
        for (uint32_t id = 0; id < count; ++id) {
            PairWork w;
            pair_deal(&w, id, count, tiles, segs);
            share_from = pair_share_from(w);
            while (w.next()) {
                if (w.s0 == 0u && w.s1 == w.segs) {
                    continue;
                }
                pairs[id].pieces.push_back({w.tile, w.s0, w.s1});
                pairs[id].together.push_back(-1);
                Cut &cut = cuts[w.tile];
                cut.first = cut.holders == 0u ? id : cut.first;
                cut.holders += 1u;
                cut.finished.assign(runs, 0u);
            }
        }
    }
    bool shared(const Cut &cut) const { return cut.holders >= share_from; }
    bool done() const { return left == pairs.size(); }
    bool place()
    {
        if (placed == pairs.size()) {
            return false;
        }
        pairs[placed++].at = 0;
        return true;
    }
    void finish(Cut &cut, uint32_t begin, uint32_t end)
    {
        for (uint32_t r = begin; r < end; ++r) {
            cut.finished[r] += 1u;
        }
    }
    // One step of a pair: false if it has to wait.  `gone` is set when it gives its place back.
    bool step(uint32_t id, bool *gone)
    {
        Pair &pair = pairs[id];
        const int pieces = (int)pair.pieces.size();
        if (pair.at == 0) {
            for (const Piece &p : pair.pieces) {
                cuts[p.tile].word += shared(cuts[p.tile]) ? 1u : 0u;
            }
        } else if (pair.at <= pieces) {
            const Piece &p = pair.pieces[pair.at - 1];
            Cut &cut = cuts[p.tile];
            if (p.s0 == 0u && !shared(cut)) {
                if (cut.published + 1u != cut.holders) {
                    return false;
                }
                finish(cut, 0u, runs);
            } else {
                cut.published += 1u;
            }
        } else if (pair.at <= 2 * pieces) {
            const int i = pair.at - 1 - pieces;
            Cut &cut = cuts[pair.pieces[i].tile];
            if (shared(cut)) {
                if (pair.together[i] < 0) {
                    if (!always && pair_undecided(cut.word, cut.holders)) {
                        cut.word |= kPairAlone;
                    }
                    pair.together[i] = always || cut.word == cut.holders ? 1 : 0;
                }
                uint32_t run, end;
                pair_share(pair.together[i] == 1, id - cut.first, cut.holders, runs, &run, &end);
                if (run < end && cut.published != cut.holders) {
                    return false;
                }
                finish(cut, run, end);
            }
        } else {
            left += 1u;
            *gone = true;
            pair.at = -2;
            return true;
        }
        pair.at += 1;
        return true;
    }
};

// 0: both launches ended and were right; 1: no step is left that anybody could take; 2: wrong
static int run_together(Launch &a, Launch &b, uint32_t places, uint32_t &state)
{
    Launch *launches[2] = {&a, &b};
    uint32_t taken = 0u;
    while (!a.done() || !b.done()) {
        bool moved = false;
        for (uint32_t tries = 0; tries < 400u && !moved; ++tries) {
            state = state * 1664525u + 1013904223u;
            Launch &l = *launches[(state >> 9) & 1u];
            if ((state >> 12) % 3u == 0u) {
                moved = taken < places && l.place();
                taken += moved ? 1u : 0u;
            } else if (l.placed != 0u) {
                const uint32_t id = (state >> 14) % l.placed;
                bool gone = false;
                moved = l.pairs[id].at >= 0 && l.step(id, &gone);
                taken -= gone ? 1u : 0u;
            }
        }
        for (int i = 0; i < 2 && !moved; ++i) {       // nothing by chance: anything at all?
            moved = taken < places && launches[i]->place();
            taken += moved ? 1u : 0u;
            for (uint32_t id = 0; id < launches[i]->placed && !moved; ++id) {
                bool gone = false;
                moved = launches[i]->pairs[id].at >= 0 && launches[i]->step(id, &gone);
                taken -= gone ? 1u : 0u;
            }
        }
        if (!moved) {
            return 1;
        }
    }
    for (Launch *l : launches) {
        for (const Launch::Cut &cut : l->cuts) {
            for (unsigned int times : cut.finished) {
                if (times != 1u) {
                    return 2;
                }
            }
        }
    }
    return 0;
}

// *stuck: how many orders had no end with holders that always wait for all
static int check_shared_places(uint32_t *stuck, unsigned long long *cases)
{
    // one tile of many segments, a few of few, units dealt evenly with one or two tiles to a pair, equal pieces
    const uint32_t shapes[][2] = {{1u, 64u}, {8u, 8u}, {20u, 4u}, {20u, 10u}, {4u, 64u}, {158u, 10u}, {39u, 16u}};
    uint32_t state = 1u;
    for (const auto &one : shapes) {
        for (const auto &other : shapes) {
            for (uint32_t places : {3u, 9u, 74u}) {
                for (uint32_t runs : {1u, 7u, 32u}) {
                    Launch a(one[0], one[1], 74u, runs, false), b(other[0], other[1], 74u, runs, false);
                    const int ended = run_together(a, b, places, state);
                    if (ended != 0) {
                        return fail(ended == 1 ? "launches of pairs that wait for each other" : "a run of rows not finished once",
                                    one[0], one[1], other[0], places);
                    }
                    *cases += 1u;
                    Launch c(one[0], one[1], 74u, runs, true), d(other[0], other[1], 74u, runs, true);
                    *stuck += run_together(c, d, places, state) == 1 ? 1u : 0u;
                }
            }
        }
    }
    return 0;
}

// `alone`, `paired`: clusters that run at the same time with one block, with two, to an SM.
static int check_route(uint32_t tokens, uint32_t smallest, uint32_t alone, uint32_t paired)
{
    const RoutePlan plan = route_plan(tokens, smallest, alone, paired);
    auto groups = [&](uint32_t group) { return (tokens + group - 1u) / group; };
    bool right = plan.group >= smallest && plan.group <= 16u && (plan.group & (plan.group - 1u)) == 0u;
    if (plan.deep) {
        right = right && groups(plan.group) <= alone && (plan.group == smallest || groups(plan.group / 2u) > alone);
    } else {
        right = right && groups(16u) > alone && plan.group == (groups(8u) <= paired ? 8u : 16u);
    }
    return right ? 0 : fail("the router's groups", tokens, alone, paired, plan.group);
}

int main()
{
    unsigned long long cases = 0;
    uint32_t stuck = 0;
    if (check_shared_places(&stuck, &cases) != 0) {
        return 1;
    }
    if (stuck == 0u) {
        std::printf("violated: holders that always wait came to an end in every order\n");
        return 1;
    }
    const unsigned int grids[] = {1u, 2u, 3u, 7u, 16u, 37u, 64u, 132u, 147u, 148u, 160u};
    const uint32_t seg_counts[] = {1u, 2u, 3u, 4u, 8u, 16u, 32u, 56u};
    for (unsigned int grid : grids) {
        for (uint32_t segs : seg_counts) {
            for (unsigned long long tiles = 1; tiles <= 700; tiles += (tiles < 40 ? 1 : 13)) {
                for (int hybrid = 0; hybrid < 2; ++hybrid) {
                    if (check(tiles, segs, grid, hybrid != 0) != 0) {
                        return 1;
                    }
                    cases += 1;
                }
            }
        }
    }
    // shapes of the benchmark and the tests: (rows of w, depth, rows of x, token tile)
    const unsigned int shapes[][4] = {{6144, 4096, 32, 32},   {4096, 4096, 32, 32},  {28672, 4096, 32, 32},
                                      {4096, 14336, 32, 32},  {151936, 8192, 8, 16}, {18992, 8192, 8, 16},
                                      {4736, 4096, 300, 128}, {4096, 4096, 2048, 128}, {28672, 4096, 2048, 128},
                                      {130, 256, 1, 16},      {128, 256, 129, 128}};
    for (const auto &shape : shapes) {
        const unsigned long long row_tiles = (shape[0] + kRows - 1u) / kRows;
        const unsigned long long tok_tiles = (shape[2] + shape[3] - 1u) / shape[3];
        for (unsigned int grid : {148u, 132u}) {
            for (int hybrid = 0; hybrid < 2; ++hybrid) {
                if (check(row_tiles * tok_tiles, shape[1] / kSegK, grid, hybrid != 0) != 0) {
                    return 1;
                }
                cases += 1;
            }
        }
    }
    // the decode kernel's ranges: two blocks per SM and odd grids
    for (uint32_t blocks : {1u, 2u, 7u, 148u, 160u, 264u, 296u}) {
        for (uint32_t units : {1u, 2u, 5u, 147u, 296u, 297u, 512u, 768u, 1792u, 3584u, 37984u}) {
            if (units < blocks) {
                continue;
            }
            if (check_decode(units, blocks) != 0) {
                return 1;
            }
            cases += 1;
        }
    }
    for (uint32_t way : {0u, 1u, 2u, 4u}) {
        for (uint32_t run_segs : {0u, 1u, 3u}) {
            for (uint32_t segs : {1u, 2u, 3u, 5u, 8u, 11u, 16u, 56u, 64u}) {
                for (uint32_t tiles = 1; tiles <= 600; tiles += (tiles < 40 ? 1 : 17)) {
                    if (check_mid(tiles, segs, 148u, way, run_segs) != 0 || check_mid(tiles, segs, 7u, way, run_segs) != 0) {
                        return 1;
                    }
                    cases += 2;
                }
            }
        }
    }
    for (uint32_t pairs : {1u, 2u, 9u, 66u, 74u}) {
        for (uint32_t segs : {1u, 2u, 3u, 4u, 5u, 7u, 8u, 9u, 10u, 11u, 13u, 16u, 18u, 31u, 36u, 38u, 56u, 64u}) {
            for (uint32_t tiles = 1; tiles <= 700; tiles += (tiles < 300 ? 1 : 7)) {
                // (the launch has as many pairs as units, at most)
                if (check_pairs(tiles, segs, tiles * segs < pairs ? tiles * segs : pairs) != 0
                    || check_first_holder(tiles, segs, tiles * segs < pairs ? tiles * segs : pairs) != 0) {
                    return 1;
                }
                cases += 1;
            }
        }
    }
    // a B200's clusters of one to eight blocks, and none known
    const uint32_t at_once[][2] = {{148u, 296u}, {74u, 148u}, {45u, 93u}, {33u, 71u}, {26u, 56u}, {22u, 45u}, {15u, 37u},
                                   {15u, 33u},   {0u, 0u}};
    for (const auto &clusters : at_once) {
        for (uint32_t smallest : {4u, 8u}) {
            for (uint32_t tokens = 1; tokens <= 5000u; ++tokens) {
                if (check_route(tokens, smallest, clusters[0], clusters[1]) != 0) {
                    return 1;
                }
                cases += 1;
            }
        }
    }
    std::printf("ok %llu\n", cases);
    return 0;
}
