// How a product of staged rows (fk_qgemm.cuh) is dealt to blocks.  Plain C++, so that the host plans with it and tests run it without a GPU.
#pragma once
#include <stddef.h>

#if defined(__CUDACC__)
#define FKQ_HD __host__ __device__
#else
#define FKQ_HD
#endif
#define FKQ_EPI 8                       // storing warps of a block
#define FKQ_ROWS 256                    // weight rows of a block
#define FKQ_MOST_ROWS 128               // rows of X of the widest tile
#define FKQ_SPLIT_ROWS 32               // .. whose parts meet in memory (two parts of a block take no more scratch than a widest tile)
#define FKQ_SUM_STEPS 10                // super-blocks (of 512 columns) summed in one go in tensor memory
#define FKQ_COUNTERS 65536              // ticket words: 8 per tile that is split
FKQ_HD inline size_t fkq_part_floats(int bn) { return (size_t)bn * FKQ_ROWS; }

// The v-th piece of work of block `b` of `G`: super-blocks [k0, k1) of a tile.
struct QWork { int tile, k0, k1; };
FKQ_HD inline bool fkq_work(int whole, int tiles, int nsb, int b, int G, int v, QWork &w) {
    if (whole) { w.tile = b + v * G; w.k0 = 0; w.k1 = nsb; return w.tile < tiles; }
    const long long T = (long long)tiles * nsb;
    const int s0 = (int)(b * T / G), s1 = (int)((b + 1) * T / G);
    w.tile = s0 / nsb + v;
    const int t0 = w.tile * nsb, a = s0 > t0 ? s0 : t0, e = s1 < t0 + nsb ? s1 : t0 + nsb;
    if (w.tile >= tiles || a >= e) return false;
    w.k0 = a - t0; w.k1 = e - t0;
    return true;
}
// the block whose run holds step s, and the scratch slot of block b's part of `tile` (two slots a block: the tile its run begins in, the one it ends in)
FKQ_HD inline int fkq_owner(int tiles, int nsb, int G, int s) { return (int)((((long long)s + 1) * G - 1) / ((long long)tiles * nsb)); }
FKQ_HD inline int fkq_slot(int tiles, int nsb, int G, int b, int tile) { return 2 * b + ((int)((long long)b * tiles * nsb / G) / nsb == tile ? 0 : 1); }

// A piece that covers part of a tile: its sums go to the scratch area and a ticket of the tile is counted; of the warps that store the same
// rows the one that counts the last of the tile's parts adds them up and sets the ticket word to zero.
FKQ_HD inline bool fkq_part(const QWork &w, int nsb) { return w.k0 != 0 || w.k1 != nsb; }
FKQ_HD inline int fkq_parts(int tiles, int nsb, int G, int tile) { return fkq_owner(tiles, nsb, G, (tile + 1) * nsb - 1) - fkq_owner(tiles, nsb, G, tile * nsb) + 1; }
// Where the sums of a piece that begin at super-block `at` end: stretches of at most FKQ_SUM_STEPS, about equally long.  The MMAs cut what an
// accumulator cannot hold (towards zero) where an addition rounds, so a sum drifts by about 6e-10 of itself per column.  Results on the
// wrong side of their rounding, gated activations, 3584 rows: over 18944 columns in one go 0.67 % (k_qmm4 0.34 %), in stretches 0.29 %; over
// 5120 columns 0.22 % (0.32 %).  The storing warps add stretches in fp32, rounded, while the MMAs wait: 1000 rows, 18944 -> 3584, 152 -> 157 us.
FKQ_HD inline int fkq_stretch(const QWork &w, int at) {
    const int n = w.k1 - w.k0, parts = (n + FKQ_SUM_STEPS - 1) / FKQ_SUM_STEPS, each = (n + parts - 1) / parts;
    return at + each < w.k1 ? at + each : w.k1;
}
// The pieces of block b in the hands of one storing warp.  take(v, w) waits for the piece and stores it (counting its ticket if it is a part); it
// returns false, with nothing counted, when the wait runs out.  From then on nothing is taken, but skip(w) still counts the
// ticket of every part: the ticket words are zero again after every launch, also after one that gave up.
#if defined(__CUDACC__)
#pragma nv_exec_check_disable
#endif
template <typename Take, typename Skip> FKQ_HD inline bool fkq_pieces(int whole, int tiles, int nsb, int b, int G, Take take, Skip skip) {
    bool ok = true;
    QWork w;
    for (int v = 0; fkq_work(whole, tiles, nsb, b, G, v, w); ++v) {
        ok = ok && take(v, w);
        if (!ok && fkq_part(w, nsb)) skip(w);
    }
    return ok;
}

// Rows of X per tile, blocks and split of a product of m rows that no cluster takes (fkq_cluster_plan): the widest tile that the rows fill, a narrower one while that gives more
// blocks a tile of their own (a step costs a block the same up to 64 rows).  Tiles of up to 32 rows are dealt in equal runs of steps (a
// part's sums are small, and the product is bound by the weights), wider ones whole.
// Measured: 100 rows, 896 -> 1152: 11 us with tiles of 16 rows, 31 with one tile of 128 split over K (its fold passes 128 rows through memory);
// 4864 -> 896: 19 against 63.
struct QPlan { int bn, mtiles, tiles, grid, whole; };
inline QPlan fkq_plan(int m, int ntiles, int nsb, int sm) {
    QPlan p;
    p.bn = m <= 16 ? 16 : m <= 32 ? 32 : m <= 64 ? 64 : 128;
    while (p.bn > 16 && (ntiles + 15) / 16 * ((m + p.bn / 2 - 1) / (p.bn / 2)) <= sm) p.bn /= 2;
    p.mtiles = (m + p.bn - 1) / p.bn; p.tiles = (ntiles + 15) / 16 * p.mtiles; p.whole = 1; p.grid = p.tiles < sm ? p.tiles : sm;
    if (p.tiles > FKQ_COUNTERS / FKQ_EPI) return p;
    if (p.bn <= FKQ_SPLIT_ROWS && p.tiles % sm) { const long long steps = (long long)p.tiles * nsb; p.whole = 0; p.grid = steps < sm ? (int)steps : sm; }
    return p;
}

// A cluster of S blocks shares a tile and splits its super-blocks (grid = tiles * S, whole = -S in a plan).
FKQ_HD inline bool fkq_cluster_work(int S, int tiles, int nsb, int b, int v, QWork &w) {      // one piece a block
    const int part = b % S;
    w.tile = b / S; w.k0 = part * nsb / S; w.k1 = (part + 1) * nsb / S;
    return v == 0 && w.tile < tiles;
}
// The same with a tile's super-blocks split over the blocks of a cluster (2, 4 or 8 of them, none without a super-block and none with more than
// FKQ_SUM_STEPS): wide tiles, so that weights are expanded once for up to 128 rows, without passing sums through memory.  True where its time by this
// reckoning, in super-blocks of a block, is shorter than the other plan's: sums that meet in memory count one and a half, in a cluster three
// quarters, the store of a tile of 128 rows a fifth, a further wave of clusters half.  most: clusters of 2, 4 and 8 blocks that are resident at once.
// A whole prompt by it and by the other plan alone, us: 0.5B shape, 20 / 100 / 300 positions 1729 / 2079, 2129 / 2283, 2720 / 3376; 7B shape, 30 / 100 positions
// 3779 / 4554, 4418 / 7265 (there 18944 -> 3584 in tiles of 16 rows expanded every weight seven times).
inline bool fkq_cluster_plan(int m, int ntiles, int nsb, int sm, const int (&most)[3], QPlan &p) {
    const QPlan q = fkq_plan(m, ntiles, nsb, sm);
    const int rowtiles = (ntiles + 15) / 16;
    double best = q.whole ? (double)((q.tiles + q.grid - 1) / q.grid) * (nsb + (q.bn == 128 ? 0.2 : 0.0)) : (double)((long long)q.tiles * nsb + q.grid - 1) / q.grid + 1.5;
    bool found = false;
    for (int bn = 128; bn >= 16; bn /= 2) {
        if (bn > 16 && m <= bn / 2) continue;
        const int tiles = rowtiles * ((m + bn - 1) / bn);
        for (int i = 0; i < 3 && (2 << i) <= nsb; ++i) {
            const int S = 2 << i, each = (nsb + S - 1) / S;
            if (each > FKQ_SUM_STEPS || most[i] < 1) continue;
            const int waves = (tiles + most[i] - 1) / most[i];
            const double t = waves * (each + 0.75 + (bn == 128 ? 0.2 : 0.0)) + 0.5 * (waves - 1);
            if (t < best - 1e-9) { best = t; found = true; p.bn = bn; p.mtiles = (m + bn - 1) / bn; p.tiles = tiles; p.grid = tiles * S; p.whole = -S; }
        }
    }
    return found;
}
// What a product runs as.  Only tiles of up to FKQ_SPLIT_ROWS rows have parts that meet in memory: the storing warps of an accumulator give up one by one
// there, and the four of a tile that is stored by whole lines meet at a barrier of the block.
inline QPlan fkq_choose(int m, int ntiles, int nsb, int sm, const int (&most)[3]) {
    QPlan p;
    return fkq_cluster_plan(m, ntiles, nsb, sm, most, p) ? p : fkq_plan(m, ntiles, nsb, sm);
}
