// fp64_cut.h -- how the FP64 kernel cuts a product among its CTAs: the units of work, each CTA's share of
// them, the stream-K pieces of a tile and the warps' parts.  Shared by the kernel, the host code that
// launches it and the CPU tests, which compile this file by itself.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MGX_HD __host__ __device__ __forceinline__
#else
#define MGX_HD inline
#endif

namespace mgx {
namespace fp64 {

constexpr int BK = 32;
constexpr int UNIT = 8;                      // columns of a work unit (one DMMA's N)
constexpr int TILE_UNITS = 16;               // widest tile: 128 columns
constexpr int BM = 64;                       // rows of a band
constexpr int CWARPS = 16;                   // consumer warps
constexpr int GROUP_M = 1024 / BM;           // stream-K raster groups of 1024 rows
// A last band of at most 16 or 32 rows computes one or two 16-row strips, spread over all four
// sub-partitions.  Its units then cost less by this measure, against COST for a whole band's; more than
// a quarter and a half of it, because a warp has fewer units to hide its loads behind.  Sizes measured
// with 2 and 4, 3 and 5, 4 and 6 of 8: 1040 x 4096 x 4096 1459, 991, 1008 us (1043 with whole bands
// only), 1056 x 2048 x 4096 602, 505, 521 (526), 80 x 4096 x 4096 144, 128, 120 (143).  One band alone,
// 8192 x 8192: 16 rows 279 -> 104 us, 32 rows 279 -> 189.
constexpr int COST = 8, COST_1 = 3, COST_2 = 5;

template <typename T>
MGX_HD T least(T a, T b)
{
    return a < b ? a : b;
}

// The cut of one product.
struct Cut {
    int bands, ucols;   // ceil(m / BM), ceil(n / 8)
    int tile_units;     // units of a whole tile (the last tile of a band may have fewer)
    int tiles_n;        // ceil(ucols / tile_units)
    int kblocks;        // K blocks of the whole reduction
    int ksplit;         // K slices (1: whole K); slice s reduces K blocks [s kb_split, (s + 1) kb_split)
    int kb_split;
    int skew;           // units that starting another band costs a CTA (see Walk)
    int strips_last;    // log2 of the 16-row strips of the last band that are computed: 0, 1 or 2
    int w_full, w_last; // what a unit of a band, and of the last band, costs (see Walk)
    int share_rem;      // length - share x grid
    long long length;   // the product's length by that measure, and its part per CTA
    long long share;
    long long sk_full;  // stream-K: K-block units of the tiles that cost w_full
};

// One piece of work: units [u0, u0 + units) of a band over K blocks [kb_begin, kb_end).
struct Item {
    int band, u0, units, kb_begin, kb_end, slice;
    int strips;  // log2 of the 16-row strips that are computed
    int tile;    // stream-K: the tile this is a piece of
};

// Tile coordinates of raster position `tile`: groups of 1024 rows sweep the columns together; the
// tiles of a last band that costs less come after all others.
MGX_HD void tile_coords(const Cut &p, int tile, int &tm, int &tn)
{
    const int bands = p.w_last < p.w_full ? p.bands - 1 : p.bands;
    if (tile >= bands * p.tiles_n) {
        tm = bands;
        tn = tile - bands * p.tiles_n;
        return;
    }
    const int per_group = GROUP_M * p.tiles_n;
    const int group = tile / per_group;
    const int first_m = group * GROUP_M;
    const int gsize = least(bands - first_m, GROUP_M);
    const int r = tile % per_group;
    tm = first_m + r % gsize;
    tn = r / gsize;
}

// c U / G, where CTA c's share of a length U begins (U = share x G + share_rem).
MGX_HD long long sk_begin(const Cut &p, unsigned c, unsigned grid)
{
    return c * p.share + c * (unsigned)p.share_rem / grid;
}

// CTA whose share holds unit u (sk_begin(c) <= u < sk_begin(c + 1)).
MGX_HD int sk_owner(long long u, long long U, long long G) { return (int)(((u + 1) * G + U - 1) / U - 1); }

// Stream-K units are the K blocks of the tiles, in raster order.  They cost w_full each, those of a last
// band of one or two strips w_last; where a unit starts on that scale, and the whole product's length.
MGX_HD long long sk_start(const Cut &p, long long x)
{
    return x < p.sk_full ? x * p.w_full : p.sk_full * p.w_full + (x - p.sk_full) * p.w_last;
}

// The first unit that starts at `pos` or later.
MGX_HD long long sk_unit(const Cut &p, long long pos)
{
    const long long rest = pos - p.sk_full * p.w_full;
    if (p.w_full == 1) return pos;
    return rest <= 0 ? (pos + p.w_full - 1) / p.w_full : p.sk_full + (rest + p.w_last - 1) / p.w_last;
}

// Which piece of its tile a stream-K item is, and where its partial sums go: a CTA has two slots, for a
// tile that its share begins with (0) and for one that it ends with (1).
struct Piece {
    int c0, pieces;  // the tile's first CTA, and how many share it
    int index;       // this CTA's piece
    int slot;        // this CTA's slot
    int slot0;       // the first piece's slot in CTA c0; the others begin their shares: slot 0
};

MGX_HD Piece piece_of(const Cut &p, const Item &it, unsigned cta, unsigned grid)
{
    const long long t0 = (long long)it.tile * p.kblocks;
    Piece q;
    q.c0 = sk_owner(sk_start(p, t0), p.length, grid);
    q.pieces = sk_owner(sk_start(p, t0 + p.kblocks - 1), p.length, grid) - q.c0 + 1;
    q.index = (int)cta - q.c0;
    q.slot = t0 + it.kb_begin == sk_unit(p, sk_begin(p, cta, grid)) ? 0 : 1;
    q.slot0 = sk_unit(p, sk_begin(p, (unsigned)q.c0, grid)) == t0 ? 0 : 1;
    return q;
}

// The work of one CTA, shared by the producer and the consumers: the units that start in its equal
// share of the product's length.
//   Regular: the units of all (band, K slice) rows, in that order, cut into pieces no wider than a
//   tile.  A share that runs on into another band works on two narrower pieces, which load A
//   twice and leave some warps without a unit, so each row is given `skew` virtual units at its
//   start that carry no work.
//   Stream-K: the pieces of consecutive tiles' K ranges.
template <bool STREAMK, typename Unit>
struct Walk {
    Unit x, x_end;  // the share's next unit and its end

    // (32 bits hold every position: make_cut sees to it)
    static MGX_HD unsigned row_unit(const Cut &p, unsigned pos)
    {
        const unsigned len = (p.ucols + p.skew) * p.w_full, head = p.skew * p.w_full;
        unsigned slice = 0;
        if (p.ksplit > 1) {
            const unsigned slice_len = (unsigned)p.length / (unsigned)p.ksplit;
            slice = pos / slice_len;
            pos -= slice * slice_len;
        }
        const unsigned band = least(pos / len, (unsigned)p.bands - 1u), off = pos - band * len;
        const unsigned w = band == p.bands - 1u ? p.w_last : p.w_full;
        unsigned first = off <= head ? 0u : off - head;
        if (w > 1) first = (first + w - 1) / w;
        return (slice * p.bands + band) * p.ucols + first;
    }

    MGX_HD void init(const Cut &p, unsigned cta, unsigned grid)
    {
        const long long begin = sk_begin(p, cta, grid), end = sk_begin(p, cta + 1, grid);
        if constexpr (STREAMK) {
            x = sk_unit(p, begin);
            x_end = sk_unit(p, end);
        } else {
            x = row_unit(p, (unsigned)begin);
            x_end = row_unit(p, (unsigned)end);
        }
    }

    MGX_HD bool next(const Cut &p, Item &it)
    {
        if (x >= x_end) return false;
        if constexpr (STREAMK) {
            it.tile = (int)(x / p.kblocks);
            int tn;
            tile_coords(p, it.tile, it.band, tn);
            it.u0 = tn * p.tile_units;
            it.units = least(p.tile_units, p.ucols - it.u0);
            it.slice = 0;
            it.kb_begin = (int)(x - (long long)it.tile * p.kblocks);
            it.kb_end = (int)least((long long)p.kblocks, it.kb_begin + (long long)(x_end - x));
            x += it.kb_end - it.kb_begin;
        } else {
            const unsigned row = x / (unsigned)p.ucols;
            const int off = (int)(x - row * p.ucols);
            const int run = least(p.ucols - off, (int)(x_end - x));  // the row's units in this share
            const int pieces = (run + TILE_UNITS - 1) / TILE_UNITS;
            it.slice = p.ksplit > 1 ? row / p.bands : 0;
            it.band = row - it.slice * p.bands;
            it.u0 = off;
            it.units = (run + pieces - 1) / pieces;
            it.kb_begin = it.slice * p.kb_split;
            it.kb_end = least(p.kblocks, it.kb_begin + p.kb_split);
            x += it.units;
        }
        it.strips = it.band == p.bands - 1 ? p.strips_last : 2;
        return true;
    }
};

// A consumer warp's strip and part of the tile's units.  Warps cw, cw + 4, ... share a sub-partition: its
// 16 rows of a whole band, so an uneven split of the units does not unbalance anything.  One or two
// strips are spread over all sub-partitions, a column's units over neighbours.
MGX_HD void warp_part(const Item &it, int cw, int &strip, int &u_first, int &units)
{
    strip = cw & ((1 << it.strips) - 1);
    const int sharers = CWARPS >> it.strips, per = (it.units + sharers - 1) >> (4 - it.strips);
    u_first = (cw >> it.strips) * per;
    const int left = least(per, it.units - u_first);
    units = left > 0 ? left : 0;
}

// Bands, units and stream-K tiles of an m x n product (tiles as even in width as the units allow, so a
// ragged last tile wastes little: 1281 columns are eleven tiles of 15 units, not ten of 16 and one).
inline Cut shape_cut(int m, int n, int k)
{
    Cut c = {};
    c.bands = (m - 1) / BM + 1;
    c.ucols = (n - 1) / UNIT + 1;
    c.tiles_n = (c.ucols + TILE_UNITS - 1) / TILE_UNITS;
    c.tile_units = (c.ucols + c.tiles_n - 1) / c.tiles_n;
    c.kblocks = (k - 1) / BK + 1;
    return c;
}

// CTAs of a stream-K launch.
inline int streamk_grid(const Cut &c, int sms)
{
    const long long units = (long long)c.bands * c.tiles_n * c.kblocks;
    return units < sms ? (int)units : sms;
}

enum class CutMode { kWhole, kPanels, kStreamK };

// The cut of an m x n x k product (all positive) on `sms` SMs into ksplit slices of kb_split K blocks (1 and
// all but for CutMode::kWhole); *grid: its CTAs.
inline Cut make_cut(int m, int n, int k, int ksplit, int kb_split, CutMode mode, int sms, int *grid)
{
    Cut p = shape_cut(m, n, k);
    const bool streamk = mode == CutMode::kStreamK;
    p.ksplit = ksplit;
    p.kb_split = kb_split;
    const long long units = (long long)p.bands * p.ucols * ksplit;
    *grid = streamk ? streamk_grid(p, sms) : units < sms ? (int)units : sms;
    // A band crossing costs a CTA about two units of time (777 x 1282 x 6000: 419 us without, 404 with
    // one and 388 with two virtual units; N = 1024 75.3, 70.8, 69.1).  With shares of a few units the
    // virtual ones would take whole shares away, so they are left out there.
    p.skew = units >= 8ll * *grid ? 2 : 0;
    // A last band of one or two strips (not in the panel form, see its kernel).  Stream-K: a CTA without
    // a unit would be counted among a tile's pieces, so shares are no shorter than the longest unit.
    // Weighed only from shares of four whole units on: below that the weights make more pieces of the other
    // tiles, whose sums cost more than the balance gives (71 x 201 x 2587, 2 units, 53.8 us with weights, 38.5
    // without; 400^3, 2, 20.6 and 18.3; 65 x 65 x 8192, 3, 96 and 82; the line at 8 or 16 changes nothing more).
    // Where every CTA has one unit at most the weights would only move units together: 80 x 512 x 1024
    // 13.0 us without them, 13.6 with.
    p.strips_last = 2;
    p.w_full = p.w_last = 1;
    const int strips = (m - (p.bands - 1) * BM + 15) / 16;
    if (strips <= 2 && mode != CutMode::kPanels) {
        const int w = strips == 1 ? COST_1 : COST_2;
        const long long row = (long long)p.tiles_n * p.kblocks;
        const bool weigh = p.bands == 1 ? false
                           : streamk    ? row * ((p.bands - 1ll) * COST + w) >= 4ll * *grid * COST
                                        : units > sms;
        if (weigh) {
            p.w_full = COST;
            p.w_last = w;
        }
        if (weigh || p.bands == 1 || !streamk) p.strips_last = strips - 1;
    }
    if (streamk) {
        p.sk_full = (long long)(p.w_last < p.w_full ? p.bands - 1 : p.bands) * p.tiles_n * p.kblocks;
        p.length = p.sk_full * p.w_full + ((long long)p.bands * p.tiles_n * p.kblocks - p.sk_full) * p.w_last;
    } else {
        auto length = [&] {
            return ksplit * ((p.bands - 1) * (long long)(p.ucols + p.skew) * p.w_full + p.skew * p.w_full +
                             (long long)p.ucols * p.w_last);
        };
        p.length = length();
        if (p.length > 0xffffffffll) {
            // Walk's positions are 32 bits wide.  Without the virtual units and the weights the length is the
            // number of units, each 512 bytes of C or of a slice's product at least: 2^32 are 2 TiB.
            p.skew = 0;
            p.w_full = p.w_last = 1;
            p.length = length();
        }
    }
    p.share = p.length / *grid;
    p.share_rem = (int)(p.length - p.share * *grid);
    return p;
}

}  // namespace fp64
}  // namespace mgx
