// matvec_rules.h -- how the tensor-core mat-vec (matvec_tc.cu) splits a pass:
// what its launch accepts, and the tile and K-chunk choices, which have to
// stay within that.  Host arithmetic only.
#pragma once
#include <cstddef>

namespace ipb {

// DB rows per pipeline stage (bytes of K): 64, so a stage is 16 KB of DB
// plus 64 bytes of every query plane (a SWIZZLE_64B tile), 32 KB at 32
// queries, and six stages fit (three with 128-row stages).  Deeper DB
// prefetch (an L2 prefetch ahead of the ring, or a separate deeper DB ring)
// measured slower: the SMs drift apart and the DB rows lose locality.
constexpr int kKT = 64;
constexpr int kMT = 256;          // m' rows per tile (two M = 128 MMAs)
constexpr int kKChunk = 32768;    // rows per exact s32 accumulation
constexpr int kPlanes = 7;        // CRT byte planes per query

// K chunks are whole stages, at most kKChunk rows, and divide the rows.
inline bool mv_kchunk_ok(size_t rows, int kchunk_rows) {
    return kchunk_rows > 0 && kchunk_rows <= kKChunk && kchunk_rows % kKT == 0 && rows % (size_t)kchunk_rows == 0;
}

// Tiles per work item for a pass of nq queries over a DB of ld columns per
// row.  Two while their accumulators fit TMEM (18 queries), if the DB is small
// enough for the tail of its few items to count or the batch large enough for
// the planes to, and if the accumulators are double-buffered or an item long
// enough for that not to matter (16 queries, 640 rows an item: 31 us with one
// tile, 36 with two; 2048 rows 214 / 217; 8192 rows 214 / 196).
// Both sides of the lines, 32768 rows, one tile / two.  By size, 1 query: 3.2 GB
// 482 / 461 us, 4.3 677 / 648, 5.4 838 / 835 (5 queries 835 / 866), 6.4 1030 / 950,
// 7.5 1155 / 1153, 8.6 1212 / 1235, 17.2 2380 / 2454: two gain up to 4.3 GB and lose
// from 8.6, and between them the items' last wave decides.  By queries over 17.2
// GB, ms: 2 2.48 / 2.54, 4 2.51 / 2.57, 5 2.68 / 2.59, 6 2.76 / 2.67, 8 2.82 / 2.68, 12
// 2.90 / 2.85.  pairs: the launch's tiles pair up
// (an even number of them in every column range).
inline int mv_tiles(int nq, size_t rows, size_t ld, int kchunk_rows, bool pairs) {
    const int npad = (kPlanes * nq + 15) / 16 * 16;
    if (!pairs || 4 * npad > 512 || (8 * npad > 512 && kchunk_rows < 4096)) return 1;
    return 2.0 * (double)rows * (double)ld <= 6e9 || nq >= 6 ? 2 : 1;
}
// Rows per exact s32 accumulation: at most 32768, halved while there are
// fewer than two work items per SM and the half is whole stages (17408 rows
// end at 1088).
inline int matvec_tc_kchunk_rows(size_t rows, size_t cols, int num_sms, int nq) {
    const size_t mtiles = (2 * cols) / kMT, sms = (size_t)num_sms;
    const bool pairs = mtiles % 2 == 0;
    auto chunk = [&](size_t tiles_per_item) {
        size_t kc = rows < (size_t)kKChunk ? rows : (size_t)kKChunk;
        while (mtiles * (rows / kc) < tiles_per_item * 2 * sms && kc > 1024 && kc % (2 * kKT) == 0) kc /= 2;
        return (int)kc;
    };
    const int one = chunk(1);
    if (mv_tiles(nq, rows, cols, one, true) == 1) return one;
    const int two = chunk(2);
    // Tiles that do not pair up: the chunks are halved once more where the last
    // wave of items is fuller then (1 query: 32768 x 38528, 301 items in three
    // waves to 602 in five, 470 -> 411 us; 8192 x 20608, 322 to 644, 72 -> 65), not
    // where only the second chunk's sum is added (4096 x 49024, 383 in three to
    // 766 in six: 70 -> 77).
    if (!pairs) {
        const size_t n = mtiles * (rows / (size_t)one);
        if (2 * ((n + sms - 1) / sms) <= (2 * n + sms - 1) / sms) return one;
    }
    // Pairs: once more where that leaves the pass on two tiles per item (21
    // groups, 8 queries: 768 -> 708 us, one tile 730).
    return mv_tiles(nq, rows, cols, two, true) == 2 ? two : one;
}
// DB columns per work item of a pass of nq queries over ranges of cols columns.
inline int matvec_tc_item_cols(int nq, size_t rows, size_t ld, size_t cols, int kchunk_rows) {
    return kMT / 2 * mv_tiles(nq, rows, ld, kchunk_rows, (2 * cols) / kMT % 2 == 0);
}

}  // namespace ipb
