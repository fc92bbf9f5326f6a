// Which groups of a pass go to the tcgen05 kernels.  Plain C++, without the CUDA headers, so
// that the rule can be tested where there is no GPU.
#pragma once

namespace bivmoe {

constexpr int kSmallTile = 8;   // rows for which the small groups' kernels read a group's weights once

// Groups of at least `min` rows (0: none) go there, if without that the small groups' kernels
// would read at least `worth` bytes of their weights again: all tiles of a group but its first
// one read tile_bytes (sh_tile_bytes: the shared expert's group) that came with the first.
struct BigGroups {
    int min = 0;
    long long worth = 0, tile_bytes = 0, sh_tile_bytes = 0;
};

// K-slices of gate+up, then of down, that a chunk is walked through; from about 32 on a group has
// chunks enough to fill the chip by itself, and longer rows cost no more before that.
inline long long big_slices(int e, int ff) { return (e + ff) / 256 < 32 ? (e + ff) / 256 : 32; }

// What those bytes have to come to.  The tcgen05 kernels walk a chunk of 128 rows at a time
// through all K-slices, one after the other, with one chunk a block, so what they cost before
// they are any faster grows with the length of the rows, where the other kernels spread a group
// over the whole chip; reading weights again costs about 0.1 us a MB.  A pass that asks for them
// in vain has two launches more, 6 us: for Q8_0 the line does not lie below 176 tiles, which
// keeps passes of few rows clear of that (BF16 gains too much there: 16 experts of 2048 / 512,
// 200 rows, 717 MB, 82 us against 141).
// Measured with 9 shapes of 512 / 256 to 4096 / 14336, 8 to 512 experts, 12 to 3072 rows, balanced
// to Zipf-skewed, all large groups by the tcgen05 kernels / none, us:
//   Q8_0   2048 / 512    381 MB 80 / 94, 501 MB 186 / 182, 678 MB 139 / 154
//          4096 / 1536   1103 MB 455 / 438, 1223 MB 702 / 719, 3280 MB 576 / 721
//          4096 / 14336  749 MB 567 / 528, 1497 MB 487 / 528, 5423 MB 655 / 932, 26000 MB 1169 / 3191
//   BF16   2048 / 512    396 MB 201 / 184, 573 MB 121 / 133
//          4096 / 1536   1170 MB 408 / 393, 2605 MB 653 / 704
//          4096 / 14336  705 MB 696 / 534, 1408 MB (four experts, none shared) 402 / 451, 3520 MB
//                        741 / 872, 48900 MB 952 / 5520
// (One number of tiles for all sizes, as found at 2048 / 512, took the second figure of the last
// line of each.)
inline long long big_worth(bool bf16, int e, int ff, long long tile_bytes) {
    const long long slices = big_slices(e, ff), mb = 1000000;
    if (bf16) return (100 + 40 * slices) * mb;
    const long long tiles = 176 * tile_bytes, bytes = (300 + 40 * slices) * mb;
    return tiles < bytes ? tiles : bytes;
}

// The same for a group that runs by itself (the shared expert's, on a rank of an expert-parallel
// layer), which the tcgen05 kernels have the whole chip for.  Measured likewise, us: Q8_0, 2048 /
// 512: 164 MB 58 / 46, 414 MB 60 / 77; 4096 / 1536: 380 MB 87 / 77, 980 MB 89 / 151; 4096 / 14336:
// 374 MB 140 / 130, 1310 MB 171 / 224.  BF16, 2048 / 512: 308 MB 63 / 69, 120 MB 60 / 46; 4096 /
// 1536: 264 MB 91 / 77, 717 MB 97 / 120; 4096 / 14336: 704 MB 240 / 253, 2466 MB 241 / 370.
inline long long big_worth_alone(int e, int ff) { return (200 + 8 * big_slices(e, ff)) * 1000000; }

// The most bytes that any routing of n rows to k experts each makes the small groups' kernels
// read again: no group is larger than n, so there are at least k of them, and a group of r rows
// has (r - 1) / kSmallTile such tiles.
inline long long big_reach(const BigGroups& b, int n, int k, int has_shared) {
    if (n < 1) return 0;
    return (long long)k * (n - 1) / kSmallTile * b.tile_bytes + (has_shared ? (n - 1) / kSmallTile * b.sh_tile_bytes : 0);
}
// `b` for a pass of n rows: `min` 0 when no group can be large enough, or all of them not worth it
inline BigGroups big_for(BigGroups b, int n, int k, int has_shared) {
    if (n < b.min || big_reach(b, n, k, has_shared) < b.worth) b.min = 0;
    return b;
}

}  // namespace bivmoe
