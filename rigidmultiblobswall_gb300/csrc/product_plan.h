// How the wall and free-space products split their work, and the scratch that
// takes: rules of sizes and limits alone, with no CUDA in them.
#pragma once
#include <stddef.h>

#include <algorithm>
#include <cmath>

namespace rmw {

constexpr int kPlanTile = 128;        // blobs per tile of the symmetric kernels
constexpr int kSplitMax = 64;         // CTAs per tile pair at most
constexpr double kSplitBytes = 64e6;  // partial sums of a split product (three components): they stay in L2

inline int sym_tiles(int n) { return (n + kPlanTile - 1) / kPlanTile; }

// partial sums of one slot per tile: `comps` (3, or 6 for [U; W]) doubles per blob and tile
inline double sym_slot_bytes(int n, int comps) { return (double)sym_tiles(n) * comps * (double)n * sizeof(double); }

// How many CTAs share the steps of a tile pair.  Below about 4,000 blobs the
// tile pairs alone leave SMs idle (2,048 blobs: 136 of them); the split fills
// the GPU with the symmetric kernel's work per pair where the one-sided kernel
// used to do each pair twice (2,048 blobs: FP64 UF 961 -> 189 us, df64 181 ->
// 71).  With P tile pairs, s CTAs each and a CTA's start and end worth e steps,
// an SM takes (P s / 152 + d)(128 / s + e) step times, d the uneven end of the
// grid: least at s = sqrt(152 * 128 d / (e P)) = sqrt(K / P).  Measured by s,
// us: FP64 UF 2,048 blobs 8: 191, 10: 189, 12: 192, 17: 199; 3,000 4: 372,
// 6: 370, 8: 374, 12: 383; 5,003 3: 942, 4: 929, 6: 940, 7: 948; 10,752
// 1: 3,769, 2: 3,735, 3: 3,732.  df64 UF 1,000 blobs 8: 38, 16: 39, 22: 44,
// 32: 50; 2,048 4: 69, 9: 71, 16: 77; 5,003 2: 281, 3: 270, 4: 266, 6: 270;
// 10,752 1: 1,009, 2: 1,027.  FP64 periodic, whose steps are nine times as
// long: 1,500 blobs 16: 957, 32: 910, 43: 906, 64: 923; 4,800 4: 7,961,
// 8: 7,830, 14: 7,836.  K = 13,000, periodic 145,000, reproduces them.
// Where even 64 CTAs per pair are fewer than 16 per SM (up to 1,024 blobs), in
// FP64 the split whose busiest SM has least to do (504 blobs 26: 41.5,
// 32: 43.0, 43: 38.8, 64: 48.0; 1,000 8: 75, 16: 71, 32: 80).
inline int sym_split_rule(bool fp64, bool periodic, int n)
{
    const double nt = (double)sym_tiles(n), pairs = 0.5 * nt * (nt + 1);
    int s = 1;
    if (fp64 && pairs * kSplitMax < 16 * 152.0) {
        const double ends = periodic ? 0.05 : 0.4;
        double cost = 0.0;
        for (int c = 1; c <= kSplitMax; ++c) {
            const double t =
                std::max(std::ceil(pairs * c / 152.0), 2.0) * (std::ceil((double)kPlanTile / c) + ends);
            if (c == 1 || t < 0.99 * cost) {
                cost = t;
                s = c;
            }
        }
    } else {
        s = (int)std::min((double)kSplitMax, std::sqrt((periodic ? 145000.0 : 13000.0) / pairs) +
                                                 (fp64 ? 0.5 : 0.05));  // whole df64 pairs have constant bounds
    }
    return s;
}

// The rule's split, or the finest below it whose partial sums stay within
// kSplitBytes and `budget` and, with the `packed` bytes of records, within
// the scratch cap (0 = none): a cap that holds the unsplit product never
// costs the symmetric kernel.
inline int sym_split(bool fp64, bool periodic, int n, int comps, double packed, double budget, double cap)
{
    const double slot = sym_slot_bytes(n, comps), most = std::min(kSplitBytes * comps / 3, budget);
    int s = sym_split_rule(fp64, periodic, n);
    while (s > 1 && (slot * s > most || (cap > 0 && packed + slot * s > cap))) --s;
    return std::max(1, s);
}

// Partial sums that a symmetric product's buffer has room for: at least what
// any smaller product takes, whose split may be finer (df64: 22 MB at 10,752
// blobs, 38 MB at 10,000), so that a buffer that served n blobs serves every
// smaller n, also where it must not grow (a stream capture).
inline double sym_reserve_bytes(int n, int comps)
{
    const double slot = sym_slot_bytes(n, comps);
    return std::max(slot, std::min(kSplitBytes * comps / 3, kSplitMax * slot));
}

// The one-sided kernels' source chunks: enough CTAs to fill the 152 SMs
// several times over, at least 256 sources each.
inline int coarse_chunks(int n)
{
    const int tiles = sym_tiles(n);
    const int s = std::min((152 * 8 + tiles - 1) / tiles, std::max(1, n / 256));
    return std::max(1, std::min(s, kSplitMax));
}

// The same in FP64 and df64 (periodic products, fewer than 256 blobs): the
// split whose busiest SM has the least to do, counting a tile's staging as two
// sources; an SM needs about two FP64 or four df64 CTAs to keep its pipe busy.
// coarse_chunks left 1,500 periodic blobs on 60 CTAs.  Finer than that only
// while the partial sums stay within kSplitBytes and, with the packed records,
// within the scratch cap (0 = none).
inline int fine_chunks(bool fp64, int n, double packed, double cap)
{
    const int base = coarse_chunks(n), tiles = sym_tiles(n), fill = fp64 ? 2 : 4;
    const double one = 3.0 * (double)n * sizeof(double);
    int best = base;
    long long cost = -1;
    for (int c = 1; c <= kSplitMax && c <= std::max(base, n / 8); ++c) {
        if (c > base && (one * c > kSplitBytes || (cap > 0 && packed + one * c > cap))) break;
        const long long ctas = ((long long)tiles * c + 151) / 152;
        const long long t = std::max<long long>(ctas, fill) * ((n + c - 1) / c + 2);
        if (cost < 0 || t < cost) {
            cost = t;
            best = c;
        }
    }
    return best;
}

// as sym_reserve_bytes, for fine_chunks
inline double fine_reserve_bytes(int n)
{
    const double one = 3.0 * (double)n * sizeof(double);
    return std::max(one * coarse_chunks(n), std::min(kSplitBytes, kSplitMax * one));
}

}  // namespace rmw
