// kv_l2.cuh — which tiles of a dense K.V stay in L2 from one K.V to the next
// (host arithmetic; the policies are those of the tile copies).
//
// A matrix of at most kL2Fits, as it is stored (rows padded), stays in L2 by
// itself and its copies carry no policy. Of a larger one, which
// least-recently-used replacement would throw out before its next use, the
// first tiles up to kL2Keep are kept (evict-last) and the others pass through
// (evict-first). 16 steps in ms / K.V back to back in us, alone:
//     MiB    no policy      all evict-first   48 MiB kept
//      36    1.27 /  4.5    1.27 /  4.5       1.27 /  4.5
//      64    1.39 /  7.5    1.38 /  7.7       1.40 /  7.8
//      68    1.74 /  8.1    1.65 /  8.3       1.66 /  8.3
//      79    1.68 /  9.3    1.56 /  9.3       1.59 /  9.3
//      98    2.57 / 14.6    2.32 / 14.0       2.16 / 13.4
//     125    2.96 / 20.1    2.70 / 19.8       2.14 / 16.0
//     250    5.08 / 39.4    4.78 / 38.9       4.33 / 34.0
//     706    13.9 / 108                       12.7 / 101
// and beside an idle handle of 250 MiB that keeps its share, to which lines
// of lower priority lose:
//      36    1.25 /  4.5    1.31 /  5.4       1.26 /  4.5
//      64    1.47 /  7.7    1.72 / 10.6       1.41 /  7.9
//      79    1.72 /  9.4    2.04 / 12.6       1.62 / 10.0
// 32 and 64 MiB kept are within 2 % of 48; without evict-first for the rest
// nothing is gained. Several live handles in alternation, no policy -> 48 MiB
// kept by each: two of 125 MiB 6.01 -> 4.28 ms a pair, four of 134 MiB 13.1
// -> 9.7 ms, four of 81 MiB 7.44 -> 7.04 ms: shares that together exceed L2
// cost nothing.
#pragma once
#include <cstdint>

constexpr int64_t kL2Keep = (int64_t)48 << 20, kL2Fits = (int64_t)64 << 20;

// Number of leading tiles to keep, -1 for no policy; tile_bytes(i) is what the
// copies of tile i read, padding included.
template <class TileBytes>
inline int64_t l2_keep_tiles(int64_t ntiles, TileBytes tile_bytes)
{
    int64_t all = 0, keep = 0, kept = 0;
    for (int64_t i = 0; i < ntiles; i++) {
        const int64_t b = tile_bytes(i);
        all += b;
        if (keep == i && kept + b <= kL2Keep) {
            keep = i + 1;
            kept += b;
        }
    }
    return all <= kL2Fits ? -1 : keep;
}
