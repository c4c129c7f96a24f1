// fi_tile2d_map.h -- where the regions and tiles of fi_tile2d.cu lie along a dimension.  Plain
// C++, so that the choice can be checked for every size without a GPU.
#pragma once

#ifdef __CUDACC__
#define FI_HD __host__ __device__ __forceinline__
#else
#define FI_HD inline
#endif

namespace fi {

constexpr int kTile2DSMs = 148;

struct Tile2DPlan {
    int shape;  // region shape
    int k;      // most iterations of one launch
};

// positions of a dimension of n cells that tiles own (the ghosts go with the ones beside them):
// the vertices, or the cells where it is periodic
FI_HD int t2_last(int n, bool per) { return per ? n : n + 1; }

// tiles of t positions along it
FI_HD int t2_tiles(int n, int t, bool per) { return (t2_last(n, per) + t - 1) / t; }

// Tile b starts at 1 + b t - t2_shift.  At the end of a bounded dimension the ghosts follow from
// the cell n, which has to lie in the part of the region that comes out right: where whole tiles
// would leave the last node n + 1 to a tile of its own, all of them start one position earlier
// (the first at the ghost 0), so that the last one starts at n.  The tiles keep their size: FP64
// 96^2 takes 1.40 us an iteration, 2.54 with tiles of two rows.
FI_HD int t2_shift(int n, int t, bool per) { return !per && n % t == 0 ? 1 : 0; }

// whether the tile at `first` writes position q: its own ones, and the ghosts beside them
FI_HD bool t2_owned(int q, int first, int t, int n, bool per) {
    const int last = t2_last(n, per);
    if (q >= first && q < first + t && q <= last) return true;
    return !per && ((q == 0 && first == 1) || (q == last + 1 && last >= first && last < first + t));
}

// Region shapes: 0 = 32 x 16, one row a thread, one CTA per SM; 1 = 32 x 32, two rows, one;
// 2 = 32 x 32, two rows, two CTAs per SM (64 registers).
//
// A launch costs about 4 us that k iterations share (launch, first loads, last stores);
// deeper launches recompute more.  While the tiles of a shape fit the SMs at once, the
// deepest such launch is best, on the smaller region (an iteration of it takes 0.5 us
// against 1.6): FP64 us per iteration, reference-shaped -> chosen (others): 128^2
// 13.8 -> 1.37 at 32x16 k = 5 (k = 3: 1.73; 32x32 k = 10: 1.91); 200^2 2.37 at 32x32
// k = 6 (32x16 k = 2: 2.27, k = 4: 2.81); 300x240 2.67 at k = 4 (k = 3: 2.98).  Beyond that
// two CTAs per SM hide each other's loads: 1021x509 21.9 -> 10.98 at k = 4 (k = 3 11.2,
// k = 2 12.2, one CTA per SM 12.1), FP32 7.8 (9.1); 1224x1000 24.0, FP32 15.9.
inline Tile2DPlan tile2d_plan(int n0, int n1) {
    auto tiles = [&](int rx, int ry, int k) {
        return (long long)t2_tiles(n0, rx - 2 * k, false) * t2_tiles(n1, ry - 2 * k, false);
    };
    for (int k = 6; k >= 3; k--)
        if (tiles(32, 16, k) <= kTile2DSMs) return {0, k};
    for (int k = 10; k >= 4; k--)
        if (tiles(32, 32, k) <= kTile2DSMs) return {1, k};
    return {2, 4};
}

}  // namespace fi
