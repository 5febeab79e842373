// How the diagnostics that sum over all nodes are dealt to warps and blocks.  Host code, without
// CUDA.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace eup {

// Lanes a row of l nodes takes of a warp: a power of two, all 32 from 17 nodes on.
inline int row_lanes_log2(int l) {
    int lg = 0;
    while (lg < 5 && (1 << lg) < l) ++lg;
    return lg;
}

// Units of a warp: 32 >> lg rows side by side (short rows), or a piece of `span` nodes of one row,
// `pieces` to a row where the lattice has too few rows for the device (long ones).
struct RowWalk {
    int l, lg, span, pieces;
    int64_t rows, units;
};

// Monitor and region sums.  A row in pieces where there are fewer row units than 32 warps on each
// of the 148 SMs: a warp per row, with all its lanes along it, took the monitor 906 us at
// 65536x2x2 FP32, 92 at 4096x8x8, 490 at 16384x4x64 and 106 at 2x512x512; now 33, 33, 98 and 45.
inline RowWalk row_walk(int l, int64_t rows) {
    RowWalk w;
    w.l = l;
    w.rows = rows;
    w.lg = row_lanes_log2(l);
    const int64_t side = 32 >> w.lg, groups = (rows + side - 1) / side, most = ((int64_t)l + 31) / 32;
    const int64_t pieces = std::max<int64_t>(1, std::min(most, (148 * 32 + groups - 1) / groups));
    const int64_t tiles = (most + pieces - 1) / pieces;  // of 32 nodes, to a piece
    w.span = (int)std::min<int64_t>(32 * tiles, 1 << 30);
    w.pieces = (int)((l + (int64_t)w.span - 1) / w.span);
    w.units = groups * w.pieces;
    return w;
}

// Plane means: blocks of 128 threads, `tx` along x and the rest over rows; a plane (axis 0: all
// rows at once, every thread keeping its x) is dealt to xblocks * shares of them.
struct PlaneWalk {
    int l, rows;          // rows of a plane (all rows for axis 0)
    int shares, xblocks;  // thread blocks a plane is dealt to, by rows and along x
    int64_t plane, row;   // row index of row t of plane p: p * plane + t * row
};
struct PlaneSplit {
    PlaneWalk w;
    int tx, ty, planes;
    int64_t blocks() const { return (int64_t)planes * w.shares * w.xblocks; }
    // doubles of partial sums; none where a plane is one block's
    int64_t scratch(int axis) const {
        if (axis == 0) return 4 * (int64_t)w.shares * ty * w.l;
        return w.shares * w.xblocks > 1 ? 4 * blocks() : 0;
    }
};

// As many blocks along x as a row fills, the rest over rows: a few waves of the 12 blocks an SM
// holds, but eight rows a thread at least, so that the partial sums stay below the size of the
// staging buffer they go to.  Planes of up to 24 nodes a thread are one block's where there are 32
// of them, and need no second launch to add partial sums: planes normal to y / z, FP32, with 32
// lanes to a row and two launches 79 / 79 us at 2x512x512, 43 / 43 at 8x256x256, 40 / 36 at
// 16x128x128; now 50 / 37, 36 / 35 and 33 / 34.  (One block for 32 nodes a thread, 33x64x64: 45 for 36.)
inline PlaneSplit plane_split(int l, int m, int n, int axis) {
    PlaneSplit p;
    const int lg = axis == 0 ? 5 : row_lanes_log2(l);
    p.tx = l > 64 ? 128 : (l > 32 ? 64 : 1 << lg);
    p.ty = 128 / p.tx;
    p.planes = axis == 0 ? 1 : (axis == 1 ? m : n);
    p.w.l = l;
    p.w.rows = axis == 0 ? m * n : (axis == 1 ? n : m);
    p.w.plane = axis == 1 ? 1 : m;
    p.w.row = axis == 1 ? m : 1;
    const int64_t fill = std::max<int64_t>(1, 148 * 12 * (axis == 0 ? 1 : 3) / p.planes);
    const int64_t along = (l - 1) / p.tx + 1;
    if (axis != 0 && p.planes >= 32 && along * ((p.w.rows - 1) / p.ty + 1) <= 24) {  // nodes to a thread
        p.w.xblocks = p.w.shares = 1;
        return p;
    }
    p.w.xblocks = (int)(axis == 0 ? along : std::min(along, fill));
    const int64_t most = p.w.rows / (8 * p.ty);
    p.w.shares = (int)std::max<int64_t>(1, std::min(most, fill / p.w.xblocks));
    return p;
}

}  // namespace eup
