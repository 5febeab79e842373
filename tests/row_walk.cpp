// The walks of csrc/row_walk.h for the tests.
#include "row_walk.h"

extern "C" void row_walk_run(int l, int64_t rows, int64_t* out) {
    const eup::RowWalk w = eup::row_walk(l, rows);
    const int64_t v[] = {w.l, w.lg, w.span, w.pieces, w.rows, w.units};
    for (int t = 0; t < 6; ++t) out[t] = v[t];
}
extern "C" void plane_split_run(int l, int m, int n, int axis, int64_t* out) {
    const eup::PlaneSplit p = eup::plane_split(l, m, n, axis);
    const int64_t v[] = {p.tx, p.ty, p.planes, p.w.rows, p.w.shares, p.w.xblocks, p.w.plane, p.w.row, p.blocks(), p.scratch(axis)};
    for (int t = 0; t < 10; ++t) out[t] = v[t];
}
