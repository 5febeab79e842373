// The rule and the grid of csrc/pbb_plan.h for the tests: out = {one pass, blocks, threads, nbx,
// rows per block, groups of rows}.
#include "pbb_plan.h"

extern "C" void pbb_plan_run(int l, int m, int n, int sbytes, int variant, int64_t sectors, int64_t voxels, int force,
                             int most, int64_t* out) {
    out[0] = eup::pbb_in_one_pass(l, (int64_t)l * m * n, sbytes, variant, sectors, voxels, force != 0, most);
    const eup::PbbSplit s = eup::pbb_split(l, m * n, force ? most : 0);
    out[1] = s.blocks();
    out[2] = s.threads;
    out[3] = s.nbx;
    out[4] = s.each;
    out[5] = s.slots;
}
