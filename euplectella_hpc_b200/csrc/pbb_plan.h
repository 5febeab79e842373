// Which form a partial-bounce-back step takes, and how its one-pass kernel is dealt to thread
// blocks.  Host code, without CUDA.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace eup {

// Thread blocks of k_pbb_whole: nbx blocks of `threads` threads to a row, `each` rows to a block,
// `slots` groups of rows.
struct PbbSplit {
    int nbx, threads, each, slots;
    int64_t blocks() const { return (int64_t)nbx * slots; }
};

// As few rounds as `most` blocks allow (the partial sums of the force have room for so many;
// 0: none are stored), with equal numbers of rows.  A row takes nbx blocks at least: more than
// `most` of them are not for this kernel (pbb_row_fits).
inline PbbSplit pbb_split(int l, int rows, int most) {
    PbbSplit s;
    s.nbx = (l - 1) / 128 + 1;
    s.threads = ((l - 1) / s.nbx + 32) / 32 * 32;
    const int64_t at_once = most > 0 ? std::max(1, most / s.nbx) : rows;
    s.each = (int)((rows + at_once - 1) / at_once);
    s.slots = (int)(((int64_t)rows + s.each - 1) / s.each);
    return s;
}

// Whether the partial sums of one row's blocks fit in `most`: to l = 128 * most (524288 nodes).
inline bool pbb_row_fits(int l, int most) { return (l - 1) / 128 + 1 <= most; }

// A partial-bounce-back step in one pass over every node, or as the plain stream-collide and a
// second pass over the listed voxels (launch_pbb_step).  The second pass costs a launch and the
// 32-byte sectors that its voxels lie in, the one pass a share of the plain step whatever the
// field.  us per step, two passes / one:
//   192x96x96, voxels anywhere, sectors of 8 nodes touched 8 %, 15 %, 28 %, 49 %, 73 %:
//     FP32 74/83 86/84 103/85 114/86 119/87, FP64 120/131 138/132 168/132 193/133 211/133,
//     FP16 79/98 82/100 82/102 97/104 116/105;  in a block: 15 % FP32 77/82 FP64 128/130
//     FP16 78/96, 49 % 116/83 183/130 167/98
//   384x192x192, anywhere 8 %, 15 %, 28 %, 49 %: FP32 518/518 619/522 728/527 827/530,
//     FP16 372/548 430/559 478/575 564/588;  block 15 %, 49 %: FP32 469/512 715/512, FP16
//     521/540 1181/554
//   48x24x12, any field: FP32 15-18/9.5, FP64 16-19/11.5, FP16 26-33/11.5
//   64x48x40 and 127x31x33, any field: FP32 17-20/13-16, FP64 20-22/18-20, FP16 26-31/18-21;
//     96x48x48 (221k nodes): FP32 19/19, FP64 24/27, FP16 29/25
// The steps that an adjoint runs again sum no force: at 192x96x96 with 18 % of the sectors touched
// FP32 80/70, FP64 133/115, FP16 no difference.  So: one pass on small lattices, and for
// fields that touch more than 3/16 (16-bit storage 3/8) of the sectors, without the force 1/8 (3/16).
// EUP_STEP_VARIANT bit 13: always two passes, bit 14: one wherever it is allowed.
// Rows of more than 128 * most nodes always take two passes, whose list is dealt to a bounded
// grid: their one-pass blocks would store more partial sums than there is room for.
inline bool pbb_in_one_pass(int l, int64_t N, int sbytes, int variant, int64_t sectors, bool force, int most) {
    if (!pbb_row_fits(l, most)) return false;
    if (variant & (8192 | 16384)) return (variant & 16384) != 0;
    if (N <= 131072) return true;
    const int64_t sixteenths = (force ? 3 : 2) + (sbytes == 2 ? (force ? 3 : 1) : 0);
    return 16 * sectors > sixteenths * ((N + 7) / 8);
}

}  // namespace eup
