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
// second pass over the listed voxels (launch_pbb_step).  The second pass costs a launch, the
// 32-byte sectors that its voxels lie in and, in 16-bit storage above all, the voxels; the one
// pass a share of the plain step whatever the field.  us per step, two passes / one, by the share
// of sectors (of 8 nodes) touched, with voxels anywhere, and by the share of voxels, in a block:
//   192x96x96, anywhere 8 %, 15 %, 28 %, 39 %, 49 %, 64 %:
//     FP32 74/84 86/85 103/86 111/87 114/87 118/87, FP64 120/131 138/132 167/133 184/133 193/133 206/133,
//     FP16 79/101 82/103 82/106 92/107 97/107 110/108
//     block 8 %, 15 %, 20 %, 25 %, 35 %: FP32 65/83 77/83 85/83 91/83 100/84,
//     FP64 114/131 128/131 138/131 147/131 163/131, FP16 65/100 78/101 96/101 109/101 130/102
//   384x192x192, anywhere 8 %, 15 %, 28 %, 39 %, 49 %, 64 %:
//     FP32 521/518 622/523 729/529 791/532 822/534 850/534, FP16 371/541 428/553 477/568 514/577 561/581 637/585
//     block 8 %, 15 %, 20 %, 25 %: FP32 419/514 474/517 507/518 540/518, FP16 385/531 521/535 614/537 705/538
//   96x64x64, anywhere 8 %, 28 %, 39 %, 49 %, 64 %: FP32 27/30 28/31 29/31 29/31 30/31,
//     FP64 40/45 43/46 46/46 48/46 50/46, FP16 42/39 42/40 41/40 41/40 41/40
//   48x24x12, any field: FP32 15-18/9.5, FP64 16-19/11.5, FP16 26-33/11.5
//   64x48x40 and 127x31x33, any field: FP32 17-20/13-16, FP64 20-22/18-20, FP16 26-31/18-21
// Steps that an adjoint runs again sum no force.  Two passes less one, us per such step:
//   192x96x96, anywhere 8 %, 15 %, 28 %, 39 %: FP32 11 23 38 47, FP64 10 27 55 72, FP16 -2 0 0 9;
//     block 8 %, 15 %, 20 %: FP32 1 9 14, FP64 1 12 19, FP16 -14 -3 12
//   384x192x192, anywhere 8 %, 28 %, 39 %, 49 %: FP32 113 318 373 405, FP16 -141 -50 -19 27;
//     block 12 %, 15 %, 20 %: FP32 23 51 82, FP16 -63 1 94
//   96x64x64, any field: FP32 4..9, FP64 2..16, FP16 2..15
// So: one pass on lattices of up to 2^17 nodes; beyond, for fields that touch more than a share of
// the sectors, in sixteenths, below / from 2^20 nodes:
//            with the force                 without
//   FP32     10 / 3                         2 / 2
//   FP64      5 / 3                         2 / 2
//   16-bit    6 / 10, or 7/32 of the voxels 3 / 6, or 5/32 of the voxels
// which takes two passes wherever they are more than a few per cent faster.  EUP_STEP_VARIANT bit
// 13: always two passes, bit 14: one wherever it is allowed.
// Rows of more than 128 * most nodes always take two passes, whose list is dealt to a bounded
// grid: their one-pass blocks would store more partial sums than there is room for.
inline bool pbb_in_one_pass(int l, int64_t N, int sbytes, int variant, int64_t sectors, int64_t voxels, bool force,
                            int most) {
    if (!pbb_row_fits(l, most)) return false;
    if (variant & (8192 | 16384)) return (variant & 16384) != 0;
    if (N <= 131072) return true;
    const bool large = N >= (1 << 20);
    int sixteenths = 2;
    if (sbytes == 2) sixteenths = force ? (large ? 10 : 6) : (large ? 6 : 3);
    else if (force) sixteenths = large ? 3 : (sbytes == 4 ? 10 : 5);
    if (16 * sectors > sixteenths * ((N + 7) / 8)) return true;
    return sbytes == 2 && large && 32 * voxels > (force ? 7 : 5) * N;
}

}  // namespace eup
