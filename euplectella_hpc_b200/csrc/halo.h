// The halo planes of one time step (CODE/SRC/bcond.bc.F90:22-690) as independent work items.
//
// The reference runs one block of loops per face, in the order front, rear, up, down, left,
// right, then the free-slip edge fixes, each block reading and writing the halo of one array.
// Here every loop iteration is an item that can run beside all others:
//
//  * every block reads interior values only, except the outflow border fix and the free-slip
//    up block on its rim (i = 0, l+1 or j = 0, m+1).  Those reads are resolved to what the
//    earlier block of the step computed (halo_rim, outflow at the clamped row), or to the value
//    of the step before;
//  * a halo value written by two blocks (only on the twelve edge lines) is stored by the last
//    one alone: a store that a later block of the step repeats is left out (halo_overwritten);
//  * the two values of the step before that the rim reads and a later block replaces,
//    a07(:,0,n) under a periodic left face and a18(:,m+1,n) under a periodic right face, are
//    read and passed on by the very item that replaces them.
//
// So the items give the reference's halo in any order (tests run them in random order against
// the oracle).  They are host code: the device runs them in the form halo_plan.cu records,
// five strided copies per face and a table for the edge lines.
// q is the reference's population number, 1..18.
#pragma once
#include <stdint.h>

#include "init_eq.h"  // EUP_HD

namespace eup {

enum : int {
    kHaloFront = 0, kHaloFrontFix, kHaloRear, kHaloUp, kHaloDown, kHaloLeft, kHaloRight, kHaloEdgeFix, kHaloBlocks
};

// Boundary flags (front, rear, right, left, up, down) and sizes.
struct HaloConf {
    int l, m, n;
    int front, rear, right, left, up, down;
    int fixes;  // free-slip edge fixes: bit 0 left-up, 1 right-up, 2 right-down, 3 left-down

    HaloConf() = default;
    HaloConf(int l_, int m_, int n_, const int bc[6])
        : l(l_), m(m_), n(n_), front(bc[0]), rear(bc[1]), right(bc[2]), left(bc[3]), up(bc[4]), down(bc[5]) {
        fixes = ((left == 3 && up == 3) ? 1 : 0) | ((right == 3 && up == 3) ? 2 : 0) |
                ((right == 3 && down == 3) ? 4 : 0) | ((left == 3 && down == 3) ? 8 : 0);
    }
};

// Iterations of a block: a = a0 .. a0+na-1 (fastest), b = b0 .. b0+nb-1.
struct HaloRange {
    int a0, na, b0, nb;
    int64_t size() const { return (int64_t)na * nb; }
};

// The iterations block b runs (none: size 0; flag 6 is an x-slab exchange face).
inline HaloRange halo_range(const HaloConf& c, int b) {
    const int l = c.l, m = c.m, n = c.n;
    const HaloRange none{0, 0, 0, 0}, xy{1, l, 1, m}, yz{1, m, 1, n}, xz{1, l, 1, n};
    switch (b) {
        case kHaloFront: return c.front == 6 ? none : c.front == 0 ? HaloRange{0, m + 1, 1, n} : yz;
        case kHaloFrontFix: return c.front == 5 ? HaloRange{1, m > n ? m : n, 0, 2} : none;
        case kHaloRear:
            return c.rear == 6 ? none : c.rear == 0 ? HaloRange{0, m + 1, 1, n} : c.rear == 1 ? yz
                                                                                           : HaloRange{0, m + 2, 0, n + 2};
        case kHaloUp: return c.up == 3 ? HaloRange{0, l + 2, 0, m + 2} : xy;
        case kHaloDown: return xy;
        case kHaloLeft: return c.left == 0 ? HaloRange{0, l + 1, 1, n} : xz;
        case kHaloRight: return c.right == 0 ? HaloRange{0, l + 1, 1, n} : xz;
        default: return c.fixes ? HaloRange{1, l, 0, 1} : none;
    }
}

inline bool halo_in(int x, int lo, int hi) { return x >= lo && x <= hi; }

// Whether block b writes population q of halo node (i, j, k).
inline bool halo_writes(const HaloConf& c, int b, int q, int i, int j, int k) {
    const int l = c.l, m = c.m, n = c.n, l1 = l + 1, m1 = m + 1, n1 = n + 1;
    const bool I = halo_in(i, 1, l), J = halo_in(j, 1, m), K = halo_in(k, 1, n);
    // no-slip blocks store one step along a tangential axis for the diagonal populations
    const bool Iup = halo_in(i, 2, l1), Idn = halo_in(i, 0, l - 1);
    const bool Jup = halo_in(j, 2, m1), Jdn = halo_in(j, 0, m - 1);
    const bool Kup = halo_in(k, 2, n1), Kdn = halo_in(k, 0, n - 1);
    switch (b) {
        case kHaloFront:
            if (i != l1 || q < 10 || q > 14) return false;
            if (c.front == 0) return K && (J || (q == 12 && j == 0));
            if (c.front == 1)
                return q == 12 ? Jdn && K : q == 13 ? J && Kdn : q == 10 ? Jup && K : q == 11 ? J && Kup : J && K;
            return c.front == 5 && J && K;
        case kHaloFrontFix:
            return c.front == 5 && i == l1 && q >= 10 && q <= 14 && ((J && (k == 0 || k == n1)) || (K && (j == 0 || j == m1)));
        case kHaloRear:
            if (i != 0 || q > 5) return false;
            if (c.rear == 0) return K && (J || (q == 1 && j == m1));
            if (c.rear == 1)
                return q == 3 ? Jdn && K : q == 4 ? J && Kdn : q == 1 ? Jup && K : q == 2 ? J && Kup : J && K;
            return c.rear == 4;
        case kHaloUp:
            if (k != n1 || !(q == 2 || q == 9 || q == 11 || q == 15 || q == 16)) return false;
            if (c.up == 0) return I && J;
            if (c.up == 3) return true;
            return q == 15 ? I && J : q == 2 ? Idn && J : q == 9 ? I && Jdn : q == 11 ? Iup && J : I && Jup;
        case kHaloDown:
            if (k != 0 || !(q == 4 || q == 6 || q == 7 || q == 13 || q == 18)) return false;
            if (c.down != 1) return I && J;
            return q == 6 ? I && J : q == 4 ? Idn && J : q == 7 ? I && Jdn : q == 13 ? Iup && J : I && Jup;
        case kHaloLeft:
            if (j != 0 || !(q == 3 || q == 7 || q == 8 || q == 9 || q == 12)) return false;
            if (c.left == 0) return K && (I || (q == 3 && i == 0));
            if (c.left == 3) return I && K;
            return q == 8 ? I && K : q == 12 ? Iup && K : q == 3 ? Idn && K : q == 7 ? I && Kdn : I && Kup;
        case kHaloRight:
            if (j != m1 || !(q == 1 || q == 10 || q == 16 || q == 17 || q == 18)) return false;
            if (c.right == 0) return K && (I || (q == 10 && i == l1));
            if (c.right == 3) return I && K;
            return q == 17 ? I && K : q == 10 ? Iup && K : q == 1 ? Idn && K : q == 18 ? I && Kdn : I && Kup;
        default:
            return I && (((c.fixes & 1) && q == 9 && j == 0 && k == n1) ||
                         ((c.fixes & 2) && q == 16 && j == m1 && k == n1) ||
                         ((c.fixes & 4) && q == 18 && j == m1 && k == 0) || ((c.fixes & 8) && q == 7 && j == 0 && k == 0));
    }
}

// Whether a block after b writes population q of halo node (i, j, k) again.  Two blocks meet
// only where two coordinates lie outside the interior.
inline bool halo_overwritten(const HaloConf& c, int b, int q, int i, int j, int k) {
    const int out = !halo_in(i, 1, c.l) + !halo_in(j, 1, c.m) + !halo_in(k, 1, c.n);
    if (out < 2) return false;
    bool again = false;
    for (int later = 0; later < kHaloBlocks; ++later)
        if (later > b) again |= halo_writes(c, later, q, i, j, k);
    return again;
}

// Outflow equilibrium at rho = 1 with the (un-normalised) momentum of x = l, :127-169:
// populations 10..14 of the halo node beyond it from the 18 moving ones.
template <typename R>
EUP_HD inline void halo_outflow(const R (&x)[18], R (&v)[5]) {
    const R xj = x[0] + x[1] + x[2] + x[3] + x[4] - x[9] - x[10] - x[11] - x[12] - x[13];
    const R yj = x[2] + x[6] + x[7] + x[8] + x[11] - x[0] - x[9] - x[15] - x[16] - x[17];
    const R zj = x[3] + x[5] + x[6] + x[12] + x[17] - x[1] - x[8] - x[10] - x[14] - x[15];
    const R rf = R(3), qf = R(1.5), t3 = R(3), one = R(1);
    const R cvsq = xj * xj + yj * yj + zj * zj;
    const R cx10 = rf * (-xj - yj) + qf * (t3 * (xj + yj) * (xj + yj) - cvsq);
    const R cx11 = rf * (-xj - zj) + qf * (t3 * (xj + zj) * (xj + zj) - cvsq);
    const R cx12 = rf * (-xj + yj) + qf * (t3 * (xj - yj) * (xj - yj) - cvsq);
    const R cx13 = rf * (-xj + zj) + qf * (t3 * (xj - zj) * (xj - zj) - cvsq);
    const R cx14 = rf * (-xj) + qf * (t3 * (xj) * (xj) - cvsq);
    const R p1 = R(1.0 / 18.0), p2 = R(1.0 / 36.0);
    v[0] = p2 * (one + cx10);
    v[1] = p2 * (one + cx11);
    v[2] = p2 * (one + cx12);
    v[3] = p2 * (one + cx13);
    v[4] = p1 * (one + cx14);
}

// Uniform inflow equilibrium, :260-321: populations 1..5 of x = 0.
template <typename R>
inline void halo_inflow(R u_inflow, R (&v)[5]) {
    const R xj = u_inflow, yj = R(0), zj = R(0);
    const R rf = R(3), qf = R(1.5), t3 = R(3), one = R(1);
    const R cvsq = xj * xj + yj * yj + zj * zj;
    const R cx01 = rf * (xj - yj) + qf * (t3 * (xj - yj) * (xj - yj) - cvsq);
    const R cx02 = rf * (xj - zj) + qf * (t3 * (xj - zj) * (xj - zj) - cvsq);
    const R cx03 = rf * (xj + yj) + qf * (t3 * (xj + yj) * (xj + yj) - cvsq);
    const R cx04 = rf * (xj + zj) + qf * (t3 * (xj + zj) * (xj + zj) - cvsq);
    const R cx05 = rf * (xj) + qf * (t3 * (xj) * (xj) - cvsq);
    const R p1 = R(1.0 / 18.0), p2 = R(1.0 / 36.0);
    v[0] = p2 * (one + cx01);
    v[1] = p2 * (one + cx02);
    v[2] = p2 * (one + cx03);
    v[3] = p2 * (one + cx04);
    v[4] = p1 * (one + cx05);
}

// Access A of the items: R the type of a value, c (HaloConf), ld(q, i, j, k) an interior value,
// old(q, i, j, k) a halo value of the step before, outflow(j, k, v) and inflow(v) the five
// populations above, lid(v, s) v plus s times the lid's force, st(b, q, i, j, k, v) the store of
// block b (to be left out where halo_overwritten).  Every item makes all its loads before its
// first store.

// What the free-slip up block reads as population q (4, 6, 7, 13 or 18) of rim node (i, j, n):
// the front or rear block's value of this step where they wrote it, else the step before's.
template <typename A>
inline typename A::R halo_rim(const A& a, int q, int i, int j) {
    const HaloConf& c = a.c;
    const bool J = halo_in(j, 1, c.m);
    if (q == 13 && i == c.l + 1) {
        if (c.front == 0 && J) return a.ld(13, 1, j, c.n);
        if (c.front == 5) {  // rows j = 0 and m+1 hold the border fix's copies of rows 1 and m
            typename A::R v[5];
            a.outflow(j < 1 ? 1 : (j > c.m ? c.m : j), c.n, v);
            return v[3];
        }
    }
    if (q == 4 && i == 0) {
        if (c.rear == 0 && J) return a.ld(4, c.l, j, c.n);
        if (c.rear == 4) {
            typename A::R v[5];
            a.inflow(v);
            return v[3];
        }
    }
    return a.old(q, i, j, c.n);
}

// One iteration (ia, ib) of a block.
template <typename A>
inline void halo_item(const A& a, int block, int ia, int ib) {
    using R = typename A::R;
    const HaloConf& c = a.c;
    const int l = c.l, m = c.m, n = c.n, l1 = l + 1, m1 = m + 1, n1 = n + 1;
    switch (block) {
        case kHaloFront: {  // x = l+1
            constexpr int b = kHaloFront;
            const int j = ia, k = ib;
            if (c.front == 0) {  // periodic, :75-105 (SERIAL corner line :90)
                if (j == 0) { a.st(b, 12, l1, 0, k, a.ld(12, 1, m, k)); return; }
                const R v10 = a.ld(10, 1, j, k), v11 = a.ld(11, 1, j, k), v12 = a.ld(12, 1, j, k),
                        v13 = a.ld(13, 1, j, k), v14 = a.ld(14, 1, j, k);
                a.st(b, 10, l1, j, k, v10);
                a.st(b, 11, l1, j, k, v11);
                a.st(b, 12, l1, j, k, v12);
                a.st(b, 13, l1, j, k, v13);
                a.st(b, 14, l1, j, k, v14);
            } else if (c.front == 1) {  // no-slip, :108-124
                const R v1 = a.ld(1, l, j, k), v2 = a.ld(2, l, j, k), v3 = a.ld(3, l, j, k), v4 = a.ld(4, l, j, k),
                        v5 = a.ld(5, l, j, k);
                a.st(b, 12, l1, j - 1, k, v1);
                a.st(b, 13, l1, j, k - 1, v2);
                a.st(b, 10, l1, j + 1, k, v3);
                a.st(b, 11, l1, j, k + 1, v4);
                a.st(b, 14, l1, j, k, v5);
            } else {
                R v[5];
                a.outflow(j, k, v);
                for (int q = 0; q < 5; ++q) a.st(b, 10 + q, l1, j, k, v[q]);
            }
            return;
        }
        case kHaloFrontFix: {  // outflow border, :172-203: copies of the edge rows
            constexpr int b = kHaloFrontFix;
            const int t = ia;
            R lo[5], hi[5];
            if (ib == 0 && t <= m) {
                a.outflow(t, 1, lo);
                a.outflow(t, n, hi);
                for (int q = 0; q < 5; ++q) {
                    a.st(b, 10 + q, l1, t, 0, lo[q]);
                    a.st(b, 10 + q, l1, t, n1, hi[q]);
                }
            }
            if (ib == 1 && t <= n) {
                a.outflow(1, t, lo);
                a.outflow(m, t, hi);
                for (int q = 0; q < 5; ++q) {
                    a.st(b, 10 + q, l1, 0, t, lo[q]);
                    a.st(b, 10 + q, l1, m1, t, hi[q]);
                }
            }
            return;
        }
        case kHaloRear: {  // x = 0
            constexpr int b = kHaloRear;
            const int j = ia, k = ib;
            if (c.rear == 0) {  // periodic, :210-238 (SERIAL corner line :223)
                if (j == 0) { a.st(b, 1, 0, m1, k, a.ld(1, l, 1, k)); return; }
                const R v1 = a.ld(1, l, j, k), v2 = a.ld(2, l, j, k), v3 = a.ld(3, l, j, k), v4 = a.ld(4, l, j, k),
                        v5 = a.ld(5, l, j, k);
                a.st(b, 1, 0, j, k, v1);
                a.st(b, 2, 0, j, k, v2);
                a.st(b, 3, 0, j, k, v3);
                a.st(b, 4, 0, j, k, v4);
                a.st(b, 5, 0, j, k, v5);
            } else if (c.rear == 1) {  // no-slip, :241-257
                const R v10 = a.ld(10, 1, j, k), v11 = a.ld(11, 1, j, k), v12 = a.ld(12, 1, j, k),
                        v13 = a.ld(13, 1, j, k), v14 = a.ld(14, 1, j, k);
                a.st(b, 3, 0, j - 1, k, v10);
                a.st(b, 4, 0, j, k - 1, v11);
                a.st(b, 1, 0, j + 1, k, v12);
                a.st(b, 2, 0, j, k + 1, v13);
                a.st(b, 5, 0, j, k, v14);
            } else {
                R v[5];
                a.inflow(v);
                for (int q = 0; q < 5; ++q) a.st(b, 1 + q, 0, j, k, v[q]);
            }
            return;
        }
        case kHaloUp: {  // z = n+1
            constexpr int b = kHaloUp;
            const int i = ia, j = ib;
            if (c.up == 0) {  // periodic, :385-409
                const R v2 = a.ld(2, i, j, 1), v9 = a.ld(9, i, j, 1), v11 = a.ld(11, i, j, 1), v15 = a.ld(15, i, j, 1),
                        v16 = a.ld(16, i, j, 1);
                a.st(b, 2, i, j, n1, v2);
                a.st(b, 9, i, j, n1, v9);
                a.st(b, 11, i, j, n1, v11);
                a.st(b, 15, i, j, n1, v15);
                a.st(b, 16, i, j, n1, v16);
                return;
            }
            if (c.up == 3 && !(halo_in(i, 1, l) && halo_in(j, 1, m))) {  // free-slip rim, :450-468
                // (9, i, 0, n+1) and (16, i, m+1, n+1): left to the item that replaces what they
                // copy (periodic left/right face), or to the edge fix that overwrites them
                const bool I = halo_in(i, 1, l);
                const bool no9 = I && j == 0 && (c.left == 0 || c.left == 3);
                const bool no16 = I && j == m1 && (c.right == 0 || c.right == 3);
                const R v6 = halo_rim(a, 6, i, j), v13 = halo_rim(a, 13, i, j), v4 = halo_rim(a, 4, i, j);
                const R v18 = no16 ? R() : halo_rim(a, 18, i, j), v7 = no9 ? R() : halo_rim(a, 7, i, j);
                a.st(b, 15, i, j, n1, v6);
                a.st(b, 11, i, j, n1, v13);
                if (!no16) a.st(b, 16, i, j, n1, v18);
                a.st(b, 2, i, j, n1, v4);
                if (!no9) a.st(b, 9, i, j, n1, v7);
                return;
            }
            const R v6 = a.ld(6, i, j, n), v13 = a.ld(13, i, j, n), v18 = a.ld(18, i, j, n), v4 = a.ld(4, i, j, n),
                    v7 = a.ld(7, i, j, n);
            if (c.up == 3) {
                a.st(b, 15, i, j, n1, v6);
                a.st(b, 11, i, j, n1, v13);
                a.st(b, 16, i, j, n1, v18);
                a.st(b, 2, i, j, n1, v4);
                a.st(b, 9, i, j, n1, v7);
            } else {  // no-slip :412-428, lid :431-447
                a.st(b, 15, i, j, n1, v6);
                a.st(b, 2, i - 1, j, n1, c.up == 2 ? a.lid(v13, 1) : v13);
                a.st(b, 9, i, j - 1, n1, v18);
                a.st(b, 11, i + 1, j, n1, c.up == 2 ? a.lid(v4, -1) : v4);
                a.st(b, 16, i, j + 1, n1, v7);
            }
            return;
        }
        case kHaloDown: {  // z = 0
            constexpr int b = kHaloDown;
            const int i = ia, j = ib;
            if (c.down == 0) {  // periodic, :472-496
                const R v4 = a.ld(4, i, j, n), v6 = a.ld(6, i, j, n), v7 = a.ld(7, i, j, n), v13 = a.ld(13, i, j, n),
                        v18 = a.ld(18, i, j, n);
                a.st(b, 4, i, j, 0, v4);
                a.st(b, 6, i, j, 0, v6);
                a.st(b, 7, i, j, 0, v7);
                a.st(b, 13, i, j, 0, v13);
                a.st(b, 18, i, j, 0, v18);
                return;
            }
            const R v15 = a.ld(15, i, j, 1), v11 = a.ld(11, i, j, 1), v16 = a.ld(16, i, j, 1), v2 = a.ld(2, i, j, 1),
                    v9 = a.ld(9, i, j, 1);
            if (c.down == 1) {  // no-slip, :499-515
                a.st(b, 6, i, j, 0, v15);
                a.st(b, 4, i - 1, j, 0, v11);
                a.st(b, 7, i, j - 1, 0, v16);
                a.st(b, 13, i + 1, j, 0, v2);
                a.st(b, 18, i, j + 1, 0, v9);
            } else {  // free-slip, :518-530
                a.st(b, 6, i, j, 0, v15);
                a.st(b, 13, i, j, 0, v11);
                a.st(b, 18, i, j, 0, v16);
                a.st(b, 4, i, j, 0, v2);
                a.st(b, 7, i, j, 0, v9);
            }
            return;
        }
        case kHaloLeft: {  // y = 0
            constexpr int b = kHaloLeft;
            const int i = ia, k = ib;
            if (c.left == 0) {  // periodic, :535-560 (corner line :547)
                if (i == 0) { a.st(b, 3, 0, 0, k, a.ld(3, l, m, k)); return; }
                const bool pass = k == n && c.up == 3;  // the up block's copy of the value replaced here
                const R was = pass ? a.old(7, i, 0, n) : R();
                const R v3 = a.ld(3, i, m, k), v7 = a.ld(7, i, m, k), v8 = a.ld(8, i, m, k), v9 = a.ld(9, i, m, k),
                        v12 = a.ld(12, i, m, k);
                if (pass) a.st(kHaloUp, 9, i, 0, n1, was);
                a.st(b, 3, i, 0, k, v3);
                a.st(b, 7, i, 0, k, v7);
                a.st(b, 8, i, 0, k, v8);
                a.st(b, 9, i, 0, k, v9);
                a.st(b, 12, i, 0, k, v12);
                return;
            }
            const R v17 = a.ld(17, i, 1, k), v1 = a.ld(1, i, 1, k), v10 = a.ld(10, i, 1, k), v16 = a.ld(16, i, 1, k),
                    v18 = a.ld(18, i, 1, k);
            if (c.left == 1) {  // no-slip, :563-579
                a.st(b, 8, i, 0, k, v17);
                a.st(b, 12, i + 1, 0, k, v1);
                a.st(b, 3, i - 1, 0, k, v10);
                a.st(b, 7, i, 0, k - 1, v16);
                a.st(b, 9, i, 0, k + 1, v18);
            } else {  // free-slip, :582-594
                a.st(b, 8, i, 0, k, v17);
                a.st(b, 3, i, 0, k, v1);
                a.st(b, 12, i, 0, k, v10);
                a.st(b, 9, i, 0, k, v16);
                a.st(b, 7, i, 0, k, v18);
            }
            return;
        }
        case kHaloRight: {  // y = m+1
            constexpr int b = kHaloRight;
            const int i = ia, k = ib;
            if (c.right == 0) {  // periodic, :600-625 (corner line :612)
                if (i == 0) { a.st(b, 10, l1, m1, k, a.ld(10, 1, 1, k)); return; }
                const bool pass = k == n && c.up == 3;
                const R was = pass ? a.old(18, i, m1, n) : R();
                const R v1 = a.ld(1, i, 1, k), v10 = a.ld(10, i, 1, k), v16 = a.ld(16, i, 1, k), v17 = a.ld(17, i, 1, k),
                        v18 = a.ld(18, i, 1, k);
                if (pass) a.st(kHaloUp, 16, i, m1, n1, was);
                a.st(b, 1, i, m1, k, v1);
                a.st(b, 10, i, m1, k, v10);
                a.st(b, 16, i, m1, k, v16);
                a.st(b, 17, i, m1, k, v17);
                a.st(b, 18, i, m1, k, v18);
                return;
            }
            const R v3 = a.ld(3, i, m, k), v7 = a.ld(7, i, m, k), v8 = a.ld(8, i, m, k), v9 = a.ld(9, i, m, k),
                    v12 = a.ld(12, i, m, k);
            if (c.right == 1) {  // no-slip, :628-644
                a.st(b, 10, i + 1, m1, k, v3);
                a.st(b, 16, i, m1, k + 1, v7);
                a.st(b, 17, i, m1, k, v8);
                a.st(b, 18, i, m1, k - 1, v9);
                a.st(b, 1, i - 1, m1, k, v12);
            } else {  // free-slip, :647-659
                a.st(b, 1, i, m1, k, v3);
                a.st(b, 18, i, m1, k, v7);
                a.st(b, 17, i, m1, k, v8);
                a.st(b, 16, i, m1, k, v9);
                a.st(b, 10, i, m1, k, v12);
            }
            return;
        }
        default: {  // free-slip edge fixes, :663-690
            constexpr int b = kHaloEdgeFix;
            const int i = ia;
            const R v1 = (c.fixes & 1) ? a.ld(18, i, 1, n) : R();
            const R v2 = (c.fixes & 2) ? a.ld(7, i, m, n) : R();
            const R v3 = (c.fixes & 4) ? a.ld(9, i, m, 1) : R();
            const R v4 = (c.fixes & 8) ? a.ld(16, i, 1, 1) : R();
            if (c.fixes & 1) a.st(b, 9, i, 0, n1, v1);
            if (c.fixes & 2) a.st(b, 16, i, m1, n1, v2);
            if (c.fixes & 4) a.st(b, 18, i, m1, 0, v3);
            if (c.fixes & 8) a.st(b, 7, i, 0, 0, v4);
        }
    }
}

}  // namespace eup
