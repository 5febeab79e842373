// The work items of csrc/halo.h on a host array of haloed populations a[19][n+2][m+2][l+2],
// run in a seeded random order.
#include <algorithm>
#include <random>
#include <vector>

#include "halo.h"

namespace {
struct Items {
    using R = double;
    eup::HaloConf c;
    R u_inflow, force;
    double* a;
    double& at(int q, int i, int j, int k) const {
        return a[(((int64_t)(q - 1) * (c.n + 2) + k) * (c.m + 2) + j) * (c.l + 2) + i];
    }
    R ld(int q, int i, int j, int k) const { return at(q, i, j, k); }
    R old(int q, int i, int j, int k) const { return at(q, i, j, k); }
    void outflow(int j, int k, R (&v)[5]) const {
        R x[18];
        for (int q = 1; q <= 18; ++q) x[q - 1] = ld(q, c.l, j, k);
        eup::halo_outflow(x, v);
    }
    void inflow(R (&v)[5]) const { eup::halo_inflow(u_inflow, v); }
    R lid(R v, int s) const { return s > 0 ? v + force : v - force; }
    void st(int b, int q, int i, int j, int k, R v) const {
        if (!eup::halo_overwritten(c, b, q, i, j, k)) at(q, i, j, k) = v;
    }
};
struct Item { int b, ia, ib; };
}  // namespace

extern "C" void halo_items_run(const int* bc, int l, int m, int n, double u_inflow, double force, unsigned seed,
                               double* a) {
    Items it{eup::HaloConf(l, m, n, bc), u_inflow, force, a};
    std::vector<Item> items;
    for (int b = 0; b < eup::kHaloBlocks; ++b) {
        const eup::HaloRange r = eup::halo_range(it.c, b);
        for (int y = 0; y < r.nb; ++y)
            for (int x = 0; x < r.na; ++x) items.push_back({b, r.a0 + x, r.b0 + y});
    }
    std::shuffle(items.begin(), items.end(), std::mt19937(seed));
    for (const Item& t : items) eup::halo_item(it, t.b, t.ia, t.ib);
}
