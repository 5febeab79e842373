// The halo items of halo.h in the form k_halo runs: per face five strided copies (outflow
// equilibria, constants), recorded from one item in the middle of the face, and a table of
// what lands on the twelve edge lines, recorded from every item that can reach them.  Host code.
#include "halo.h"
#include "internal.h"

namespace eup {

namespace {

// A value as the place it comes from.
struct Sym {
    enum Kind : int { kCopy, kOld, kOutflow, kConst } kind = kCopy;
    int q = 0, i = 0, j = 0, k = 0;  // population 1..18 and node; kOutflow: row j, k; kOutflow/kConst: q = 0..4
    int lid = 0;
};

struct Store_ {
    int q, i, j, k;
    Sym v;
};

struct Recorder {
    using R = Sym;
    HaloConf c;
    int block;  // whose stores are kept (the up block's store made by a periodic left or right item goes with that face)
    bool edges_only;
    std::vector<Store_>* out;
    static Sym at(Sym::Kind kind, int q, int i, int j, int k) {
        Sym s;
        s.kind = kind; s.q = q; s.i = i; s.j = j; s.k = k;
        return s;
    }
    Sym ld(int q, int i, int j, int k) const { return at(Sym::kCopy, q, i, j, k); }
    Sym old(int q, int i, int j, int k) const { return at(Sym::kOld, q, i, j, k); }
    void outflow(int j, int k, Sym (&v)[5]) const {
        for (int t = 0; t < 5; ++t) v[t] = at(Sym::kOutflow, t, c.l, j, k);
    }
    void inflow(Sym (&v)[5]) const {
        for (int t = 0; t < 5; ++t) v[t] = at(Sym::kConst, t, 0, 0, 0);
    }
    Sym lid(Sym v, int s) const {
        v.lid = s;
        return v;
    }
    void st(int b, int q, int i, int j, int k, const Sym& v) const {
        if (b != block) return;
        if (edges_only) {
            const int outside = !halo_in(i, 1, c.l) + !halo_in(j, 1, c.m) + !halo_in(k, 1, c.n);
            if (outside < 2 || halo_overwritten(c, b, q, i, j, k)) return;
        }
        out->push_back({q, i, j, k, v});
    }
};

}  // namespace

HaloEdges build_halo_edges(const Geo& g, const int bc[6]) {
    HaloEdges out;
    std::vector<Store_> st;
    Recorder rec{HaloConf(g.l, g.m, g.n, bc), 0, true, &st};
    const HaloConf& c = rec.c;
    for (int b = 0; b < kHaloBlocks; ++b) {
        rec.block = b;
        out.first[b] = (int64_t)out.e.size();
        const HaloRange r = halo_range(c, b);
        const bool all = b == kHaloFrontFix || b == kHaloEdgeFix;
        st.clear();
        for (int y = 0; y < r.nb; ++y) {
            // an item reaches an edge line only from the outermost rows and columns of its range
            const bool row = all || y == 0 || y == r.nb - 1;
            for (int x = 0; x < r.na; ++x) {
                if (!row && x > 0) x = r.na - 1;
                halo_item(rec, b, r.a0 + x, r.b0 + y);
            }
        }
        for (const Store_& s : st) {
            HaloEdge e;
            e.dst = (int64_t)(s.q - 1) * g.G + g.gidx(s.i, s.j, s.k);
            e.q = s.v.q - 1;
            switch (s.v.kind) {
                case Sym::kCopy:
                    e.kind = s.v.lid == 0 ? kEdgeCopy : (s.v.lid > 0 ? kEdgeCopyPlus : kEdgeCopyMinus);
                    e.src = g.lin(s.v.i, s.v.j, s.v.k);
                    break;
                case Sym::kOld:
                    e.kind = kEdgeOld;
                    e.src = (int64_t)(s.v.q - 1) * g.G + g.gidx(s.v.i, s.v.j, s.v.k);
                    break;
                case Sym::kOutflow:
                    e.kind = kEdgeOutflow;
                    e.q = s.v.q;
                    e.src = (int64_t)(s.v.j - 1) + (int64_t)(s.v.k - 1) * g.m;
                    break;
                default:
                    e.kind = kEdgeConst;
                    e.q = s.v.q;
                    e.src = 0;
            }
            out.e.push_back(e);
        }
    }
    out.first[kHaloBlocks] = (int64_t)out.e.size();
    return out;
}

HaloFace record_halo_face(const Geo& g, const int bc[6], int b) {
    HaloFace f{};
    f.kind = kFaceNone;
    std::vector<Store_> st;
    const Recorder rec{HaloConf(g.l, g.m, g.n, bc), b, false, &st};
    const HaloConf& c = rec.c;
    if (b == kHaloFrontFix || b == kHaloEdgeFix || halo_range(c, b).size() == 0) return f;
    halo_item(rec, b, 1, 1);  // tangential coordinates (1, 1)
    const bool x = b == kHaloFront || b == kHaloRear, z = b == kHaloUp || b == kHaloDown;
    f.na = x ? g.m : g.l;
    f.nb = z ? g.m : g.n;
    f.dst_b = x ? g.m + 2 : g.l;  // halo row stride (lbm_common.cuh, Geo::gidx)
    f.src_b = x ? g.m : (z ? (int64_t)g.l : g.lm);
    f.lin_a = x ? g.l : 1;
    f.lin_b = z ? (int64_t)g.l : g.lm;
    int t = 0;
    for (const Store_& s : st) {
        if (t == 5) break;
        const int da = (x ? s.j : s.i) - 1, db = (z ? s.j : s.k) - 1;
        f.da[t] = da;
        f.db[t] = db;
        f.q[t] = s.q - 1;
        // the slot of tangential coordinates (1, 1) of this face, moved by (da, db)
        const int hi = b == kHaloFront ? g.l + 1 : (b == kHaloRear ? 0 : 1);
        const int hj = b == kHaloRight ? g.m + 1 : (b == kHaloLeft ? 0 : 1);
        const int hk = b == kHaloUp ? g.n + 1 : (b == kHaloDown ? 0 : 1);
        f.dst[t] = (int64_t)(s.q - 1) * g.G + g.gidx(hi, hj, hk) + da + db * f.dst_b;
        f.lid[t] = s.v.lid;
        if (s.v.kind == Sym::kOutflow) {
            f.kind = kFaceOutflow;
        } else if (s.v.kind == Sym::kConst) {
            f.kind = kFaceConst;
            f.src_q[t] = s.v.q;
        } else {
            f.kind = x ? kFaceCopyX : kFaceCopy;
            f.src_q[t] = s.v.q - 1;
            f.lin[t] = g.lin(s.v.i, s.v.j, s.v.k);
            f.src[t] = x ? xface_idx(g, s.v.i == 1 ? 0 : 1, s.v.q - 1, 1, 1) : g.lin(s.v.i, s.v.j, s.v.k);
        }
        ++t;
    }
    // the up block's copy of the value that a periodic left or right face replaces on its row k = n
    f.pass = -1;
    if (c.up == 3 && ((b == kHaloLeft && c.left == 0) || (b == kHaloRight && c.right == 0))) {
        const int q = b == kHaloLeft ? 7 : 18, to = b == kHaloLeft ? 9 : 16, j = b == kHaloLeft ? 0 : g.m + 1;
        if (!halo_overwritten(c, kHaloUp, to, 1, j, g.n + 1)) {
            for (int u = 0; u < 5; ++u)
                if (f.q[u] == q - 1) f.pass = u;
            f.pass_dst = (int64_t)(to - 1) * g.G + g.gidx(1, j, g.n + 1);
        }
    }
    return f;
}

}  // namespace eup
