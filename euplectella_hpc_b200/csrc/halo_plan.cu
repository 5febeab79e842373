// The halo items of halo.h in the form k_halo runs: per face five strided copies (outflow
// equilibria, constants), recorded from one item in the middle of the face, and a table of
// what lands on the twelve edge lines, recorded on the host from the items near the ends of the
// lines and one between, which repeats along the line, and written out on the device.
#include <algorithm>
#include <utility>

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

namespace {

HaloEdge edge_of(const Geo& g, const Store_& s) {
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
    return e;
}

// The coordinates lo .. lo+count-1 as runs (first, length): one by one within four of a place where
// an item's conditions change, else as long as possible.  An item reads and writes within one node of
// its own coordinates, so the items of a run differ by a shift alone.
std::vector<std::pair<int, int>> runs_along(int lo, int count, std::vector<int> changes, bool one_by_one) {
    changes.push_back(lo);
    changes.push_back(lo + count - 1);
    std::vector<std::pair<int, int>> out;
    for (int64_t c = lo; c < (int64_t)lo + count;) {
        int64_t next = (int64_t)lo + count;
        bool near = one_by_one;
        for (const int64_t p : changes) {
            near |= c >= p - 4 && c <= p + 4;
            if (p - 4 > c) next = std::min(next, p - 4);
        }
        const int64_t length = near ? 1 : next - c;
        out.push_back({(int)c, (int)length});
        c += length;
    }
    return out;
}

// Thread t writes edge t: it lies in the group of the last run that starts at or before it.
__global__ void k_fill_edges(const HaloEdgeRun* runs, int nruns, int64_t total, HaloEdge* out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    int lo = 0, hi = nruns;  // runs[lo].at <= t, and runs[hi].at > t or hi = nruns
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (runs[mid].at <= t) lo = mid;
        else hi = mid;
    }
    const int64_t u = t - runs[lo].at, along = u / runs[lo].stores;
    const HaloEdgeRun r = runs[lo - (runs[lo].stores - 1) + (int)(u - along * runs[lo].stores)];
    HaloEdge e = r.e;
    e.dst += along * r.dst_step;
    e.src += along * r.src_step;
    out[t] = e;
}

}  // namespace

HaloEdges build_halo_edges(const Geo& g, const int bc[6], bool one_by_one) {
    HaloEdges out;
    std::vector<Store_> st, one, next;
    Recorder rec{HaloConf(g.l, g.m, g.n, bc), 0, true, &st};
    const HaloConf& c = rec.c;
    int64_t at = 0;
    // the stores of items (ia, ib) and, if it is another, (ia2, ib), and of the `length - 1` pairs
    // behind them along a or b
    auto record = [&](int b, int ia, int ia2, int ib, int length, bool along_a) {
        auto items = [&](int d, std::vector<Store_>& to) {
            st.clear();
            halo_item(rec, b, ia + (along_a ? d : 0), ib + (along_a ? 0 : d));
            if (ia2 != ia) halo_item(rec, b, ia2, ib + (along_a ? 0 : d));
            to = st;
        };
        items(0, one);
        if (length > 1) items(1, next);
        for (size_t t = 0; t < one.size(); ++t) {
            HaloEdgeRun r{edge_of(g, one[t]), 0, 0, at, (int32_t)one.size(), 0};
            if (length > 1) {
                const HaloEdge e = edge_of(g, next[t]);
                r.dst_step = e.dst - r.e.dst;
                r.src_step = e.src - r.e.src;
            }
            out.runs.push_back(r);
        }
        at += (int64_t)length * (int64_t)one.size();
    };
    for (int b = 0; b < kHaloBlocks; ++b) {
        rec.block = b;
        out.first[b] = at;
        const HaloRange r = halo_range(c, b);
        if (r.size() == 0) continue;
        // an item reaches an edge line only from the outermost rows and columns of its range
        const bool all = b == kHaloFrontFix || b == kHaloEdgeFix;
        const auto xs = runs_along(r.a0, r.na, b == kHaloFrontFix ? std::vector<int>{c.m, c.n} : std::vector<int>{},
                                   one_by_one);
        for (const auto& y : runs_along(r.b0, r.nb, {}, one_by_one)) {
            if (all || y.first == r.b0 || y.first == r.b0 + r.nb - 1) {
                for (const auto& x : xs) record(b, x.first, x.first, y.first, x.second, true);
            } else {
                record(b, r.a0, r.a0 + r.na - 1, y.first, y.second, false);
            }
        }
    }
    out.first[kHaloBlocks] = at;
    return out;
}

cudaError_t put_halo_edges(const HaloEdges& edges, HaloEdgesDevice* out, cudaStream_t st) {
    const int64_t total = edges.first[kHaloBlocks];
    HaloEdge* table = nullptr;
    cudaError_t e = cudaMalloc(&table, sizeof(HaloEdge) * (total + 1));
    if (e != cudaSuccess) return e;
    out->e = table;
    for (int b = 0; b <= kHaloBlocks; ++b) out->first[b] = edges.first[b];
    if (total == 0) return cudaSuccess;
    HaloEdgeRun* runs = nullptr;
    const size_t bytes = sizeof(HaloEdgeRun) * edges.runs.size();
    if ((e = cudaMalloc(&runs, bytes)) != cudaSuccess) return e;
    e = cudaMemcpyAsync(runs, edges.runs.data(), bytes, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) {
        k_fill_edges<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(runs, (int)edges.runs.size(), total, table);
        e = cudaGetLastError();
    }
    const cudaError_t es = cudaStreamSynchronize(st);
    cudaFree(runs);
    return e == cudaSuccess ? es : e;
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

// The edge table on the host, for tests: `out` takes (dst, src, q, kind, block) of each store, at most
// `cap` of them; the items recorded one by one, or as runs.  Returns how many there are.
extern "C" int64_t eup_internal_halo_edges(int l, int m, int n, const int* bc, int one_by_one, int64_t* out, int64_t cap) {
    using namespace eup;
    Geo g{};
    g.init(l, m, n);
    const HaloEdges e = build_halo_edges(g, bc, one_by_one != 0);
    const int64_t total = e.first[kHaloBlocks];
    for (size_t r = 0; r < e.runs.size(); r += e.runs[r].stores) {
        const int stores = e.runs[r].stores;
        const int64_t at = e.runs[r].at, end = r + stores < e.runs.size() ? e.runs[r + stores].at : total;
        int block = 0;
        while (at >= e.first[block + 1]) ++block;
        for (int64_t t = at; t < end && t < cap; ++t) {
            const HaloEdgeRun& run = e.runs[r + (t - at) % stores];
            int64_t* o = out + 5 * t;
            o[0] = run.e.dst + (t - at) / stores * run.dst_step;
            o[1] = run.e.src + (t - at) / stores * run.src_step;
            o[2] = run.e.q;
            o[3] = run.e.kind;
            o[4] = block;
        }
    }
    return total;
}
