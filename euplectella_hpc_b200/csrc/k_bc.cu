// Boundary side of the time step: halo planes (CODE/SRC/bcond.bc.F90) and
// bounce-back on solid voxels with the momentum-exchange force
// (CODE/SRC/bcond.obs.F90), O(surface) and O(solid surface) work; the diagnostics,
// some of a few nodes (CODE/SRC/probe_global.F90, lines, control volume), some of all of
// them (the FP64 monitor of CODE/SRC/diagno.F90, region sums, plane means); and the
// host-layout scatter/gather of upload and download, which move the whole state.
#include "init_eq.h"
#include <algorithm>

#include "halo.h"
#include "internal.h"
#include "row_walk.h"

namespace eup {

namespace {

constexpr int kTpb = 256;

// ---- bounce-back + momentum exchange ---------------------------------------------------
//
// For each solid voxel x touching fluid or halo and each moving q, the
// reference sets a_q(x) = a_opp(q)(x + c_q) (CODE/SRC/bcond.obs.F90:56-73), so
// that the next pull returns to the fluid node x + c_q its own post-collision
// population.  Links whose neighbour is itself solid are skipped: their value
// is only ever pulled into solid voxels.  The same reads give the force: the
// population a_opp(q)(y) leaving fluid node y = x + c_q towards x transfers
// 2 c_opp(q) a_opp(q)(y) = -2 c_q a_opp(q)(y); across a periodic axis y is the
// wrapped node and its interior value is used.
//
// One thread per link.  Like the halo this is a short kernel bound by latency and instruction
// fetch, so a link is a few instructions with the population's pointers and weights in the
// parameter bank, the halo links have their source slots in the list, and the partial forces
// are added by the halo launch that follows instead of by the last block behind a fence and an
// atomic.  Bounce-back and force of a step (CUDA events, launch included), one thread per voxel
// with its 18 directions written out and the sum in the kernel / this: 14.4 / 7.0 us at 64x32x8,
// 16.6 / 8.7 us at 256x128x64, 18.7 / 14.9 us at 768x384x384 FP32.
template <typename S, typename R>
struct BounceArgs {
    Lat<S, R> L;
    Geo g;
    LinksDevice links;
    const S* from[18];  // population opp(q), moved so that the solid voxel's index reads x + c_q
    R w[18];
    double c2[18][3];   // -2 c_q
    double* partials;
    int bounce;         // store, or the force alone
    int finish;         // the last block adds the partial sums (series, cap, d_itime)
    unsigned int* counter;
    ForceSum sum;
};

// A force is a small difference of large sums (the pressure on either side of a body), and the
// links come population by population, so that a plain sum adds up one side before it meets the
// other.  FP32 values do so exactly in FP64 (populations of 2^-6 and more: below 2^24).  FP64
// values lost 2e-14 at 256x128x64, where voxel by voxel 1e-17 to 8e-15 are lost, so each is split at
// 2^-24: the multiples add up exactly below 2^29, the rest, at most 2^-25 each, loses 2^-20 of what
// the plain sum lost, and the two meet when the sum is complete.  (Values beyond 2^27 or below
// 2^-25 add up as in a plain sum.)
template <typename R>
struct Force {
    static constexpr int kSums = sizeof(R) == 8 ? 6 : 3;  // three sums, or three of multiples and three of the rest
    static constexpr int kPad = sizeof(R) == 8 ? 8 : 4;
    double v[kPad] = {};
    __device__ __forceinline__ void add(const double (&c2)[3], double x) {
        if constexpr (sizeof(R) == 8) {
            const double grid = 402653184.0;  // 1.5 2^28: its last digit is worth 2^-24
            const double hi = (x + grid) - grid, lo = x - hi;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                v[c] += c2[c] * hi;
                v[3 + c] += c2[c] * lo;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) v[c] += c2[c] * x;
        }
    }
    // The sums over the block, sum c in the lanes 32 / kPad * c of the first warp and the ones
    // behind it; kTpb threads, fixed order.  Lanes that are 16, 8 and (eight sums) 4 apart trade
    // halves of what they still hold: six or nine exchanges, where fifteen or thirty sum one by one.
    __device__ __forceinline__ double block_sum() {
        static_assert(kTpb / 32 == 8, "eight warps' sums");
        constexpr int kLanes = 32 / kPad;  // to a sum
        __shared__ double sh[kPad][kTpb / 32];
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int h = kPad / 2; h > 0; h >>= 1) {
            const bool up = lane & (kLanes * h);
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const double give = up ? v[i] : v[i + h], keep = up ? v[i + h] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, give, kLanes * h);
            }
        }
        double s = v[0];  // sum lane / kLanes of the lanes that many apart
#pragma unroll
        for (int o = kLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        __syncthreads();
        if (lane % kLanes == 0) sh[lane / kLanes][threadIdx.x >> 5] = s;
        __syncthreads();
        if (threadIdx.x < 32) {
            s = sh[lane / kLanes][lane % kLanes];
            if constexpr (kLanes == 4) s += sh[lane / kLanes][4 + lane % kLanes];
#pragma unroll
            for (int o = kLanes / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        }
        return s;
    }
    // Which sum this thread has to store (-1: none).
    static __device__ __forceinline__ int mine() {
        constexpr int kLanes = 32 / kPad;
        return threadIdx.x < kLanes * kSums && threadIdx.x % kLanes == 0 ? (int)threadIdx.x / kLanes : -1;
    }
};

// One block: the partial sums of the force in a fixed order into the force history.
template <typename R>
__device__ __forceinline__ void sum_partials(const ForceSum& a, bool advance) {
    constexpr int W = Force<R>::kSums;
    const int64_t t = *a.d_itime;
    Force<R> f;
    for (int b = threadIdx.x; b < a.blocks; b += kTpb)
#pragma unroll
        for (int c = 0; c < W; ++c) f.v[c] += __ldcg(a.partials + W * b + c);
    double s = f.block_sum();  // every thread has read d_itime before thread 0 writes it
    if (threadIdx.x < 32) {
        if constexpr (W == 6) s += __shfl_down_sync(0xffffffffu, s, 12);  // the rest of the same component
        const int c = Force<R>::mine();
        if (c >= 0 && c < 3) {
            a.series[3 * (t % a.cap) + c] = s;
            if (a.host) a.host[c] = s;
        }
    }
    if (advance && threadIdx.x == 0) *a.d_itime = t + 1;
}

// Where the links are many the loads in flight count: with 20 % of the voxels solid at random,
// 256x128x64 FP16, a step takes 81.9 us with 32 registers (16-bit storage spills one of them once) and
// 86.1 with 36; FP64's six sums take 40, and 214 us for 210 with three plain sums.
template <typename S, typename R>
__global__ void __launch_bounds__(kTpb, sizeof(R) == 8 ? 6 : 8) k_bounce(const __grid_constant__ BounceArgs<S, R> p) {
    chain_open();
    Force<R> f;
    const int64_t total = p.links.nfluid + p.links.nhalo;
    int64_t t = (int64_t)blockIdx.x * kTpb + threadIdx.x;
    FluidLink k = {};  // of this pass, fetched during the one before, or during the wait
    if (t < p.links.nfluid) k = p.links.fluid[t];
    chain_wait();
    for (; t < total; t += (int64_t)gridDim.x * kTpb) {
        int32_t lin;
        uint32_t e;
        S raw;
        R val, push;  // the value stored, and the one that pushes the solid
        bool counts = true;
        if (t < p.links.nfluid) {
            lin = k.lin;
            e = k.q;
            raw = p.from[e & kLinkQ][lin];
            if constexpr (DevStore<S>::value) val = p.w[e & kLinkQ] + DevStore<S>::to_f(raw) * p.L.inv_scale;
            else val = raw;
            push = val;
            const int64_t next = t + (int64_t)gridDim.x * kTpb;
            if (next < p.links.nfluid) k = p.links.fluid[next];
        } else {
            const HaloLink k = p.links.halo[t - p.links.nfluid];
            lin = k.lin;
            e = k.q;
            const int q = e & kLinkQ;
            raw = Store<S, R>::store(p.L.ghost[k.ghost], q, p.L.scale);
            val = Store<S, R>::load(raw, q, p.L.inv_scale);
            counts = k.wrap >= 0;
            push = R(0);
            if (counts) push = Store<S, R>::load(p.L.pop[opp_of(q)][k.wrap], q, p.L.inv_scale);
        }
        const int q = e & kLinkQ;
        if (p.bounce) {
            p.L.pop[q][lin] = raw;
            if (e > kLinkQ) {  // a column the x-face copy holds
                R* x = p.L.xface + (p.g.xr + xface_slot(q) * p.g.mn + lin / p.g.l);
                if (e & kLinkXFirst) x[0] = val;
                if (e & kLinkXLast) x[p.g.xs] = val;
            }
        }
        if (counts) f.add(p.c2[q], (double)push);
    }
    const double s = f.block_sum();
    const int c = Force<R>::mine();
    if (c >= 0) p.partials[Force<R>::kSums * (int64_t)blockIdx.x + c] = s;
    if (!p.finish) return;
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(p.counter, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    sum_partials<R>(p.sum, false);
    if (threadIdx.x == 0) *p.counter = 0u;
}

// ---- halo planes ---------------------------------------------------------------------
//
// One launch for the halo of a step.  A segment is a run of thread blocks with one job: a face
// (one thread per node of the face, five populations each) or the edge stores of one of the
// reference's blocks (one thread per store).  The x faces read the compact x-face copy written
// by the stream-collide kernel (coalesced in j; a strided read of a column costs a sector per
// node), the others the lattice.  One more thread block adds the partial forces of the
// bounce-back launch.
//
// What bounds it on all but the largest lattices is the latency of a short kernel, and there
// instruction fetch: a launch starts with cold instruction caches, and ncu puts 80 % of the
// stalls of such kernels on missing instructions.  So the code is kept short and straight: the
// five copies of every face flag are one piece of code with strides from the plan, and whatever
// is irregular is in the table instead of in branches.  Halo planes of one step (CUDA events,
// launch included), as eight dependent launches / as one: 38 / 6.9 us at 64x32x8, 41 / 8.4 us at
// 256x128x64, 48 / 10.6 us at 384x192x192, 61 / 19.4 us at 768x384x384 FP32.  (One launch with
// the items' conditions written out: 12 and 23 us at the first two.)
constexpr int kHaloSegments = 2 * kHaloBlocks;  // six faces, eight blocks' edges, the force

template <typename S, typename R>
struct HaloSegment {
    int kind;  // kFace*, or kSegEdges
    unsigned count;
    unsigned na, nb;
    int64_t src_b, dst_b;
    const void* src[5];
    R* dst[5];
    R w[5];    // 16-bit storage: weight of the population; kFaceConst: the value
    R add[5];  // what the lid adds
    int da[5], db[5];
    int lid, pass;
    R* pass_dst;
    const HaloEdge* edges;
};
constexpr int kSegEdges = 100, kSegForce = 101;

template <typename S, typename R>
struct HaloPlan {
    Lat<S, R> L;
    Geo g;
    R force;
    R inflow[5];
    ForceSum sum;
    unsigned first[kHaloSegments + 1];  // first thread block of each segment
    HaloSegment<S, R> seg[kHaloSegments];
};

template <typename S, typename R>
__device__ __forceinline__ void outflow_row(const Lat<S, R>& L, const Geo& g, int64_t row, R (&v)[5]) {
    R x[18];
    const R* col = L.xface + (g.xs + g.xr + row);  // column x = l
#pragma unroll
    for (int q = 0; q < 18; ++q) x[q] = col[xface_slot(q) * g.mn];
    halo_outflow(x, v);
}

template <typename S, typename R>
__global__ void __launch_bounds__(kTpb) k_halo(const __grid_constant__ HaloPlan<S, R> p) {
    chain_open();
    int s = 0;
#pragma unroll
    for (int i = 1; i < kHaloSegments; ++i) s += blockIdx.x >= p.first[i];
    const HaloSegment<S, R>& f = p.seg[s];
    const unsigned t = (blockIdx.x - p.first[s]) * kTpb + threadIdx.x;
    if (t >= f.count) return;
    if (f.kind == kSegForce) {
        chain_wait();
        sum_partials<R>(p.sum, true);
        return;
    }
    R v[5];
    if (f.kind == kSegEdges) {
        const HaloEdge e = f.edges[t];
        chain_wait();
        if (e.kind <= kEdgeCopyMinus) {
            v[0] = Store<S, R>::load(p.L.pop[e.q][e.src], e.q, p.L.inv_scale);
            if (e.kind == kEdgeCopyPlus) v[0] = v[0] + p.force;
            if (e.kind == kEdgeCopyMinus) v[0] = v[0] - p.force;
        } else if (e.kind == kEdgeOld) {
            v[0] = p.L.ghost[e.src];
        } else if (e.kind == kEdgeConst) {
            v[0] = p.inflow[e.q];
        } else {
            outflow_row(p.L, p.g, e.src, v);
            v[0] = e.q == 0 ? v[0] : (e.q == 1 ? v[1] : (e.q == 2 ? v[2] : (e.q == 3 ? v[3] : v[4])));
        }
        p.L.ghost[e.dst] = v[0];
        return;
    }
    const unsigned b = t / f.na, a = t - b * f.na;
    const int64_t from = a + b * f.src_b, to = a + b * f.dst_b;
    chain_wait();
    if (f.kind == kFaceOutflow) {
        outflow_row(p.L, p.g, from, v);
    } else if (f.kind == kFaceConst) {
#pragma unroll
        for (int c = 0; c < 5; ++c) v[c] = f.w[c];
    } else if (!DevStore<S>::value || f.kind == kFaceCopyX) {
#pragma unroll
        for (int c = 0; c < 5; ++c) v[c] = static_cast<const R*>(f.src[c])[from];
    } else {
        if constexpr (DevStore<S>::value) {
            S raw[5];
#pragma unroll
            for (int c = 0; c < 5; ++c) raw[c] = static_cast<const S*>(f.src[c])[from];
#pragma unroll
            for (int c = 0; c < 5; ++c) v[c] = f.w[c] + DevStore<S>::to_f(raw[c]) * p.L.inv_scale;
        }
    }
    if (f.lid) {  // a moving lid: populations 2 and 11 alone
#pragma unroll
        for (int c = 0; c < 5; ++c)
            if (f.lid & (1 << c)) v[c] = v[c] + f.add[c];
    }
    if (f.pass >= 0 && b == f.nb - 1) f.pass_dst[a] = f.dst[f.pass][to];
#pragma unroll
    for (int c = 0; c < 5; ++c)
        if (a + f.da[c] < f.na && b + f.db[c] < f.nb) f.dst[c][to] = v[c];
}

// ---- FP64 monitor, CODE/SRC/diagno.F90:67-120 -------------------------------------------
//
// The diagnostics over all nodes walk the lattice by rows along x, a warp to a row (row_walk.h: or to
// a piece of a long one, or to several short ones): the loads of every population are
// coalesced, the row index is all the mask needs (32 nodes share a word), and no node pays for
// a division.  What bounds them is the read of the state, for 4- and 8-byte
// storage; for 16-bit storage the conversions to FP64 and the FP64 adds.  Monitor, a thread per
// node with three divisions / a warp per row: 298 / 232 us at 384x192x192 FP32, 2290 / 1560 at
// 768x384x384, 5.3 / 3.3..3.8 ms at 1024x512x512 FP16.

// Density and momentum of node lin in FP64.
template <typename S, typename R>
__device__ __forceinline__ void node_sums(const Lat<S, R>& L, int64_t lin, double& rho, double& xj, double& yj,
                                          double& zj, double& usq) {
    S raw[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) raw[q] = L.pop[q][lin];
    double a[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) a[q] = (double)Store<S, R>::load(raw[q], q, L.inv_scale);
    rho = 0.0;
#pragma unroll
    for (int q = 0; q < 19; ++q) rho += a[q];
    const double ri = 1.0 / rho;
    xj = (a[0] + a[1] + a[2] + a[3] + a[4] - a[9] - a[10] - a[11] - a[12] - a[13]) * ri;
    yj = (a[2] + a[6] + a[7] + a[8] + a[11] - a[0] - a[9] - a[15] - a[16] - a[17]) * ri;
    zj = (a[3] + a[5] + a[6] + a[12] + a[17] - a[1] - a[8] - a[10] - a[14] - a[15]) * ri;
    usq = xj * xj + yj * yj + zj * zj;
}

// f(row, x) for every node, x from 0, by the warps of the grid.
template <typename F>
__device__ __forceinline__ void walk_rows(const RowWalk& w, F&& f) {
    const int lane = threadIdx.x & 31, xl = lane & ((1 << w.lg) - 1);
    const int64_t step = (int64_t)gridDim.x * (kTpb / 32);
    for (int64_t u = (int64_t)blockIdx.x * (kTpb / 32) + (threadIdx.x >> 5); u < w.units; u += step) {
        const int64_t group = w.pieces == 1 ? u : u / w.pieces;
        const int first = (int)(u - group * w.pieces) * w.span, end = min(w.l - first, w.span);
        const int64_t r = (group << (5 - w.lg)) + (lane >> w.lg);
        if (r < w.rows)
            for (int x = xl; x < end; x += 32) f(r, first + x);
    }
}

template <typename S, typename R>
__global__ void __launch_bounds__(kTpb) k_monitor(Lat<S, R> L, RowWalk w, Mask mk, Reduce red, double* out) {
    double s[5] = {0, 0, 0, 0, 0};
    walk_rows(w, [&](int64_t r, int x) {
        if (mk.bits != nullptr && (mk.bits[r * mk.wpr + (x >> 5)] >> (x & 31)) & 1u) {
            s[0] += 1.0;
            return;
        }
        double rho, xj, yj, zj, usq;
        node_sums(L, r * w.l + x, rho, xj, yj, zj, usq);
        s[0] += rho; s[1] += xj; s[2] += yj; s[3] += zj; s[4] += usq;
    });
    block_reduce_store<5>(s, red, out);
}

// FP64 sums over the fluid nodes with region[lin] != 0 (the cavity of a shell,
// a probe box, ...): {count, sum rho, sum ux, sum uy, sum uz, sum u^2}, u = j/rho
// as CODE/SRC/diagno.F90:86-105 computes it.
template <typename S, typename R>
__global__ void __launch_bounds__(kTpb) k_region_sums(Lat<S, R> L, RowWalk w, Mask mk, const uint8_t* region,
                                                      Reduce red, double* out) {
    double s[6] = {0, 0, 0, 0, 0, 0};
    walk_rows(w, [&](int64_t r, int x) {
        if (!region[r * w.l + x]) return;
        if (mk.bits != nullptr && (mk.bits[r * mk.wpr + (x >> 5)] >> (x & 31)) & 1u) return;
        double rho, xj, yj, zj, usq;
        node_sums(L, r * w.l + x, rho, xj, yj, zj, usq);
        s[0] += 1.0; s[1] += rho; s[2] += xj; s[3] += yj; s[4] += zj; s[5] += usq;
    });
    block_reduce_store<6>(s, red, out);
}

// ---- reference-form diagnostics: line profiles, plane means, control-volume drag ----------

// Macroscopic values of one interior node in R, in the expression order of
// CODE/SRC/prof_i.F90:45-79 (div = true: momentum / den) and
// CODE/SRC/varm.F90:53-85 (div = false: momentum * (1 / den)).
template <typename S, typename R>
__device__ __forceinline__ void ref_macro(const Lat<S, R>& L, int64_t lin, bool div, R& den, R& u, R& w, R& v) {
    S raw[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) raw[q] = L.pop[q][lin];
    R f[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) f[q] = Store<S, R>::load(raw[q], q, L.inv_scale);
    const R r = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8] + f[9] + f[10] + f[11] + f[12] + f[13] +
                f[14] + f[15] + f[16] + f[17] + f[18];
    const R mx = f[0] + f[1] + f[2] + f[3] + f[4] - f[9] - f[10] - f[11] - f[12] - f[13];
    const R my = f[2] + f[6] + f[7] + f[8] + f[11] - f[0] - f[9] - f[15] - f[16] - f[17];
    const R mz = f[3] + f[5] + f[6] + f[12] + f[17] - f[1] - f[8] - f[10] - f[14] - f[15];
    den = r;
    if (div) {
        u = mx / r; w = my / r; v = mz / r;
    } else {
        const R ri = R(1) / r;
        u = mx * ri; w = my * ri; v = mz * ri;
    }
}

// prof_i / prof_j / prof_k (axis 0/1/2) at the two fixed coordinates c1, c2:
// out[4t + 0..3] = u, w (y), v (z), den of the t-th node, computed in R.
template <typename S, typename R>
__global__ void k_line(Lat<S, R> L, Geo g, int axis, int c1, int c2, double* out) {
    const int len = axis == 0 ? g.l : (axis == 1 ? g.m : g.n);
    const int t = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (t > len) return;
    const int i = axis == 0 ? t : c1, j = axis == 1 ? t : (axis == 0 ? c1 : c2), k = axis == 2 ? t : c2;
    R den, u, w, v;
    ref_macro(L, g.lin(i, j, k), true, den, u, w, v);
    out[4 * (t - 1) + 0] = (double)u;
    out[4 * (t - 1) + 1] = (double)w;
    out[4 * (t - 1) + 2] = (double)v;
    out[4 * (t - 1) + 3] = (double)den;
}

// Plane means (CODE/SRC/varm.F90:42-98 for axis z): FP64 sums of u, w, v (momentum times 1/den
// in R) and den over the nodes of each plane, divided by their number, in two passes (one for small
// planes, row_walk.h) with a fixed order.  A thread keeps its x and walks rows, so the state is read once and coalesced
// for every axis: rows of one plane for the planes normal to y and z, with a sum over the block
// at the end, and a share of all rows for those normal to x, where the thread's column is the
// plane.  (One block per plane, walked by 256 threads, a row's stride apart for the planes
// normal to x, took 1110 / 848 / 803 us for the planes normal to x / y / z at 384x192x192 FP32
// and 27.9 / 6.2 / 5.8 ms at 1024x512x512 FP16; now 200 us and 2.6..3.5 ms.  A warp per row
// with a sum over its lanes at the end of each: 226 us, 3.5 ms.)
template <typename S, typename R, bool COLUMN>
__global__ void __launch_bounds__(128) k_plane_sums(Lat<S, R> L, PlaneWalk w, double cnt, double* part) {
    const int xb = blockIdx.x % w.xblocks, ps = blockIdx.x / w.xblocks;  // ps = plane * shares + share
    const int share = ps % w.shares;
    const int64_t first = (int64_t)(ps / w.shares) * w.plane;
    const int x = xb * blockDim.x + threadIdx.x;
    double s[4] = {0, 0, 0, 0};
    auto column = [&](int64_t xi) {
        for (int t = share * blockDim.y + threadIdx.y; t < w.rows; t += w.shares * blockDim.y) {
            R den, u, v, z;
            ref_macro(L, (first + t * w.row) * w.l + xi, false, den, u, v, z);
            s[0] += (double)u; s[1] += (double)v; s[2] += (double)z; s[3] += (double)den;
        }
    };
    if constexpr (COLUMN) {
        if (x < w.l) column(x);
    } else {
        for (int64_t xi = x; xi < w.l; xi += (int64_t)w.xblocks * blockDim.x) column(xi);
    }
    if constexpr (COLUMN) {  // part[((share * blockDim.y + threadIdx.y) * 4 + c) * l + x]
        if (x < w.l)
#pragma unroll
            for (int c = 0; c < 4; ++c) part[((int64_t)(share * blockDim.y + threadIdx.y) * 4 + c) * w.l + x] = s[c];
    } else {
        __shared__ double sh[4][4];
        const int tid = threadIdx.y * blockDim.x + threadIdx.x;
#pragma unroll
        for (int c = 0; c < 4; ++c)
            for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_down_sync(0xffffffffu, s[c], o);
        if ((tid & 31) == 0)
#pragma unroll
            for (int c = 0; c < 4; ++c) sh[tid >> 5][c] = s[c];
        __syncthreads();
        if (tid < 4)  // cnt: nodes of the plane, where this block has all of them
            part[4 * (int64_t)blockIdx.x + tid] = ((sh[0][tid] + sh[1][tid]) + (sh[2][tid] + sh[3][tid])) / cnt;
    }
}

// out[4 p + c] = sum over t < n of in[p * plane + c * comp + t * stride], over cnt; one block of
// (4 components) x 64 threads per plane p.
__global__ void __launch_bounds__(256) k_add_planes(const double* in, int64_t plane, int64_t comp, int64_t stride,
                                                    int n, double cnt, double* out) {
    const int c = threadIdx.x & 3, u = threadIdx.x >> 2;
    double s = 0.0;
    for (int t = u; t < n; t += 64) s += in[(int64_t)blockIdx.x * plane + c * comp + t * stride];
    __shared__ double sh[64][4];
    sh[u][c] = s;
    __syncthreads();
    if (u == 0) {
        double a = 0.0;
        for (int t = 0; t < 64; ++t) a += sh[t][c];
        out[4 * blockIdx.x + c] = a / cnt;
    }
}

// Non-equilibrium stresses xx and xy of one node, CODE/SRC/flux_X.F90:162-240
// and CODE/SRC/flux_Y.F90, in R and the reference's expression order.
template <typename S, typename R>
__device__ __forceinline__ void ref_stress(const Lat<S, R>& L, int64_t lin, R omega, R& sxx, R& sxy) {
    R f[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) f[q] = Store<S, R>::load(L.pop[q][lin], q, L.inv_scale);
    const R one = R(1), rf = R(3), qf = R(1.5), tre = R(3);
    const R p1 = Const<R>::p1(), p2 = Const<R>::p2();
    const R rho = f[0] + f[1] + f[2] + f[3] + f[4] + f[5] + f[6] + f[7] + f[8] + f[9] + f[10] + f[11] + f[12] +
                  f[13] + f[14] + f[15] + f[16] + f[17] + f[18];
    const R rhoinv = one / rho;
    const R xj = (f[0] + f[1] + f[2] + f[3] + f[4] - f[9] - f[10] - f[11] - f[12] - f[13]) * rhoinv;
    const R yj = (f[2] + f[6] + f[7] + f[8] + f[11] - f[0] - f[9] - f[15] - f[16] - f[17]) * rhoinv;
    const R zj = (f[3] + f[5] + f[6] + f[12] + f[17] - f[1] - f[8] - f[10] - f[14] - f[15]) * rhoinv;
    const R cvsq = xj * xj + yj * yj + zj * zj;
    auto fe = [&](R w, R e, R sq) { return rho * w * (one + rf * e + qf * (tre * sq * sq - cvsq)); };
    const R e[18] = {fe(p2, xj - yj, xj - yj),  fe(p2, xj - zj, xj - zj),  fe(p2, xj + yj, xj + yj),
                     fe(p2, xj + zj, xj + zj),  fe(p1, xj, xj),            fe(p1, zj, zj),
                     fe(p2, yj + zj, yj + zj),  fe(p1, yj, yj),            fe(p2, yj - zj, yj - zj),
                     fe(p2, -xj - yj, xj + yj), fe(p2, -xj - zj, xj + zj), fe(p2, -xj + yj, xj - yj),
                     fe(p2, -xj + zj, xj - zj), fe(p1, -xj, xj),           fe(p1, -zj, zj),
                     fe(p2, -yj - zj, yj + zj), fe(p1, -yj, yj),           fe(p2, -yj + zj, yj - zj)};
    const R visc = one - R(0.5) * omega;
    R xx = -rho / rf, xy = R(0);
#pragma unroll
    for (int q = 0; q < 18; ++q) {
        const R fn = f[q] - e[q];
        xx = xx - visc * R(cx_of(q)) * R(cx_of(q)) * fn;
        xy = xy - visc * R(cx_of(q)) * R(cy_of(q)) * fn;
    }
    sxx = xx;
    sxy = xy;
}

// The four faces of a control volume, FP64 sums: face 0/1 x = i1/i2 (stress
// xx over j1..j2, k1..k2), face 2/3 y = j1/j2 (stress xy over i1..i2, k1..k2).
struct CvBox {
    int i1, i2, j1, j2, k1, k2;
};

template <typename S, typename R>
__global__ void k_cv_drag(Lat<S, R> L, Geo g, CvBox b, R omega, Reduce red, double* out) {
    const int64_t nx = (int64_t)(b.j2 - b.j1 + 1) * (b.k2 - b.k1 + 1);
    const int64_t ny = (int64_t)(b.i2 - b.i1 + 1) * (b.k2 - b.k1 + 1);
    const int64_t total = 2 * nx + 2 * ny;
    double s[4] = {0, 0, 0, 0};
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total;
         t += (int64_t)gridDim.x * blockDim.x) {
        int face, i, j, k;
        if (t < 2 * nx) {
            face = (int)(t / nx);
            const int64_t r = t % nx;
            i = face ? b.i2 : b.i1;
            j = b.j1 + (int)(r % (b.j2 - b.j1 + 1));
            k = b.k1 + (int)(r / (b.j2 - b.j1 + 1));
        } else {
            const int64_t u = t - 2 * nx;
            face = 2 + (int)(u / ny);
            const int64_t r = u % ny;
            j = face == 3 ? b.j2 : b.j1;
            i = b.i1 + (int)(r % (b.i2 - b.i1 + 1));
            k = b.k1 + (int)(r / (b.i2 - b.i1 + 1));
        }
        R xx, xy;
        ref_stress(L, g.lin(i, j, k), omega, xx, xy);
        s[face] += face < 2 ? (double)xx : (double)xy;
    }
    block_reduce_store<4>(s, red, out);
}

// Population q of the seeded equilibrium state (init_eq.h) over the haloed
// node range, into a staging buffer laid out like one host array.
template <typename T>
__global__ void k_init_population(T* out, int q, int64_t total, double u_in, double amp, uint64_t seed) {
    for (int64_t L = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; L < total; L += (int64_t)gridDim.x * blockDim.x) {
        T f[19];
        init_node<T>(L, u_in, amp, seed, f);
        out[L] = f[q];
    }
}

template <typename S, typename R>
__global__ void k_probes(Lat<S, R> L, Geo g, int npts, const int32_t* ijk, double* out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= npts) return;
    const int i = ijk[3 * p], j = ijk[3 * p + 1], k = ijk[3 * p + 2];
    double a[19];
    for (int q = 0; q < 19; ++q) a[q] = (double)lat_load(L, g, q, i, j, k);
    double rho = 0.0;
    for (int q = 0; q < 19; ++q) rho += a[q];
    out[4 * p] = rho;
    out[4 * p + 1] = (a[0] + a[1] + a[2] + a[3] + a[4] - a[9] - a[10] - a[11] - a[12] - a[13]) / rho;
    out[4 * p + 2] = (a[2] + a[6] + a[7] + a[8] + a[11] - a[0] - a[9] - a[15] - a[16] - a[17]) / rho;
    out[4 * p + 3] = (a[3] + a[5] + a[6] + a[12] + a[17] - a[1] - a[8] - a[10] - a[14] - a[15]) / rho;
}

// ---- host layout <-> device layout ------------------------------------------------------
// Host values (T = float or double) of populations q0 + blockIdx.y into the lattice and the
// halo shell, `stride` values apart.  16-bit storage
// from double converts in double: f = w + D/scale is exact there, so a state downloaded as
// double and uploaded again keeps every bit of D (through float, deviations below 2^-6
// lose their low bits to the rounding of f).  A host value that is not finite sets bit q
// of *bad (the caller rejects the state).
template <typename S, typename R, typename T>
__global__ void k_scatter(const __grid_constant__ Lat<S, R> L, Geo g, int q0, const T* from, int64_t stride,
                          int64_t total, unsigned int* bad) {
    constexpr bool exact16 = DevStore<S>::value && sizeof(T) == 8;
    const int q = q0 + (int)blockIdx.y;
    const T* src = from + blockIdx.y * stride;
    const int64_t L2 = g.l + 2, M2 = g.m + 2;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(idx % L2), j = (int)((idx / L2) % M2), k = (int)(idx / (L2 * M2));
        if (!isfinite(src[idx])) atomicOr(bad, 1u << q);
        const R v = (R)src[idx];
        if (g.interior(i, j, k)) {
            if constexpr (exact16)
                L.pop[q][g.lin(i, j, k)] =
                    DevStore<S>::from_d(((double)src[idx] - (double)weight<float>(q)) * (double)L.scale);
            else
                L.pop[q][g.lin(i, j, k)] = Store<S, R>::store(v, q, L.scale);
        } else {
            L.ghost[(int64_t)q * g.G + g.gidx(i, j, k)] = v;
        }
    }
}

// The lattice and halo shell as host values; 16-bit storage to double in double (exact).
template <typename S, typename R, typename T>
__global__ void k_gather(const __grid_constant__ Lat<S, R> L, Geo g, int q0, T* to, int64_t stride, int64_t total) {
    constexpr bool exact16 = DevStore<S>::value && sizeof(T) == 8;
    const int q = q0 + (int)blockIdx.y;
    T* dst = to + blockIdx.y * stride;
    const int64_t L2 = g.l + 2, M2 = g.m + 2;
    for (int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
         idx += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(idx % L2), j = (int)((idx / L2) % M2), k = (int)(idx / (L2 * M2));
        if constexpr (exact16) {
            if (g.interior(i, j, k)) {
                dst[idx] = (double)weight<float>(q) +
                           (double)DevStore<S>::to_f(L.pop[q][g.lin(i, j, k)]) * (double)L.inv_scale;
                continue;
            }
        }
        dst[idx] = (T)lat_load(L, g, q, i, j, k);
    }
}

// x-face copy of the current lattice (after an upload): one thread per (j,k).
template <typename S, typename R>
__global__ void k_fill_xface(Lat<S, R> L, Geo g) {
    // one thread per (side, q, j, k), j fastest: the stores are coalesced, and every load
    // (a column of the lattice, stride l) is in flight at once
    const int64_t mn = (int64_t)g.m * g.n;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 36 * mn) return;
    const int sq = (int)(t / mn);  // side * 18 + q
    const int64_t jk = t - sq * mn;
    const int side = sq / 18, q = sq - 18 * side;
    const int j = (int)(jk % g.m) + 1, k = (int)(jk / g.m) + 1;
    L.xface[xface_idx(g, side, q, j, k)] = lat_load(L, g, q, side ? g.l : 1, j, k);
}

unsigned grid_for(int64_t work, int tpb, unsigned cap = 148u * 16u) {
    int64_t b = (work + tpb - 1) / tpb;
    if (b < 1) b = 1;
    if (b > cap) b = cap;
    return (unsigned)b;
}

}  // namespace

// x-slab faces: pack the five populations leaving through column x = 1 (side 0,
// cx = -1: q 9..13) or x = l (side 1, cx = +1: q 0..4), halo rows j = 0, m+1
// and k = 0, n+1 included, as a later load returns them; unpack received
// planes into the x = 0 (side 0, q 0..4) or x = l+1 (side 1, q 9..13) halo.
template <typename S, typename R>
__global__ void k_pack_x(Lat<S, R> L, Geo g, int side, R* out) {
    const int64_t plane = (int64_t)(g.m + 2) * (g.n + 2);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 5 * plane) return;
    const int c = (int)(t / plane);
    const int64_t jk = t % plane;
    const int j = (int)(jk % (g.m + 2)), k = (int)(jk / (g.m + 2));
    const int q = side ? c : 9 + c;
    const int i = side ? g.l : 1;
    out[t] = bc_load(L, g, q, i, j, k);
}

// The rim of the x-face copy's plane messages: the five outgoing populations on the
// halo rows of each exchange face column (sides: bit 0 = x = 1, bit 1 = x = l), read
// after the halo kernels wrote them.
template <typename S, typename R>
__global__ void k_pack_x_rim(Lat<S, R> L, Geo g, int sides) {
    const int64_t per = g.xr / 5;  // halo-row nodes of one face plane
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 2 * g.xr) return;
    const int side = (int)(t / g.xr);
    if (!((sides >> side) & 1)) return;
    const int64_t r = t - side * g.xr;
    const int c = (int)(r / per);
    int j, k;
    xface_rim_node(g, r - c * per, &j, &k);
    const int q = side ? c : 9 + c;
    L.xface[xface_rim_offset(g, side) + r] = lat_load(L, g, q, side ? g.l : 1, j, k);
}

// A received plane message into the x = 0 (side 0, q 0..4) or x = l+1 (side 1,
// q 9..13) halo plane.  It left the neighbour's opposite side: into side 0 come
// the five m*n blocks then the rim, into side 1 the rim then the blocks.
template <typename S, typename R>
__global__ void k_unpack_x_view(Lat<S, R> L, Geo g, int side, const R* in) {
    const int64_t mn = g.mn, per = g.xr / 5;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 5 * mn + g.xr) return;
    const int64_t b = side ? t - g.xr : t;  // position among the blocks (< 0: on the rim)
    int c, j, k;
    if (b >= 0 && b < 5 * mn) {
        c = (int)(b / mn);
        const int64_t jk = b - c * mn;
        j = (int)(jk % g.m) + 1;
        k = (int)(jk / g.m) + 1;
    } else {
        const int64_t r = side ? t : t - 5 * mn;
        c = (int)(r / per);
        xface_rim_node(g, r - c * per, &j, &k);
    }
    const int q = side ? 9 + c : c;
    const int i = side ? g.l + 1 : 0;
    L.ghost[(int64_t)q * g.G + g.gidx(i, j, k)] = in[t];
}

template <typename S, typename R>
__global__ void k_unpack_x(Lat<S, R> L, Geo g, int side, const R* in) {
    const int64_t plane = (int64_t)(g.m + 2) * (g.n + 2);
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 5 * plane) return;
    const int c = (int)(t / plane);
    const int64_t jk = t % plane;
    const int j = (int)(jk % (g.m + 2)), k = (int)(jk / (g.m + 2));
    const int q = side ? 9 + c : c;
    const int i = side ? g.l + 1 : 0;
    L.ghost[(int64_t)q * g.G + g.gidx(i, j, k)] = in[t];
}

template <typename S, typename R>
void launch_pack_x(const Lat<S, R>& L, const Geo& g, int side, R* out, cudaStream_t st) {
    const int64_t work = 5 * (int64_t)(g.m + 2) * (g.n + 2);
    k_pack_x<S, R><<<(unsigned)((work + kTpb - 1) / kTpb), kTpb, 0, st>>>(L, g, side, out);
}

template <typename S, typename R>
void launch_pack_x_rim(const Lat<S, R>& L, const Geo& g, int sides, cudaStream_t st) {
    const int64_t work = 2 * g.xr;
    k_pack_x_rim<S, R><<<(unsigned)((work + kTpb - 1) / kTpb), kTpb, 0, st>>>(L, g, sides);
}

template <typename S, typename R>
void launch_unpack_x_view(const Lat<S, R>& L, const Geo& g, int side, const R* in, cudaStream_t st) {
    const int64_t work = 5 * (int64_t)(g.m + 2) * (g.n + 2);
    k_unpack_x_view<S, R><<<(unsigned)((work + kTpb - 1) / kTpb), kTpb, 0, st>>>(L, g, side, in);
}

template <typename S, typename R>
void launch_unpack_x(const Lat<S, R>& L, const Geo& g, int side, const R* in, cudaStream_t st) {
    const int64_t work = 5 * (int64_t)(g.m + 2) * (g.n + 2);
    k_unpack_x<S, R><<<(unsigned)((work + kTpb - 1) / kTpb), kTpb, 0, st>>>(L, g, side, in);
}

template <typename S, typename R>
int launch_bc(const Lat<S, R>& L, const Geo& g, const int bc[6], const Phys<R>& ph, const HaloEdgesDevice& edges,
              const LaunchTo& to, bool separate, const ForceSum* force) {
    HaloPlan<S, R> p{};
    p.L = L;
    p.g = g;
    p.force = ph.force;
    halo_inflow(ph.u_inflow, p.inflow);
    int n = 0, launches = 0;
    auto run = [&] {
        if (n == 0) return;
        const unsigned blocks = p.first[n];
        for (int s = n; s <= kHaloSegments; ++s) p.first[s] = 0xffffffffu;  // no block reaches them
        launch(k_halo<S, R>, blocks, kTpb, to, p);
        ++launches;
        n = 0;
        p.first[0] = 0;
    };
    auto add = [&](const HaloSegment<S, R>& f) {
        p.seg[n] = f;
        p.first[n + 1] = p.first[n] + (f.count + kTpb - 1) / kTpb;
        ++n;
    };
    p.first[0] = 0;
    if (force) {
        p.sum = *force;
        HaloSegment<S, R> f{};
        f.kind = kSegForce;
        f.count = kTpb;
        add(f);
    }
    for (int b = 0; b < kHaloBlocks; ++b) {
        const int before = n;
        const HaloFace face = record_halo_face(g, bc, b);
        if (face.kind != kFaceNone) {
            HaloSegment<S, R> f{};
            f.kind = face.kind;
            f.na = (unsigned)face.na;
            f.nb = (unsigned)face.nb;
            f.count = f.na * f.nb;
            f.src_b = face.src_b;
            f.dst_b = face.dst_b;
            f.pass = face.pass;
            f.pass_dst = L.ghost + face.pass_dst;
            for (int c = 0; c < 5; ++c) {
                f.dst[c] = L.ghost + face.dst[c];
                f.da[c] = face.da[c];
                f.db[c] = face.db[c];
                f.add[c] = face.lid[c] < 0 ? -ph.force : ph.force;
                f.lid |= face.lid[c] != 0 ? 1 << c : 0;
                if (face.kind == kFaceConst) f.w[c] = p.inflow[face.src_q[c]];
                if (face.kind == kFaceCopyX) f.src[c] = L.xface + face.src[c];
                if (face.kind == kFaceCopy) {
                    f.src[c] = L.pop[face.src_q[c]] + face.src[c];
                    f.w[c] = wclass_of(face.src_q[c]) == 1 ? R(1.0 / 18.0) : R(1.0 / 36.0);
                }
            }
            add(f);
        }
        if (edges.first[b + 1] > edges.first[b]) {
            HaloSegment<S, R> f{};
            f.kind = kSegEdges;
            f.count = (unsigned)(edges.first[b + 1] - edges.first[b]);
            f.edges = edges.e + edges.first[b];
            add(f);
        }
        if (separate && n > before) run();
    }
    run();
    return launches;
}

template <typename S, typename R>
BounceArgs<S, R> bounce_args(const Lat<S, R>& L, const Geo& g, const LinksDevice& links, const Reduce& red) {
    BounceArgs<S, R> p{};
    p.L = L;
    p.g = g;
    p.links = links;
    for (int q = 0; q < 18; ++q) {
        p.from[q] = L.pop[opp_of(q)] + (cx_of(q) + (int64_t)cy_of(q) * g.l + (int64_t)cz_of(q) * g.lm);
        p.w[q] = wclass_of(q) == 1 ? R(1.0 / 18.0) : R(1.0 / 36.0);
        p.c2[q][0] = -2.0 * cx_of(q);
        p.c2[q][1] = -2.0 * cy_of(q);
        p.c2[q][2] = -2.0 * cz_of(q);
    }
    p.partials = red.partials;
    p.counter = red.counter;
    return p;
}

template <typename S, typename R>
ForceSum launch_bounce(const Lat<S, R>& L, const Geo& g, const LinksDevice& links, const Reduce& red, double* series,
                       int64_t cap, int64_t* d_itime, const LaunchTo& to) {
    ForceSum sum{red.partials, 0, series, cap, d_itime, nullptr};
    if (links.nfluid + links.nhalo == 0) return sum;
    BounceArgs<S, R> p = bounce_args(L, g, links, red);
    p.bounce = 1;
    sum.blocks = (int)grid_for(links.nfluid + links.nhalo, kTpb, (unsigned)red.max_blocks);
    launch(k_bounce<S, R>, (unsigned)sum.blocks, kTpb, to, p);
    return sum;
}

template <typename S, typename R>
void launch_force(const Lat<S, R>& L, const Geo& g, const LinksDevice& links, const Reduce& red, double* series,
                  int64_t cap, int64_t* d_itime, double* host, cudaStream_t st) {
    BounceArgs<S, R> p = bounce_args(L, g, links, red);
    p.finish = 1;
    p.sum = ForceSum{red.partials, (int)grid_for(links.nfluid + links.nhalo, kTpb, (unsigned)red.max_blocks), series,
                     cap, d_itime, host};
    k_bounce<S, R><<<(unsigned)p.sum.blocks, kTpb, 0, st>>>(p);
}

template <typename S, typename R>
void launch_fill_xface(const Lat<S, R>& L, const Geo& g, cudaStream_t st) {
    const int64_t work = 36 * (int64_t)g.m * g.n;
    k_fill_xface<S, R><<<(unsigned)((work + kTpb - 1) / kTpb), kTpb, 0, st>>>(L, g);
}

template <typename S, typename R>
void launch_monitor(const Lat<S, R>& L, const Geo& g, const Mask& mk, const Reduce& red, double* out,
                    cudaStream_t st) {
    const RowWalk w = row_walk(g.l, (int64_t)g.m * g.n);
    k_monitor<S, R><<<grid_for(w.units, kTpb / 32, (unsigned)red.max_blocks), kTpb, 0, st>>>(L, w, mk, red, out);
}

template <typename S, typename R>
void launch_region_sums(const Lat<S, R>& L, const Geo& g, const Mask& mk, const uint8_t* region, const Reduce& red,
                        double* out, cudaStream_t st) {
    const RowWalk w = row_walk(g.l, (int64_t)g.m * g.n);
    k_region_sums<S, R><<<grid_for(w.units, kTpb / 32, (unsigned)red.max_blocks), kTpb, 0, st>>>(L, w, mk, region, red,
                                                                                                out);
}

template <typename S, typename R>
void launch_line(const Lat<S, R>& L, const Geo& g, int axis, int c1, int c2, double* out, cudaStream_t st) {
    const int len = axis == 0 ? g.l : (axis == 1 ? g.m : g.n);
    k_line<S, R><<<(len + 127) / 128, 128, 0, st>>>(L, g, axis, c1, c2, out);
}

int64_t plane_means_scratch(const Geo& g, int axis) { return plane_split(g.l, g.m, g.n, axis).scratch(axis); }

template <typename S, typename R>
void launch_plane_means(const Lat<S, R>& L, const Geo& g, int axis, double* out, double* scratch, cudaStream_t st) {
    const PlaneSplit p = plane_split(g.l, g.m, g.n, axis);
    const PlaneWalk& w = p.w;
    const dim3 block(p.tx, p.ty);
    const unsigned blocks = (unsigned)p.blocks();
    const int parts = w.shares * w.xblocks;
    const double nodes = axis == 0 ? (double)g.m * g.n : (double)g.l * w.rows;
    if (axis == 0) {
        k_plane_sums<S, R, true><<<blocks, block, 0, st>>>(L, w, 1.0, scratch);
        k_add_planes<<<g.l, 256, 0, st>>>(scratch, 1, g.l, 4 * (int64_t)g.l, w.shares * p.ty, nodes, out);
    } else if (parts == 1) {
        k_plane_sums<S, R, false><<<blocks, block, 0, st>>>(L, w, nodes, out);
    } else {
        k_plane_sums<S, R, false><<<blocks, block, 0, st>>>(L, w, 1.0, scratch);
        k_add_planes<<<p.planes, 256, 0, st>>>(scratch, 4 * (int64_t)parts, 1, 4, parts, nodes, out);
    }
}

template <typename S, typename R>
void launch_cv_drag(const Lat<S, R>& L, const Geo& g, const int box[6], R omega, const Reduce& red, double* out,
                    cudaStream_t st) {
    const CvBox b{box[0], box[1], box[2], box[3], box[4], box[5]};
    const int64_t total = 2 * (int64_t)(b.j2 - b.j1 + 1) * (b.k2 - b.k1 + 1) +
                          2 * (int64_t)(b.i2 - b.i1 + 1) * (b.k2 - b.k1 + 1);
    k_cv_drag<S, R><<<grid_for(total, kTpb, (unsigned)red.max_blocks), kTpb, 0, st>>>(L, g, b, omega, red, out);
}

template <typename T>
void launch_init_population(T* staging, const Geo& g, int q, double u_in, double amp, uint64_t seed, cudaStream_t st) {
    const int64_t total = (int64_t)(g.l + 2) * (g.m + 2) * (g.n + 2);
    k_init_population<T><<<grid_for(total, kTpb), kTpb, 0, st>>>(staging, q, total, u_in, amp, seed);
}
template void launch_init_population<float>(float*, const Geo&, int, double, double, uint64_t, cudaStream_t);
template void launch_init_population<double>(double*, const Geo&, int, double, double, uint64_t, cudaStream_t);

template <typename S, typename R>
void launch_probes(const Lat<S, R>& L, const Geo& g, int npts, const int32_t* ijk, double* out,
                   cudaStream_t st) {
    k_probes<S, R><<<(npts + 127) / 128, 128, 0, st>>>(L, g, npts, ijk, out);
}

template <typename S, typename R, typename T>
void launch_scatter(const Lat<S, R>& L, const Geo& g, int q, int nq, const T* staging, unsigned int* bad,
                    cudaStream_t st) {
    const int64_t total = (int64_t)(g.l + 2) * (g.m + 2) * (g.n + 2);
    k_scatter<S, R, T><<<dim3(grid_for(total, kTpb), nq), kTpb, 0, st>>>(L, g, q, staging, total, total, bad);
}

template <typename S, typename R, typename T>
void launch_gather(const Lat<S, R>& L, const Geo& g, int q, int nq, T* staging, cudaStream_t st) {
    const int64_t total = (int64_t)(g.l + 2) * (g.m + 2) * (g.n + 2);
    k_gather<S, R, T><<<dim3(grid_for(total, kTpb), nq), kTpb, 0, st>>>(L, g, q, staging, total, total);
}

#define EUP_INST(S, R)                                                                                 \
    template int launch_bc<S, R>(const Lat<S, R>&, const Geo&, const int*, const Phys<R>&, const HaloEdgesDevice&, \
                                 const LaunchTo&, bool, const ForceSum*);                                    \
    template ForceSum launch_bounce<S, R>(const Lat<S, R>&, const Geo&, const LinksDevice&, const Reduce&, double*, \
                                          int64_t, int64_t*, const LaunchTo&);                         \
    template void launch_force<S, R>(const Lat<S, R>&, const Geo&, const LinksDevice&, const Reduce&, double*, \
                                     int64_t, int64_t*, double*, cudaStream_t);                        \
    template void launch_fill_xface<S, R>(const Lat<S, R>&, const Geo&, cudaStream_t);                 \
    template void launch_pack_x<S, R>(const Lat<S, R>&, const Geo&, int, R*, cudaStream_t);              \
    template void launch_unpack_x<S, R>(const Lat<S, R>&, const Geo&, int, const R*, cudaStream_t);      \
    template void launch_pack_x_rim<S, R>(const Lat<S, R>&, const Geo&, int, cudaStream_t);              \
    template void launch_unpack_x_view<S, R>(const Lat<S, R>&, const Geo&, int, const R*, cudaStream_t); \
    template void launch_line<S, R>(const Lat<S, R>&, const Geo&, int, int, int, double*, cudaStream_t);   \
    template void launch_plane_means<S, R>(const Lat<S, R>&, const Geo&, int, double*, double*, cudaStream_t); \
    template void launch_cv_drag<S, R>(const Lat<S, R>&, const Geo&, const int*, R, const Reduce&, double*, \
                                       cudaStream_t);                                                     \
    template void launch_region_sums<S, R>(const Lat<S, R>&, const Geo&, const Mask&, const uint8_t*,   \
                                           const Reduce&, double*, cudaStream_t);                         \
    template void launch_monitor<S, R>(const Lat<S, R>&, const Geo&, const Mask&, const Reduce&,       \
                                       double*, cudaStream_t);                                         \
    template void launch_probes<S, R>(const Lat<S, R>&, const Geo&, int, const int32_t*, double*,      \
                                      cudaStream_t);                                                   \
    template void launch_scatter<S, R, float>(const Lat<S, R>&, const Geo&, int, int, const float*,         \
                                              unsigned int*, cudaStream_t);                            \
    template void launch_scatter<S, R, double>(const Lat<S, R>&, const Geo&, int, int, const double*,       \
                                               unsigned int*, cudaStream_t);                           \
    template void launch_gather<S, R, float>(const Lat<S, R>&, const Geo&, int, int, float*, cudaStream_t); \
    template void launch_gather<S, R, double>(const Lat<S, R>&, const Geo&, int, int, double*, cudaStream_t);

EUP_INST(float, float)
EUP_INST(double, double)
EUP_INST(__half, float)
EUP_INST(__nv_bfloat16, float)

}  // namespace eup
