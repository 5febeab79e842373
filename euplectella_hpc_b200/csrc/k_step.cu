// Fused pull stream + collide: for every interior node x,
//   f_q = a_q(x - c_q)            (CODE/SRC/movef.F90:48-65; a19 stays, :125 of col)
//   a'  = collide(f)              (CODE/SRC/col.F90:127-229)
// reading the source lattice and halo shell, writing the destination lattice.
// Nodes whose 18 upstream neighbours are all interior take the fast path
// (plain shifted loads); nodes on the six boundary planes resolve each pull
// through the halo shell.
#include <string.h>

#include <type_traits>

#include "internal.h"
#include "pbb_plan.h"

namespace eup {

namespace {

// What the kernels compute with: the population f itself (FP32/FP64 storage,
// reference arithmetic), or the scaled deviation D = (f - w)*S (16-bit
// storage, collide_dev).  Values from the halo shell are always f.
template <typename S, typename R>
struct KOps {
    static constexpr bool dev = DevStore<S>::value;
    static __device__ __forceinline__ R val(S raw, int q, const Lat<S, R>& L) {
        if constexpr (dev) return DevStore<S>::to_f(raw);
        else return Store<S, R>::load(raw, q, L.inv_scale);
    }
    static __device__ __forceinline__ R from_shell(R f, int q, const Lat<S, R>& L) {
        if constexpr (dev) return (f - weight<R>(q)) * L.scale;
        else return f;
    }
    static __device__ __forceinline__ R pull(const Lat<S, R>& L, const Geo& g, int q, int i, int j, int k) {
        if (g.interior(i, j, k)) return val(L.pop[q][g.lin(i, j, k)], q, L);
        return from_shell(L.ghost[(int64_t)q * g.G + g.gidx(i, j, k)], q, L);
    }
    static __device__ __forceinline__ void collide_node(R* x, const Phys<R>& ph, const Lat<S, R>& L) {
        if constexpr (dev) collide_dev(x, ph.omega, ph.omega1, ph.fgrad, L.scale, L.inv_scale);
        else collide<R>(x, ph.omega, ph.omega1, ph.fgrad);
    }
    static __device__ __forceinline__ S store(R v, int q, const Lat<S, R>& L) {
        if constexpr (dev) return DevStore<S>::from_f(v);
        else return Store<S, R>::store(v, q, L.scale);
    }
};

// Whether the row (j - cy, k - cz) that population q is pulled from lies on a y or z halo
// plane, and where it starts in the shell then (*row: the element of x = 1; an x plane's element
// only ever replaces the end values of a row).  j and k belong to the row, so this is
// uniform over a block of the row kernels; rows away from the boundary planes never ask.
template <typename R>
__device__ __forceinline__ bool halo_row(const R* ghost, const Geo& g, int q, int j, int k, const R** row) {
    const int cy = cy_of(q), cz = cz_of(q);
    const bool oy = cy == 1 ? j == 1 : (cy == -1 ? j == g.m : false);
    const bool oz = cz == 1 ? k == 1 : (cz == -1 ? k == g.n : false);
    const int64_t y = (cy == 1 ? g.oy0 : g.oym) + (int64_t)(k - cz) * g.l;
    const int64_t z = (cz == 1 ? g.oz0 : g.ozn) + (int64_t)(j - cy - 1) * g.l;
    *row = ghost + ((int64_t)q * g.G + (oy ? y : z));
    return oy | oz;
}

// Streamed populations of interior node (i, j, k); rowlin = l*((j-1) + m*(k-1))
// is the linear index of x = 1 on its row (32-bit: one lattice holds fewer than
// 2^31 nodes).  Every source row pointer depends on the row only, so it is the
// same for the whole warp and each load is that pointer plus the thread's x.
// All 18 shifted loads are issued unconditionally, and the five x-halo values of
// the first/last node of a row replace them afterwards: a shifted index off the end
// of a row reads the neighbouring row, the population's padding, or on a halo row the
// neighbouring element of the shell.  A row on the y/z boundary planes pulls some
// populations from halo rows instead (halo_row): only the pointers differ.
template <typename S, typename R>
__device__ __forceinline__ void gather_node(const Lat<S, R>& src, const Geo& g, int i, int j, int k, int rowlin,
                                            R (&x)[19]) {
    using K = KOps<S, R>;
    const int l = g.l, lm = (int)g.lm;
    const bool face_yz = (j == 1) | (j == g.m) | (k == 1) | (k == g.n);
    if (!face_yz) {
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            const S* rp = src.pop[q] + (rowlin - cy_of(q) * l - cz_of(q) * lm);
            x[q] = K::val(rp[i - 1 - cx_of(q)], q, src);
        }
    } else if constexpr (!K::dev) {
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            const R* halo;
            const bool out = halo_row(src.ghost, g, q, j, k, &halo);
            const S* rp = out ? halo : src.pop[q] + (rowlin - cy_of(q) * l - cz_of(q) * lm);
            x[q] = rp[i - 1 - cx_of(q)];
        }
    } else {  // lattice and shell hold different types: both loads, one of them at a place that is there
        S raw[18];
        R f[18];
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            const R* halo;
            const bool out = halo_row(src.ghost, g, q, j, k, &halo);
            raw[q] = (src.pop[q] + (out ? rowlin : rowlin - cy_of(q) * l - cz_of(q) * lm))[i - 1 - cx_of(q)];
            f[q] = (out ? halo : src.ghost)[out ? i - 1 - cx_of(q) : 0];
        }
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            const R* halo;
            x[q] = halo_row(src.ghost, g, q, j, k, &halo) ? K::from_shell(f[q], q, src) : K::val(raw[q], q, src);
        }
    }
    if (i == 1) {
#pragma unroll
        for (int q = 0; q < 18; ++q)
            if (cx_of(q) == 1)
                x[q] = K::from_shell(src.ghost[(int64_t)q * g.G + g.gidx(0, j - cy_of(q), k - cz_of(q))], q, src);
    }
    if (i == l) {
#pragma unroll
        for (int q = 0; q < 18; ++q)
            if (cx_of(q) == -1)
                x[q] = K::from_shell(src.ghost[(int64_t)q * g.G + g.gidx(l + 1, j - cy_of(q), k - cz_of(q))], q, src);
    }
    x[18] = K::val(src.pop[18][rowlin + i - 1], 18, src);
}

template <typename S, typename R>
__device__ __forceinline__ void scatter_node(const Lat<S, R>& dst, const Geo& g, int i, int j, int k, int rowlin,
                                             const R (&x)[19]) {
    using K = KOps<S, R>;
    S out[19];
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        out[q] = K::store(x[q], q, dst);
        (dst.pop[q] + rowlin)[i - 1] = out[q];
    }
    if (i == 1 || i == g.l) {
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            const R v = Store<S, R>::load(out[q], q, dst.inv_scale);
            if (i == 1) dst.xface[xface_idx(g, 0, q, j, k)] = v;
            if (i == g.l) dst.xface[xface_idx(g, 1, q, j, k)] = v;
        }
    }
}

template <typename S, typename R>
__device__ __forceinline__ void node_step(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g,
                                          const Phys<R>& ph, int i, int j, int k) {
    const int rowlin = g.l * ((j - 1) + g.m * (k - 1));
    R x[19];
    gather_node(src, g, i, j, k, rowlin, x);
    KOps<S, R>::collide_node(x, ph, src);
    scatter_node(dst, g, i, j, k, rowlin, x);
}

// Plane of thread block z: upwards, or with DOWN from k = n down (see launch_stream_collide).
template <bool DOWN>
__device__ __forceinline__ int plane_of_block(const Geo& g) {
    return DOWN ? g.n - (int)blockIdx.z : (int)blockIdx.z + 1;
}

// One thread per node of the columns i0 .. i0+ni-1; grid (ceil(ni/bx), m, n).
template <typename S, typename R, bool DOWN>
__global__ void __launch_bounds__(128) k_stream_collide_scalar(Lat<S, R> src, Lat<S, R> dst, Geo g, Phys<R> ph,
                                                               int i0, int ni) {
    chain_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ni) return;
    node_step(src, dst, g, ph, i0 + t, (int)blockIdx.y + 1, plane_of_block<DOWN>(g));
}

// The columns i = 1 and i = l (the only ones that pull from the x halo planes): one thread
// per (side, j, k); sides = 1 when l == 1.
template <typename S, typename R>
__global__ void __launch_bounds__(128) k_stream_collide_scalar_faces(Lat<S, R> src, Lat<S, R> dst, Geo g,
                                                                     Phys<R> ph, int sides) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)sides * g.m * g.n) return;
    const int side = (int)(t % sides);
    const int64_t row = t / sides;
    node_step(src, dst, g, ph, side ? g.l : 1, (int)(row % g.m) + 1, (int)(row / g.m) + 1);
}

// The partial-bounce-back step in one pass (the same values as in two, launch_pbb_step): streams and
// collides a node, and where n_s > 0 mixes the collided values, as storage rounds them, with the
// pulled ones and adds the momentum the solid takes.  Grid: nbx blocks to a row, `each` rows to a
// block.  The 38 values of a node cost occupancy (FP32 72 registers, FP64 124): at 192x96x96
// FP32 a step takes 82 us summing the force and 70 without, where the plain step takes 57.
// Pulling the values again after the collision instead of keeping them: 93-157 us; rows of a
// block far apart instead of next to one another: no change.
template <typename S, typename R>
__global__ void __launch_bounds__(128) k_pbb_whole(Lat<S, R> src, Lat<S, R> dst, Geo g, Phys<R> ph, const R* ns,
                                                   int nbx, int each, int down, Reduce red, double* series,
                                                   int64_t cap, int64_t* d_itime) {
    using K = KOps<S, R>;
    const int first = (int)blockIdx.x / nbx;
    const int i = ((int)blockIdx.x - first * nbx) * (int)blockDim.x + (int)threadIdx.x + 1;
    const int rows = g.m * g.n, end = i <= g.l ? min(rows, (first + 1) * each) : 0;
    double f[3] = {0.0, 0.0, 0.0};
    chain_begin();
    for (int r = first * each; r < end; ++r) {
        const int row = down ? rows - 1 - r : r;
        const int k = row / g.m + 1, j = row - (k - 1) * g.m + 1;
        const int rowlin = g.l * row;
        R pre[19], x[19];
        const R s = ns[rowlin + i - 1], s1 = R(1) - s;
        gather_node(src, g, i, j, k, rowlin, pre);
#pragma unroll
        for (int q = 0; q < 19; ++q) x[q] = pre[q];
        K::collide_node(x, ph, src);
        if (s > R(0)) {
            if (series) pbb_momentum(pre, s, K::dev ? 1.0 / (double)src.scale : 1.0, f);
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                if constexpr (K::dev) x[q] = DevStore<S>::to_f(DevStore<S>::from_f(x[q]));
                x[q] = s1 * x[q] + s * pre[opp_of(q)];
            }
        }
        scatter_node(dst, g, i, j, k, rowlin, x);
    }
    if (series) block_reduce_store<3>(f, red, nullptr, series, cap, d_itime, 1, 1);
}

// ---------------------------------------------------------------------------
// Pair kernel (FP32 arithmetic, l even): one thread streams and collides the
// two x-adjacent nodes (i, i+1), i odd.  The collision runs once on F2 values
// -- the packed FP32 instructions of sm_100 (fma .f32x2), rounded per lane
// exactly as the scalar code -- so the FP32 instruction count per node halves
// and the results equal the one-node kernel's bit for bit.  FP32 storage: the
// pulls with cx = 0 and every store move both nodes as one aligned 8-byte
// access, pulls with cx = +-1 are two scalar loads.  16-bit storage shifts
// population q by cx_q elements in memory, so all 19 pulls are aligned 4-byte
// loads (two nodes in one register: twice the bytes in flight per register);
// the stores of the ten populations with cx = +-1 are then two scalar stores.
// grid (ceil(l/2 / 128), m, n).
// ---------------------------------------------------------------------------
template <typename S> struct Vec2;
template <> struct Vec2<float> {
    using T = float2;
    static __device__ __forceinline__ float2 unpack(float2 v) { return v; }
    static __device__ __forceinline__ float2 pack(float2 v) { return v; }
    static __device__ __forceinline__ float lo(float2 v) { return v.x; }
    static __device__ __forceinline__ float hi(float2 v) { return v.y; }
};
template <> struct Vec2<__half> {
    using T = __half2;
    static __device__ __forceinline__ float2 unpack(__half2 v) { return __half22float2(v); }
    static __device__ __forceinline__ __half2 pack(float2 v) { return __float22half2_rn(v); }
    static __device__ __forceinline__ __half lo(__half2 v) { return __low2half(v); }
    static __device__ __forceinline__ __half hi(__half2 v) { return __high2half(v); }
};
template <> struct Vec2<__nv_bfloat16> {
    using T = __nv_bfloat162;
    static __device__ __forceinline__ float2 unpack(__nv_bfloat162 v) { return __bfloat1622float2(v); }
    static __device__ __forceinline__ __nv_bfloat162 pack(float2 v) { return __float22bfloat162_rn(v); }
    static __device__ __forceinline__ __nv_bfloat16 lo(__nv_bfloat162 v) { return __low2bfloat16(v); }
    static __device__ __forceinline__ __nv_bfloat16 hi(__nv_bfloat162 v) { return __high2bfloat16(v); }
};

// Population q's source pointer moved back by c_q: the pull a_q(x - c_q) of node index x
// (0-based, x = i-1 + l (j-1 + m (k-1))) is base[q][x].  Set on the host per launch.
template <typename S>
struct PullBase {
    const S* p[19];
};

// 16-bit storage: the 19 pulls of the pair (i, i+1) of an interior row as raw words
// (aligned in the shifted layout whatever cx is): one index for all of them.
template <typename S>
__device__ __forceinline__ void load_pair_raw(const PullBase<S>& pb, int i, int rowlin,
                                              typename Vec2<S>::T (&r)[19]) {
    using T2 = typename Vec2<S>::T;
    const uint32_t x = (uint32_t)(rowlin + i - 1);
#pragma unroll
    for (int q = 0; q < 19; ++q) r[q] = *reinterpret_cast<const T2*>(pb.p[q] + x);
}

// The x-halo values of the first (LO: node i = 1 in the low lane) and last (HI: node i+1 = l in
// the high lane) node of a row replace what the shifted loads brought.
template <typename S>
__device__ __forceinline__ void x_halo_ends(const Lat<S, float>& src, const Geo& g, bool lo, bool hi, int j, int k,
                                            F2 (&x)[19]) {
    using K = KOps<S, float>;
    if (lo) {
#pragma unroll
        for (int q = 0; q < 18; ++q)
            if (cx_of(q) == 1)
                x[q].v.x = K::from_shell(src.ghost[(int64_t)q * g.G + g.gidx(0, j - cy_of(q), k - cz_of(q))], q, src);
    }
    if (hi) {
#pragma unroll
        for (int q = 0; q < 18; ++q)
            if (cx_of(q) == -1)
                x[q].v.y =
                    K::from_shell(src.ghost[(int64_t)q * g.G + g.gidx(g.l + 1, j - cy_of(q), k - cz_of(q))], q, src);
    }
}

// x-face copy of the first/last column: the value a later load returns.
template <typename S>
__device__ __forceinline__ void store_x_face(const Lat<S, float>& dst, const Geo& g, bool lo, bool hi, int j, int k,
                                             const F2 (&x)[19]) {
    using V2 = Vec2<S>;
    if (lo | hi) {
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            const typename V2::T o = V2::pack(x[q].v);
            if (lo) dst.xface[xface_idx(g, 0, q, j, k)] = Store<S, float>::load(V2::lo(o), q, dst.inv_scale);
            if (hi) dst.xface[xface_idx(g, 1, q, j, k)] = Store<S, float>::load(V2::hi(o), q, dst.inv_scale);
        }
    }
}

template <typename S>
__device__ __forceinline__ void collide_pair(const Lat<S, float>& src, const Phys<float>& ph, F2 (&x)[19]) {
    if constexpr (DevStore<S>::value) collide_dev<F2>(x, ph.omega, ph.omega1, ph.fgrad, src.scale, src.inv_scale);
    else collide<F2>(x, F2(ph.omega), F2(ph.omega1), F2(ph.fgrad));
}

// Everything after the pulls of a pair: the x-halo values of the first and
// last node of the row, the collision of both nodes as packed FP32, the x-face copy and
// the stores.
template <typename S>
__device__ __forceinline__ void finish_pair(const Lat<S, float>& src, const Lat<S, float>& dst, const Geo& g,
                                            const Phys<float>& ph, int i, int j, int k, int rowlin, F2 (&x)[19]) {
    using V2 = Vec2<S>;
    using T2 = typename V2::T;
    constexpr bool dev = DevStore<S>::value;
    x_halo_ends(src, g, i == 1, i + 1 == g.l, j, k, x);
    collide_pair<S>(src, ph, x);
    store_x_face<S>(dst, g, i == 1, i + 1 == g.l, j, k, x);
#pragma unroll
    for (int q = 0; q < 19; ++q) {
        const T2 o = V2::pack(x[q].v);
        S* op = dst.pop[q] + rowlin + (i - 1);
        if (!dev || q == 18 || cx_of(q) == 0) {
            *reinterpret_cast<T2*>(op) = o;
        } else {  // odd address in the shifted layout
            op[0] = V2::lo(o);
            op[1] = V2::hi(o);
        }
    }
}

// The pair (i, i+1) of row (j, k).  A row on the y/z boundary planes (warp-uniform in the row
// kernel, where a block is one row) takes the populations that halo_row names from the shell;
// FP32 rows of both kinds share the collision and the stores.  (With the boundary rows node by
// node through the shell these rows took 12 us each, whatever the lattice: all of a 64x32x8
// step's kernel, and the tail of a larger one's, whose last rows are the plane k = n.  Per
// launch, before / now, CUDA events: 64x32x8 FP32 11.6 / 7.5 us, FP16 16.0 / 9.9; 256x128x64
// FP32 61.8 / 58.5, FP16 56 / 44.5; 768x384x384 FP32 2656 / 2645, FP16 1690 / 1664.)
template <typename S>
__device__ __forceinline__ void pair_step(const Lat<S, float>& src, const Lat<S, float>& dst, const Geo& g,
                                          const Phys<float>& ph, const PullBase<S>& pb, int i, int j, int k) {
    using K = KOps<S, float>;
    using V2 = Vec2<S>;
    using T2 = typename V2::T;
    constexpr bool dev = DevStore<S>::value;
    const int l = g.l, lm = (int)g.lm;
    const int rowlin = l * ((j - 1) + g.m * (k - 1));
    const bool face_yz = (j == 1) | (j == g.m) | (k == 1) | (k == g.n);
    F2 x[19];
    if (face_yz) {
        if constexpr (dev) {
            // one 4-byte load from the lattice (both nodes) or two from the shell, one per node;
            // a lattice row repeats its load.  By groups, so that the raw words of a few
            // populations are live beside the values of the others.
            const uint32_t n0 = (uint32_t)(rowlin + i - 1);
            constexpr int kGroup = 9;
#pragma unroll
            for (int q0 = 0; q0 < 18; q0 += kGroup) {
                uint32_t a[kGroup], b[kGroup];
#pragma unroll
                for (int c = 0; c < kGroup; ++c) {
                    const int q = q0 + c;
                    const float* halo;
                    const bool out = halo_row(src.ghost, g, q, j, k, &halo);
                    const void* p = out ? static_cast<const void*>(halo + (i - 1 - cx_of(q)))
                                        : static_cast<const void*>(pb.p[q] + n0);
                    a[c] = static_cast<const uint32_t*>(p)[0];
                    b[c] = static_cast<const uint32_t*>(p)[out ? 1 : 0];
                }
#pragma unroll
                for (int c = 0; c < kGroup; ++c) {
                    const int q = q0 + c;
                    const float* halo;
                    if (halo_row(src.ghost, g, q, j, k, &halo)) {
                        x[q] = F2(K::from_shell(__uint_as_float(a[c]), q, src),
                                  K::from_shell(__uint_as_float(b[c]), q, src));
                    } else {
                        T2 r;
                        memcpy(&r, &a[c], 4);
                        x[q] = F2(V2::unpack(r));
                    }
                }
            }
            x[18] = F2(V2::unpack(*reinterpret_cast<const T2*>(pb.p[18] + n0)));
            finish_pair(src, dst, g, ph, i, j, k, rowlin, x);
            return;  // its own collision: sharing the one below costs it 2 % at 1024x512x512
        } else {
#pragma unroll
            for (int q = 0; q < 18; ++q) {
                const float* halo;
                const bool out = halo_row(src.ghost, g, q, j, k, &halo);
                const S* rp = out ? halo : src.pop[q] + (rowlin - cy_of(q) * l - cz_of(q) * lm);
                x[q] = F2(rp[i - 1 - cx_of(q)], rp[i - cx_of(q)]);
            }
            x[18] = F2(src.pop[18][rowlin + i - 1], src.pop[18][rowlin + i]);
        }
    } else if constexpr (dev) {
        T2 r[19];
        load_pair_raw(pb, i, rowlin, r);
#pragma unroll
        for (int q = 0; q < 19; ++q) x[q] = F2(V2::unpack(r[q]));
    } else {
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const int cx = (q == 18) ? 0 : cx_of(q), cy = (q == 18) ? 0 : cy_of(q), cz = (q == 18) ? 0 : cz_of(q);
            const S* rp = src.pop[q] + (rowlin - cy * l - cz * lm);
            if (cx == 0) {
                const float2 v = V2::unpack(*reinterpret_cast<const T2*>(rp + (i - 1)));
                x[q] = F2(K::val(v.x, q, src), K::val(v.y, q, src));
            } else {
                // both shifted loads are in bounds (see gather_node)
                x[q] = F2(K::val(rp[i - 1 - cx], q, src), K::val(rp[i - cx], q, src));
            }
        }
    }
    finish_pair(src, dst, g, ph, i, j, k, rowlin, x);
}

// Pairs p0 .. p0+np-1 of every row (pair p: nodes 2p+1, 2p+2); grid (ceil(np/128), m, n).
template <typename S, int MINB, bool DOWN>
__global__ void __launch_bounds__(128, MINB) k_stream_collide_pair(Lat<S, float> src, Lat<S, float> dst, Geo g,
                                                                   Phys<float> ph, PullBase<S> pb, int p0, int np) {
    chain_begin();
    const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (t >= np) return;
    pair_step(src, dst, g, ph, pb, 2 * (p0 + t) + 1, (int)blockIdx.y + 1, plane_of_block<DOWN>(g));
}

// The first and last pair of every row (the only ones that pull from the x halo planes):
// one thread per (side, j, k); sides = 1 when l == 2.
template <typename S>
__global__ void __launch_bounds__(128, 6) k_stream_collide_pair_faces(Lat<S, float> src, Lat<S, float> dst, Geo g,
                                                                      Phys<float> ph, PullBase<S> pb, int sides) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (int64_t)sides * g.m * g.n) return;
    const int side = (int)(t % sides);
    const int64_t row = t / sides;
    pair_step(src, dst, g, ph, pb, side ? g.l - 1 : 1, (int)(row % g.m) + 1, (int)(row / g.m) + 1);
}

// Whether a step walks the planes from k = n down.  A step leaves the planes it wrote last in
// L2 (126 MB), and a step that starts with them finds them there: successive steps walk in
// turn, since they swap source and destination and the direction is the order of the two in
// memory.  Step with all upward / in turn: 256x128x64 FP32 (159 MB a lattice) 68.1 / 64.7 us, FP16
// 53.4 / 48.8, FP64 118.4 / 116.3; 127^3 FP32 75.6 / 70.8; 384x192x192 FP32 (1.1 GB) 358.9 / 354.6,
// FP16 242 / 234.  At 768x384x384 FP32 (8.6 GB) nothing is left of it, and the downward 16-bit
// kernel, whose plane index takes one more register, was the slower by 2 % there: beyond 2 GB
// every step goes up.
template <typename S, typename R>
bool sweep_down(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g) {
    if ((double)g.N * Q * sizeof(S) > 2147483648.0) return false;
    return reinterpret_cast<uintptr_t>(src.pop[0]) > reinterpret_cast<uintptr_t>(dst.pop[0]);
}

template <typename S, typename R>
bool launch_pair(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g, const Phys<R>& ph, int occ, int part,
                 const LaunchTo& to) {
    if constexpr (sizeof(R) != 4) {
        return false;
    } else {
        if (g.l % 2 != 0) return false;
        // pair accesses: FP32 at the node's own address, 16-bit storage at the address
        // shifted back by cx_q (and its stores of cx = 0 populations)
        constexpr bool dev = DevStore<S>::value;
        for (int q = 0; q < Q; ++q) {
            const int cx = (q == 18) ? 0 : cx_of(q);
            const S* s0 = dev ? src.pop[q] - cx : src.pop[q];
            if (reinterpret_cast<uintptr_t>(s0) % (2 * sizeof(S)) != 0) return false;
            if ((!dev || cx == 0) && reinterpret_cast<uintptr_t>(dst.pop[q]) % (2 * sizeof(S)) != 0) return false;
        }
        // blocks of at most 128 threads, the row's pairs split evenly over its blocks (a
        // warp multiple), so short rows leave no idle threads (l = 192: one block of 96)
        const int npr = part == kStreamInterior ? g.l / 2 - 2 : (part == kStreamFaces ? 0 : g.l / 2);
        const int nblk = npr > 0 ? (npr + 127) / 128 : 1;
        const int bx = npr > 0 ? ((npr + nblk - 1) / nblk + 31) / 32 * 32 : 128;
        PullBase<S> pb;
        for (int q = 0; q < Q; ++q) {
            const int64_t c = (q == 18) ? 0 : (int64_t)cy_of(q) * g.l + (int64_t)cz_of(q) * g.lm + cx_of(q);
            pb.p[q] = src.pop[q] - c;  // only ever indexed at x >= c: the pull lies in the population
        }
        if (part == kStreamFaces) {
            const int sides = g.l == 2 ? 1 : 2;
            const int64_t threads = (int64_t)sides * g.m * g.n;
            k_stream_collide_pair_faces<S><<<(unsigned)((threads + 127) / 128), 128, 0, to.st>>>(src, dst, g, ph, pb,
                                                                                             sides);
            return true;
        }
        // all pairs, or all but the first and last of each row
        const int p0 = part == kStreamInterior ? 1 : 0;
        const int np = part == kStreamInterior ? g.l / 2 - 2 : g.l / 2;
        if (np <= 0) return true;
        dim3 grid((np + bx - 1) / bx, g.m, g.n);
        // resident blocks of 128 threads per SM the register budget is sized for: by default
        // 6 (80 registers) for FP32 storage, 8 (64) for 16-bit storage, whose loads need fewer
        const int minb = occ > 0 ? occ + 3 : (sizeof(S) == 4 ? 6 : 8);
        auto run = [&](auto down) {
            constexpr bool D = decltype(down)::value;
            switch (minb) {
                case 4: launch(k_stream_collide_pair<S, 4, D>, grid, bx, to, src, dst, g, ph, pb, p0, np); break;
                case 5: launch(k_stream_collide_pair<S, 5, D>, grid, bx, to, src, dst, g, ph, pb, p0, np); break;
                case 6: launch(k_stream_collide_pair<S, 6, D>, grid, bx, to, src, dst, g, ph, pb, p0, np); break;
                case 7: launch(k_stream_collide_pair<S, 7, D>, grid, bx, to, src, dst, g, ph, pb, p0, np); break;
                default: launch(k_stream_collide_pair<S, 8, D>, grid, bx, to, src, dst, g, ph, pb, p0, np); break;
            }
        };
        if (sweep_down(src, dst, g)) run(std::true_type());
        else run(std::false_type());
        return true;
    }
}

// ---------------------------------------------------------------------------
// Vectorised variant: each thread owns VW consecutive x-nodes of one (j,k)
// row, so every population moves as one 16-byte (or 8-byte) load and store.
// Pulls along x (cx = +-1) need one element of the neighbouring thread's
// vector: it comes from the adjacent lane by warp shuffle; lane 31/0 read it
// from global memory (an L2 hit: the neighbouring warp loads the same line),
// and the first/last thread of a row reads the x halo of the source row from
// the halo shell.  Rows on the y/z boundary planes pull through the shell
// node by node.  Requires l % (32*VW) == 0 and blockDim.x % 32 == 0, so a warp
// never spans two rows and every branch below is warp-uniform.
// ---------------------------------------------------------------------------
template <int BYTES> struct RawVec;
template <> struct RawVec<16> { using T = uint4; };
template <> struct RawVec<8> { using T = uint2; };

template <typename S, int VW>
struct Pack {
    using T = typename RawVec<sizeof(S) * VW>::T;
    union {
        T raw;
        S s[VW];
    };
};

template <typename S, int VW>
__device__ __forceinline__ void ld_pack(Pack<S, VW>& p, const S* ptr) {
    p.raw = __ldg(reinterpret_cast<const typename Pack<S, VW>::T*>(ptr));
}
template <typename S, int VW>
__device__ __forceinline__ void st_pack(S* ptr, const Pack<S, VW>& p) {
    *reinterpret_cast<typename Pack<S, VW>::T*>(ptr) = p.raw;
}

template <typename S, typename R, int VW>
__global__ void __launch_bounds__(256) k_stream_collide_vec(Lat<S, R> src, Lat<S, R> dst, Geo g, Phys<R> ph) {
    using K = KOps<S, R>;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;  // vector index within the row
    const int j = blockIdx.y * blockDim.y + threadIdx.y + 1;
    const int k = blockIdx.z + 1;
    if (j > g.m) return;  // whole warps only
    const int nvec = g.l / VW;
    const int lane = threadIdx.x & 31;
    const int i0 = t * VW + 1;
    const int64_t row = (int64_t)(j - 1) * g.l + (int64_t)(k - 1) * g.lm;
    const bool face = (j == 1) | (j == g.m) | (k == 1) | (k == g.n);

    Pack<S, VW> in[19];
    R edge[19];  // x-neighbour element for cx = +1 (left) and cx = -1 (right) populations
    if (!face) {
        // 1) every vector load of the node group first, so all 19 are in flight together
#pragma unroll
        for (int q = 0; q < 19; ++q) {
            const int cy = (q == 18) ? 0 : cy_of(q), cz = (q == 18) ? 0 : cz_of(q);
            ld_pack<S, VW>(in[q], src.pop[q] + row - (int64_t)cy * g.l - (int64_t)cz * g.lm + (int64_t)t * VW);
        }
        // 2) the edge elements this lane cannot get from a neighbour lane: predicated
        //    loads from the row (lanes 0/31) or from the x halo (row ends)
        const bool lo_row = (t == 0), hi_row = (t == nvec - 1);
        const bool lo_glob = (lane == 0) && !lo_row, hi_glob = (lane == 31) && !hi_row;
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            if (cx_of(q) == 0) continue;
            const S* rp = src.pop[q] + row - (int64_t)cy_of(q) * g.l - (int64_t)cz_of(q) * g.lm;
            R e = R(0);
            if (cx_of(q) == 1) {
                if (lo_glob) e = K::val(__ldg(rp + (int64_t)t * VW - 1), q, src);
                if (lo_row) e = K::from_shell(src.ghost[(int64_t)q * g.G + g.gidx(0, j - cy_of(q), k - cz_of(q))], q, src);
            } else {
                if (hi_glob) e = K::val(__ldg(rp + (int64_t)t * VW + VW), q, src);
                if (hi_row)
                    e = K::from_shell(src.ghost[(int64_t)q * g.G + g.gidx(g.l + 1, j - cy_of(q), k - cz_of(q))], q, src);
            }
            edge[q] = e;
        }
        // 3) neighbour-lane elements by shuffle
#pragma unroll
        for (int q = 0; q < 18; ++q) {
            if (cx_of(q) == 1) {
                const R e = __shfl_up_sync(0xffffffffu, K::val(in[q].s[VW - 1], q, src), 1);
                if (!lo_glob && !lo_row) edge[q] = e;
            } else if (cx_of(q) == -1) {
                const R e = __shfl_down_sync(0xffffffffu, K::val(in[q].s[0], q, src), 1);
                if (!hi_glob && !hi_row) edge[q] = e;
            }
        }
    }

    Pack<S, VW> out[19];
#pragma unroll
    for (int e = 0; e < VW; ++e) {
        R x[19];
        if (!face) {
#pragma unroll
            for (int q = 0; q < 19; ++q) {
                const int c = (q == 18) ? 0 : cx_of(q);
                if (c == 0) x[q] = K::val(in[q].s[e], q, src);
                else if (c == 1) x[q] = (e == 0) ? edge[q] : K::val(in[q].s[e - 1], q, src);
                else x[q] = (e == VW - 1) ? edge[q] : K::val(in[q].s[e + 1], q, src);
            }
        } else {
            const int i = i0 + e;
#pragma unroll
            for (int q = 0; q < 18; ++q) x[q] = K::pull(src, g, q, i - cx_of(q), j - cy_of(q), k - cz_of(q));
            x[18] = K::val(src.pop[18][row + i - 1], 18, src);
        }
        K::collide_node(x, ph, src);
#pragma unroll
        for (int q = 0; q < 19; ++q) out[q].s[e] = K::store(x[q], q, dst);
        if ((e == 0 && t == 0) || (e == VW - 1 && t == nvec - 1)) {  // x = 1 or x = l column
            const int side = (e == 0 && t == 0) ? 0 : 1;
#pragma unroll
            for (int q = 0; q < 18; ++q)
                dst.xface[xface_idx(g, side, q, j, k)] = Store<S, R>::load(out[q].s[e], q, dst.inv_scale);
        }
    }
#pragma unroll
    for (int q = 0; q < 19; ++q) st_pack<S, VW>(dst.pop[q] + row + (int64_t)t * VW, out[q]);
}

// Nodes per thread of the vector kernels: 16-byte vectors (4 FP32, 2 FP64,
// 8 FP16/BF16) or 8-byte vectors (half that).
template <typename S> struct VecWidth { static constexpr int value = 16 / sizeof(S); };

template <typename S, typename R, int VW>
bool launch_vec(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g, const Phys<R>& ph, cudaStream_t st) {
    if (g.l % (32 * VW) != 0) return false;
    for (int q = 0; q < Q; ++q)  // every row must start on a vector boundary
        if (reinterpret_cast<uintptr_t>(src.pop[q]) % (sizeof(S) * VW) != 0 ||
            reinterpret_cast<uintptr_t>(dst.pop[q]) % (sizeof(S) * VW) != 0)
            return false;
    const int nvec = g.l / VW;
    int tx = nvec;
    while (tx > 256) tx /= 2;  // nvec is a multiple of 32; keep tx a multiple of 32 dividing nvec
    if (tx % 32 != 0 || nvec % tx != 0) tx = 32;
    const int ty = (256 / tx) > 0 ? 256 / tx : 1;
    dim3 block(tx, ty, 1);
    dim3 grid(nvec / tx, (g.m + ty - 1) / ty, g.n);
    k_stream_collide_vec<S, R, VW><<<grid, block, 0, st>>>(src, dst, g, ph);
    return true;
}

}  // namespace

template <typename S, typename R>
void launch_stream_collide(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g, const Phys<R>& ph,
                           int variant, const LaunchTo& to, int part) {
    const cudaStream_t st = to.st;
    // EUP_STEP_VARIANT bit 0: 16-byte vectors, bit 2: 8-byte vectors (when l allows), bit 3: one
    // node per thread, bits 4-6: occupancy target of the two-node kernel (n + 3 blocks per SM);
    // default: two nodes per thread (FP32 arithmetic, l even).  (Bit 12 concerns the halo: all
    // blocks in one launch instead of one launch per block.)  A split step (interior columns,
    // then the two x-face columns) uses the two-node or the one-node kernel.
    constexpr int VW = VecWidth<S>::value;
    if (part == kStreamAll) {
        if ((variant & 1) && launch_vec<S, R, VW>(src, dst, g, ph, st)) return;
        if ((variant & 4) && launch_vec<S, R, (VW / 2 > 0 ? VW / 2 : 1)>(src, dst, g, ph, st)) return;
    }
    if (!(variant & 8) && launch_pair<S, R>(src, dst, g, ph, (variant >> 4) & 7, part, to)) return;
    const int bx = 128;
    if (part == kStreamFaces) {
        const int sides = g.l == 1 ? 1 : 2;
        const int64_t threads = (int64_t)sides * g.m * g.n;
        k_stream_collide_scalar_faces<S, R><<<(unsigned)((threads + bx - 1) / bx), bx, 0, st>>>(src, dst, g, ph, sides);
        return;
    }
    const int i0 = part == kStreamInterior ? 2 : 1;
    const int ni = part == kStreamInterior ? g.l - 2 : g.l;
    if (ni <= 0) return;
    dim3 grid((ni + bx - 1) / bx, g.m, g.n);
    if (sweep_down(src, dst, g)) launch(k_stream_collide_scalar<S, R, true>, grid, bx, to, src, dst, g, ph, i0, ni);
    else launch(k_stream_collide_scalar<S, R, false>, grid, bx, to, src, dst, g, ph, i0, ni);
}

template <typename S, typename R>
void launch_pbb_whole(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g, const Phys<R>& ph, const R* ns,
                      const Reduce& red, double* series, int64_t cap, int64_t* d_itime, const LaunchTo& to) {
    const PbbSplit s = pbb_split(g.l, g.m * g.n, series ? red.max_blocks : 0);
    launch(k_pbb_whole<S, R>, (unsigned)s.blocks(), s.threads, to, src, dst, g, ph, ns, s.nbx, s.each,
           (int)sweep_down(src, dst, g), red, series, cap, d_itime);
}

#define EUP_PBB_WHOLE(S, R)                                                                                     \
    template void launch_pbb_whole<S, R>(const Lat<S, R>&, const Lat<S, R>&, const Geo&, const Phys<R>&,          \
                                         const R*, const Reduce&, double*, int64_t, int64_t*, const LaunchTo&);
EUP_PBB_WHOLE(float, float)
EUP_PBB_WHOLE(double, double)
EUP_PBB_WHOLE(__half, float)
EUP_PBB_WHOLE(__nv_bfloat16, float)

template void launch_stream_collide<float, float>(const Lat<float, float>&, const Lat<float, float>&,
                                                  const Geo&, const Phys<float>&, int, const LaunchTo&, int);
template void launch_stream_collide<double, double>(const Lat<double, double>&, const Lat<double, double>&,
                                                    const Geo&, const Phys<double>&, int, const LaunchTo&, int);
template void launch_stream_collide<__half, float>(const Lat<__half, float>&, const Lat<__half, float>&,
                                                   const Geo&, const Phys<float>&, int, const LaunchTo&, int);
template void launch_stream_collide<__nv_bfloat16, float>(const Lat<__nv_bfloat16, float>&,
                                                          const Lat<__nv_bfloat16, float>&, const Geo&,
                                                          const Phys<float>&, int, const LaunchTo&, int);

}  // namespace eup
