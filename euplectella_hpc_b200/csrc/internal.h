// Internal interfaces between the host entry points (abi.cu) and the CUDA
// kernels (k_bc.cu, k_step.cu, k_setup.cu).  Not part of the C ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>
#include <vector>

#include "lbm_common.cuh"

namespace eup {

// ---- launches of a step ------------------------------------------------------------------
// Where a kernel of a step goes.  `chained`: it may be brought onto the device while the kernel
// before it in the stream still runs (programmatic dependent launch); its threads wait in
// chain_begin until that one has completed and its stores are visible.  Every kernel of a step
// calls chain_begin before its first access, so the wait reaches back through the whole
// chain, and the launch latency of each is hidden behind the one before.  With the steps of a
// run chained too (16 to a CUDA graph), a step takes, launches in turn / chained: 64x32x8
// FP32 12.3 / 10.4 us, 256x128x64 FP32 65.9 / 61.3, FP16 48.7 / 44.6, FP64 115.1 / 111.1;
// 384x192x192 FP32 349.6 / 345.2; nothing at 768x384x384.
struct LaunchTo {
    cudaStream_t st;
    bool chained;
    LaunchTo(cudaStream_t s, bool c = false) : st(s), chained(c) {}
};

template <typename... P, typename... A>
void launch(void (*kernel)(P...), dim3 grid, dim3 block, const LaunchTo& to, const A&... args) {
    cudaLaunchConfig_t c = {};
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.gridDim = grid;
    c.blockDim = block;
    c.stream = to.st;
    c.attrs = &at;
    c.numAttrs = to.chained ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

__device__ __forceinline__ void chain_begin() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
// The same in two parts, for kernels that fetch what no kernel of a step writes (lists, indices)
// while they wait: 0.6 us of a step.  A thread with nothing to do may return between the two.
__device__ __forceinline__ void chain_open() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Bit-packed solid mask: one bit per interior node, rows along x padded to
// 32-bit words (wpr words per (j,k) row).
struct Mask {
    const uint32_t* bits;
    int wpr;
    __device__ __forceinline__ bool solid(const Geo& g, int i, int j, int k) const {
        if (bits == nullptr || !g.interior(i, j, k)) return false;
        const int64_t row = (int64_t)(j - 1) + (int64_t)g.m * (k - 1);
        return (bits[row * wpr + ((i - 1) >> 5)] >> ((i - 1) & 31)) & 1u;
    }
};

// Reduction scratch: per-block partial sums and a completion counter.  The
// last block to finish adds the partials in block order, so results do not
// depend on scheduling.
struct Reduce {
    double* partials;     // [max_blocks * width]
    unsigned int* counter;
    int max_blocks;
};

constexpr int kReduceMaxBlocks = 4096;
constexpr int kReduceWidth = 8;

// ---- block reduction into deterministic per-block partials ----------------------------
template <int W>
__device__ __forceinline__ void block_reduce_store(double (&v)[W], const Reduce& red, double* out, double* series = nullptr,
                                   int64_t cap = 0, int64_t* d_itime = nullptr, int advance = 0,
                                   int slot_offset = 0) {
    __shared__ double sh[32][W];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int c = 0; c < W; ++c)
        for (int o = 16; o > 0; o >>= 1) v[c] += __shfl_down_sync(0xffffffffu, v[c], o);
    if (lane == 0)
        for (int c = 0; c < W; ++c) sh[warp][c] = v[c];
    __syncthreads();
    if (threadIdx.x == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        for (int c = 0; c < W; ++c) {
            double s = 0.0;
            for (int w = 0; w < nw; ++w) s += sh[w][c];
            red.partials[(int64_t)blockIdx.x * W + c] = s;
        }
        __threadfence();
        const unsigned done = atomicAdd(red.counter, 1u);
        last = (done == gridDim.x - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the last block adds the partials: thread t takes blocks t, t+blockDim, ...
    // (independent loads, fixed assignment), then the same fixed tree as above
    double s[W];
#pragma unroll
    for (int c = 0; c < W; ++c) s[c] = 0.0;
    for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x)
#pragma unroll
        for (int c = 0; c < W; ++c) s[c] += __ldcg(red.partials + (int64_t)b * W + c);
#pragma unroll
    for (int c = 0; c < W; ++c)
        for (int o = 16; o > 0; o >>= 1) s[c] += __shfl_down_sync(0xffffffffu, s[c], o);
    __syncthreads();
    if (lane == 0)
        for (int c = 0; c < W; ++c) sh[warp][c] = s[c];
    __syncthreads();
    if (threadIdx.x == 0) {
        double* dst = out;
        if (series) {
            const int64_t t = *(volatile int64_t*)d_itime;
            dst = series + W * ((t + slot_offset) % cap);
            if (advance) *d_itime = t + 1;
        }
        const int nw = (blockDim.x + 31) >> 5;
        for (int c = 0; c < W; ++c) {
            double tot = 0.0;
            for (int w = 0; w < nw; ++w) tot += sh[w][c];
            dst[c] = tot;
        }
        *red.counter = 0u;
    }
}

// ---- halo planes (halo.h, halo_plan.cu) -----------------------------------------------
// One store to an edge line: ghost[dst] = a value of kind.
enum : int32_t {
    kEdgeCopy,       // population q of interior node src
    kEdgeCopyPlus,   //   ... plus the lid's force
    kEdgeCopyMinus,  //   ... minus it
    kEdgeOld,        // ghost[src], a halo value no item of a step writes
    kEdgeOutflow,    // outflow population 10 + q of row src = (j-1) + (k-1) m
    kEdgeConst       // inflow population 1 + q
};
struct HaloEdge {
    int64_t dst, src;
    int32_t q, kind;
};
// The edge stores of a step, grouped by the block that makes them (first[b] .. first[b + 1]): in
// groups of `stores` runs that take turns from `at` on, each at a constant distance from its last.
// (Run after run, the five outflow stores of a row would read its 18 x-face values in five places of
// the table: 0.9 us of a 44 us step at 256x128x64 FP16.)  Recorded item by item
// the table took 0.2 ms at 64x32x8 (free-slip y and z), 4.7 at 1024x512x512, 75 at 65536x2x2; as
// runs 0.1, 0.1, 0.03.
struct HaloEdgeRun {
    HaloEdge e;
    int64_t dst_step, src_step, at;
    int32_t stores, pad;
};
struct HaloEdges {
    std::vector<HaloEdgeRun> runs;
    int64_t first[9];
};
struct HaloEdgesDevice {
    const HaloEdge* e = nullptr;
    int64_t first[9] = {};
};
HaloEdges build_halo_edges(const Geo& g, const int bc[6], bool one_by_one = false);
// Allocates out->e (cudaFree) and fills it; synchronises st.
cudaError_t put_halo_edges(const HaloEdges& edges, HaloEdgesDevice* out, cudaStream_t st);

// One face of the halo away from the edge lines: nodes (a, b) of the face, a = 0 .. na-1 and
// b = 0 .. nb-1, a fastest.  Population t of the five goes to ghost[dst[t] + a + b dst_b] where
// (a + da, b + db) is on the face (a no-slip block stores one node along a tangential axis;
// beyond the face lies an edge line).
enum : int { kFaceNone = -1, kFaceCopy, kFaceCopyX, kFaceOutflow, kFaceConst };
struct HaloFace {
    int kind;  // copy from the lattice, from the x-face copy, outflow equilibrium, inflow constants
    int na, nb;
    int64_t src_b, dst_b;
    int q[5], src_q[5], da[5], db[5], lid[5];
    int64_t src[5], dst[5];
    int64_t lin[5], lin_a, lin_b;  // interior node copied, at (0, 0), and its strides
    int pass;          // >= 0: on row b = nb-1 the old value of population `pass` goes to pass_dst + a first
    int64_t pass_dst;
};
HaloFace record_halo_face(const Geo& g, const int bc[6], int block);

// Halo planes of one step (CODE/SRC/bcond.bc.F90) in one launch, or one launch per block of
// the reference; with `force` its sum too.  Returns the number of kernels launched.
template <typename S, typename R>
int launch_bc(const Lat<S, R>& L, const Geo& g, const int bc[6], const Phys<R>& ph, const HaloEdgesDevice& edges,
              const LaunchTo& to, bool separate = false, const struct ForceSum* force = nullptr);

// ---- bounce-back and momentum-exchange force --------------------------------------------
// The links of the solid voxels to fluid and to halo nodes, population by population (q
// outermost, voxels ascending), so that neighbouring threads read and write neighbouring
// values of one population.
struct FluidLink {
    int32_t lin;  // solid voxel
    uint32_t q;   // population 0..17, kLinkXFirst / kLinkXLast when the voxel lies on x = 1 / x = l
};
struct HaloLink {
    int32_t lin;
    uint32_t q;
    int64_t ghost;  // halo value the bounce-back reads
    int64_t wrap;   // interior fluid node beyond a periodic face, whose value enters the force; -1: none
};
constexpr uint32_t kLinkXFirst = 32u, kLinkXLast = 64u, kLinkQ = 31u;
struct LinksDevice {
    const FluidLink* fluid = nullptr;
    const HaloLink* halo = nullptr;
    int64_t nfluid = 0, nhalo = 0;
};
// Builds the links of the n boundary-solid voxels of `list`, classified by `words` (see
// launch_bsolid_links); allocates out->fluid and out->halo, synchronises st.  scratch: device
// memory to work in (256-byte aligned), more is allocated where it does not suffice.
cudaError_t build_links(const Geo& g, const int bc[6], const int32_t* list, const uint64_t* words, int64_t n,
                        LinksDevice* out, void* scratch, size_t scratch_bytes, cudaStream_t st);

// Where a sum of the force goes: series[3 * (*d_itime % cap)]; `blocks` partial sums of the
// bounce-back launch (three each, for FP64 six) are added in their order, and
// the device step counter advances.
struct ForceSum {
    const double* partials;
    int blocks;
    double* series;
    int64_t cap;
    int64_t* d_itime;
    double* host;  // the sum also goes here (page-locked host memory), if not null
};
// Bounce-back on solid voxels touching fluid/halo (CODE/SRC/bcond.obs.F90) with partial sums of
// the FP64 momentum-exchange force of the state it reads; the halo launch of the step adds
// them (launch_bc with the ForceSum returned).  No launch without links (blocks = 0).
template <typename S, typename R>
ForceSum launch_bounce(const Lat<S, R>& L, const Geo& g, const LinksDevice& links, const Reduce& red, double* series,
                       int64_t cap, int64_t* d_itime, const LaunchTo& to);
// The force alone, of the state in L, in one launch, to the history and to `host` (page-locked);
// the step counter stays.
template <typename S, typename R>
void launch_force(const Lat<S, R>& L, const Geo& g, const LinksDevice& links, const Reduce& red, double* series,
                  int64_t cap, int64_t* d_itime, double* host, cudaStream_t st);

// x-slab faces: the five populations crossing an x face, (m+2)(n+2) values each.
template <typename S, typename R>
void launch_pack_x(const Lat<S, R>& L, const Geo& g, int side, R* out, cudaStream_t st);
template <typename S, typename R>
void launch_unpack_x(const Lat<S, R>& L, const Geo& g, int side, const R* in, cudaStream_t st);
template <typename S, typename R>
void launch_pack_x_rim(const Lat<S, R>& L, const Geo& g, int sides, cudaStream_t st);
template <typename S, typename R>
void launch_unpack_x_view(const Lat<S, R>& L, const Geo& g, int side, const R* in, cudaStream_t st);

// x-face copy of the current lattice (needed once after an upload).
template <typename S, typename R>
void launch_fill_xface(const Lat<S, R>& L, const Geo& g, cudaStream_t st);

// Fused pull stream + collide (CODE/SRC/movef.F90 + CODE/SRC/col.F90): src -> dst, over
// every node (kStreamAll), or split into the columns that do not pull from the x halo
// planes (kStreamInterior) and the two that do (kStreamFaces), so that an x-slab can
// receive its halo planes while the interior streams.
enum { kStreamAll = 0, kStreamInterior = 1, kStreamFaces = 2 };
template <typename S, typename R>
void launch_stream_collide(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g,
                           const Phys<R>& ph, int variant, const LaunchTo& to, int part = kStreamAll);

// Doubles of device scratch launch_plane_means needs.
int64_t plane_means_scratch(const Geo& g, int axis);
// Reference-form diagnostics (CODE/SRC/prof_*.F90, varm.F90, flux_X/flux_Y.F90):
// a line of per-node u, w, v, den in R; per-plane means; the FP64 face sums of
// the control-volume stresses of box = {i1, i2, j1, j2, k1, k2} (already clipped).
template <typename S, typename R>
void launch_line(const Lat<S, R>& L, const Geo& g, int axis, int c1, int c2, double* out, cudaStream_t st);
template <typename S, typename R>
void launch_plane_means(const Lat<S, R>& L, const Geo& g, int axis, double* out, double* scratch, cudaStream_t st);
template <typename S, typename R>
void launch_cv_drag(const Lat<S, R>& L, const Geo& g, const int box[6], R omega, const Reduce& red, double* out,
                    cudaStream_t st);

// FP64 sums over the fluid nodes of a region (device byte mask, one per node) into out[6].
template <typename S, typename R>
void launch_region_sums(const Lat<S, R>& L, const Geo& g, const Mask& mk, const uint8_t* region, const Reduce& red,
                        double* out, cudaStream_t st);

// Population q of the seeded equilibrium initial state (init_eq.h) into a
// haloed staging array of (l+2)(m+2)(n+2) elements.
template <typename T>
void launch_init_population(T* staging, const Geo& g, int q, double u_in, double amp, uint64_t seed, cudaStream_t st);

// FP64 sums of CODE/SRC/diagno.F90 into out[5] (device pointer).
template <typename S, typename R>
void launch_monitor(const Lat<S, R>& L, const Geo& g, const Mask& mk, const Reduce& red,
                    double* out, cudaStream_t st);

// rho,u at given nodes into out[4*npts] (device pointers).
template <typename S, typename R>
void launch_probes(const Lat<S, R>& L, const Geo& g, int npts, const int32_t* ijk, double* out,
                   cudaStream_t st);

// Scatter nq haloed host-layout arrays (T), one behind the other, into lattice populations
// q .. q+nq-1 and the shell; a value that is not finite sets its population's bit of *bad
// (device pointer).
template <typename S, typename R, typename T>
void launch_scatter(const Lat<S, R>& L, const Geo& g, int q, int nq, const T* staging, unsigned int* bad,
                    cudaStream_t st);
template <typename S, typename R, typename T>
void launch_gather(const Lat<S, R>& L, const Geo& g, int q, int nq, T* staging, cudaStream_t st);

// Set-up kernels (k_setup.cu).
void launch_build_mask(const int32_t* obs, const Geo& g, uint32_t* bits, int wpr, cudaStream_t st);
// Device voxeliser (geometry.h): the bit-packed mask of shape S.
struct VoxShape;
void launch_voxelise(const Geo& g, const VoxShape& S, uint32_t* bits, int wpr, cudaStream_t st);
// out[0..2] = solid voxels, solid voxels at i = 1, at i = l.
void launch_mask_counts(const uint32_t* bits, const Geo& g, int wpr, unsigned long long* out, cudaStream_t st);
// The nsolid solid voxels of the mask, i fastest, as Fortran records [12][i][j][k][12]
// (rec holds 5 nsolid int32); synchronises st.
cudaError_t obstacle_records(const Geo& g, const Mask& mk, int64_t nsolid, int32_t* rec, cudaStream_t st);
void launch_flag_boundary_solid(const Geo& g, const Mask& mk, uint8_t* flags, cudaStream_t st);
void launch_links(const Geo& g, const Mask& mk, uint32_t* links, cudaStream_t st);
// Neighbour classification of each boundary-solid voxel: bit q (0..17) neighbour
// x + c_q is interior fluid, bit 18+q it is a halo node, bit 36+q that halo node
// wraps across a periodic axis onto interior fluid.
void launch_bsolid_links(const Geo& g, const Mask& mk, const int bc[6], const int32_t* list, int64_t n,
                         uint64_t* links, cudaStream_t st);
// Ordered compaction of flagged linear indices; returns the count (synchronous).
int64_t compact_flags(const uint8_t* flags, int64_t n, int32_t* out, void* scratch, size_t scratch_bytes,
                      cudaStream_t st, cudaError_t* err);

// ---- partial bounce-back and its adjoint (k_adjoint.cu) -------------------------
// Where the adjoint of each halo value goes, on the device.  copy_*: halo slots holding a copy of
// an interior population, grouped by source key q << 32 | lin (CSR: copy_start), ascending within a
// group.  out_*: halo slots holding an outflow equilibrium, grouped by the x = l node
// (j-1) + (k-1)*m they are computed from, with the population produced, by population and slot.
struct HaloAdjointDevice {
    const int64_t* copy_key = nullptr;
    const int32_t* copy_start = nullptr;
    const int64_t* copy_slot = nullptr;
    int64_t ncopy = 0;
    const int32_t* out_jk = nullptr;
    const int32_t* out_start = nullptr;
    const int64_t* out_slot = nullptr;
    const int8_t* out_q = nullptr;
    int64_t nout = 0;
    void* memory = nullptr;  // what the arrays lie in (cudaFree)
};
// Builds the tables from the halo plan (faces and edge table) of these flags; synchronises st.
// cudaSuccess with *err set: the flags are not supported (err says why).
cudaError_t build_halo_adjoint(const Geo& g, const int bc[6], const HaloEdgesDevice& edges, HaloAdjointDevice* out,
                               std::string* err, cudaStream_t st);

// Momentum the solid takes from a voxel of solid fraction s: 2 s j, j the momentum of the pulled
// kernel values pre (of deviations the same, sum_q c_q w_q = 0) times js, in FP64, the signed
// terms alone.
template <typename R>
__device__ __forceinline__ void pbb_momentum(const R (&pre)[19], R s, double js, double (&f)[3]) {
    double jx = 0.0, jy = 0.0, jz = 0.0;
#pragma unroll
    for (int q = 0; q < 18; ++q) {
        const double v = (double)pre[q];
        if (cx_of(q) != 0) jx = cx_of(q) > 0 ? jx + v : jx - v;
        if (cy_of(q) != 0) jy = cy_of(q) > 0 ? jy + v : jy - v;
        if (cz_of(q) != 0) jz = cz_of(q) > 0 ? jz + v : jz - v;
    }
    f[0] += 2.0 * (double)s * (jx * js);
    f[1] += 2.0 * (double)s * (jy * js);
    f[2] += 2.0 * (double)s * (jz * js);
}

// The partial-bounce-back step as one kernel over every node.
template <typename S, typename R>
void launch_pbb_whole(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g, const Phys<R>& ph, const R* ns,
                      const Reduce& red, double* series, int64_t cap, int64_t* d_itime, const LaunchTo& to);

// One partial-bounce-back step src -> dst (any storage; FP32 arithmetic for 16-bit storage):
// with `whole` in one pass over every node, else the plain stream-collide, then the mixing
// f* = (1 - n_s) BGK(f) + n_s f_opp on the ns_count voxels of ns_list (those with n_s > 0).  With `series` the FP64 force of the step goes to
// series[(itime + 1) % cap] and the device step counter advances; series == nullptr skips it
// (recomputation in the adjoint).
template <typename S, typename R>
void launch_pbb_step(const Lat<S, R>& src, const Lat<S, R>& dst, const Geo& g, const Phys<R>& ph, const R* ns,
                     const int32_t* ns_list, int64_t ns_count, bool whole, const Reduce& red, double* series,
                     int64_t cap, int64_t* d_itime, const LaunchTo& to);
// Adjoint of one partial-bounce-back step from state f (its halo shell holding the step's
// halo values); the adjoint fields lam are in the arithmetic type.  The adjoint is pushed:
// node x writes lam_out_q at the node x - c_q it pulled from, each slot once.  parts:
// kAdjInterior, the nodes 2..l-1 x 2..m-1 x 2..n-1, which read no halo value; kAdjFaces,
// the boundary-plane nodes (they read the step's halo values and write the halo part gmu);
// these two write disjoint slots and may run on different streams.  kAdjTransposes adds the
// halo adjoints back onto the interior slots they were copied from or computed from; it
// runs after both, since those slots may be ones the interior part writes.
enum { kAdjInterior = 1, kAdjFaces = 2, kAdjTransposes = 4, kAdjAll = 7 };
template <typename S, typename R>
void launch_pbb_adjoint(const Lat<S, R>& f, const Geo& g, const Phys<R>& ph, const R* ns, const Lat<R, R>& lam_in,
                        const Lat<R, R>& lam_out, R* gmu, double* grad, R gamma, const HaloAdjointDevice& t,
                        cudaStream_t st, int parts = kAdjAll);

}  // namespace eup
