// Transpose of the halo planes for the adjoint step: which halo slots hold a copy of which
// interior population, and which an outflow equilibrium of which node, grouped by source.
//
// The halo plan (halo_plan.cu) already says where every halo value of a step comes from, so one
// thread per planned store emits its (source, slot) pair if an interior node pulls the slot, and
// two stable radix sorts, by slot and then by source, put the pairs in the order the adjoint sums
// them in.  (The host ran the reference's halo blocks on symbols over the whole shell, searched
// all nodes for pulled halo slots and sorted: 3.6 ms at 48x24x12, 119 ms at 192x96x96, 10 s at
// 1024x512x512; an adjoint of 400 steps at 192x96x96 takes 138 ms on the device.)
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_run_length_encode.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/transform_iterator.h>

#include "halo.h"
#include "internal.h"

namespace eup {

namespace {

constexpr uint64_t kNone = ~0ull;  // no pair: sorts behind every source

struct Faces {
    int n;
    HaloFace f[6];
    int block[6];
    int64_t first[7];  // first item of each face (five per face node)
    int64_t nedges;
    const HaloEdge* edges;
};

// Item t as (source, slot): copies into key_c, outflow values into key_o; the other gets none.
__global__ void k_emit(Geo g, Faces p, int64_t items, uint64_t* key_c, uint64_t* key_o, uint64_t* slot,
                       unsigned long long* counts) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    unsigned is_c = 0, is_o = 0;
    if (t < items) {
        uint64_t kc = kNone, ko = kNone;
        int64_t s = 0;
        int kind = kEdgeConst, q_src = 0;
        int64_t src = 0;
        bool there = false;
        if (t < p.first[p.n]) {
            int f = 0;
            while (t >= p.first[f + 1]) ++f;
            const HaloFace& F = p.f[f];
            const int64_t nodes = (int64_t)F.na * F.nb, r = t - p.first[f];
            const int c = (int)(r / nodes);
            const int a = (int)((r - c * nodes) % F.na), b = (int)((r - c * nodes) / F.na);
            there = a + F.da[c] >= 0 && a + F.da[c] < F.na && b + F.db[c] >= 0 && b + F.db[c] < F.nb;
            s = F.dst[c] + a + b * F.dst_b;
            if (F.kind == kFaceOutflow) {
                kind = kEdgeOutflow;
                q_src = c;
                src = a + (int64_t)b * g.m;
            } else if (F.kind != kFaceConst) {
                kind = kEdgeCopy;
                q_src = F.src_q[c];
                src = F.lin[c] + a * F.lin_a + b * F.lin_b;
            }
        } else {
            const HaloEdge e = p.edges[t - p.first[p.n]];
            there = true;
            s = e.dst;
            kind = e.kind;
            q_src = e.q;
            src = e.src;
        }
        const int q = (int)(s / g.G);
        if (there) {  // pulled by an interior node?
            int i, j, k;
            g.shell_node(s - (int64_t)q * g.G, &i, &j, &k);
            there = g.interior(i + cx_of(q), j + cy_of(q), k + cz_of(q));
        }
        if (there && kind <= kEdgeCopyMinus) kc = (uint64_t)q_src << 32 | (uint64_t)src;
        // the population produced: the free-slip rim moves it to another population's slot
        if (there && kind == kEdgeOutflow) ko = (uint64_t)src << 5 | (uint64_t)(9 + q_src);
        key_c[t] = kc;
        key_o[t] = ko;
        slot[t] = (uint64_t)s;
        is_c = kc != kNone;
        is_o = ko != kNone;
    }
    is_c = __reduce_add_sync(0xffffffffu, is_c);
    is_o = __reduce_add_sync(0xffffffffu, is_o);
    if ((threadIdx.x & 31) == 0) {
        if (is_c) atomicAdd(counts, (unsigned long long)is_c);
        if (is_o) atomicAdd(counts + 1, (unsigned long long)is_o);
    }
}

struct RowOf {  // of an outflow key
    __host__ __device__ int32_t operator()(uint64_t key) const { return (int32_t)(key >> 5); }
};
__global__ void k_outflow_q(const uint64_t* key, int64_t n, int8_t* q) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) q[t] = (int8_t)(key[t] & 31u);
}
// CSR starts end with the number of entries.
__global__ void k_close_csr(int32_t* start, const int* runs, int32_t n) { start[*runs] = n; }

int bits_of(uint64_t v) {
    int b = 1;
    while (v >>= 1) ++b;
    return b;
}

size_t align(size_t n) { return (n + 255) / 256 * 256; }

}  // namespace

cudaError_t build_halo_adjoint(const Geo& g, const int bc[6], const HaloEdgesDevice& edges, HaloAdjointDevice* out,
                               std::string* err, cudaStream_t st) {
    *out = HaloAdjointDevice{};
    err->clear();
    Faces p{};
    for (int b = 0; b < kHaloBlocks; ++b) {
        const HaloFace f = record_halo_face(g, bc, b);
        if (f.kind == kFaceNone) continue;
        if (f.pass >= 0) {  // the up block reads what this face replaces
            *err = "the adjoint needs every halo value of a step to follow from the state entering it; "
                   "with these boundary flags a halo block reads a value written one step earlier";
            return cudaSuccess;
        }
        p.f[p.n] = f;
        p.first[p.n + 1] = p.first[p.n] + 5 * (int64_t)f.na * f.nb;
        ++p.n;
    }
    p.nedges = edges.first[kHaloBlocks];
    p.edges = edges.e;
    const int64_t items = p.first[p.n] + p.nedges;
    if (items > 2147483647LL) return cudaErrorInvalidValue;
    const int n = (int)items;
    const int slot_bits = bits_of((uint64_t)Q * (uint64_t)g.G);

    // scratch: two key arrays, the slots, two sort outputs, the counts, CUB's own
    size_t tmp_bytes = 0, need = 0;
    cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, (uint64_t*)nullptr, (uint64_t*)nullptr,
                                                    (uint64_t*)nullptr, (uint64_t*)nullptr, n, 0, 64, st);
    if (e == cudaSuccess)
        e = cub::DeviceRunLengthEncode::Encode(nullptr, need, (uint64_t*)nullptr, (uint64_t*)nullptr, (int*)nullptr,
                                               (int*)nullptr, n, st);
    tmp_bytes = std::max(tmp_bytes, need);
    if (e == cudaSuccess)
        e = cub::DeviceScan::ExclusiveSum(nullptr, need, (int*)nullptr, (int32_t*)nullptr, n, st);
    tmp_bytes = std::max(tmp_bytes, need);
    if (e != cudaSuccess) return e;
    tmp_bytes += (size_t)1 << 16;  // for the encoding over an iterator, not queried above
    const size_t arr = align(sizeof(uint64_t) * (size_t)n);
    char* scratch = nullptr;
    if ((e = cudaMalloc(&scratch, 7 * arr + align(tmp_bytes) + 256)) != cudaSuccess) return e;
    uint64_t* key_c = reinterpret_cast<uint64_t*>(scratch);
    uint64_t* key_o = reinterpret_cast<uint64_t*>(scratch + arr);
    uint64_t* slot = reinterpret_cast<uint64_t*>(scratch + 2 * arr);
    uint64_t* key1 = reinterpret_cast<uint64_t*>(scratch + 3 * arr);   // by slot
    uint64_t* slot1 = reinterpret_cast<uint64_t*>(scratch + 4 * arr);
    uint64_t* key2 = reinterpret_cast<uint64_t*>(scratch + 5 * arr);   // then by source
    uint64_t* slot2 = reinterpret_cast<uint64_t*>(scratch + 6 * arr);
    void* tmp = scratch + 7 * arr;
    unsigned long long* counts = reinterpret_cast<unsigned long long*>(scratch + 7 * arr + align(tmp_bytes));
    int* runs = reinterpret_cast<int*>(counts + 2);

    unsigned long long cnt[2] = {0, 0};
    e = cudaMemsetAsync(counts, 0, sizeof(cnt), st);
    if (e == cudaSuccess && n > 0) {
        k_emit<<<(unsigned)((items + 255) / 256), 256, 0, st>>>(g, p, items, key_c, key_o, slot, counts);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(cnt, counts, sizeof(cnt), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    const size_t nc = (size_t)cnt[0], no = (size_t)cnt[1];
    // the tables: at most as many groups as entries
    const size_t o_cslot = align(sizeof(int64_t) * nc), o_cstart = o_cslot + align(sizeof(int64_t) * nc),
                 o_oslot = o_cstart + align(sizeof(int32_t) * (nc + 1)), o_ojk = o_oslot + align(sizeof(int64_t) * no),
                 o_ostart = o_ojk + align(sizeof(int32_t) * no), o_oq = o_ostart + align(sizeof(int32_t) * (no + 1)),
                 bytes = o_oq + align(no) + 256;
    char* mem = nullptr;
    if (e == cudaSuccess) e = cudaMalloc(&mem, bytes);
    if (e == cudaSuccess) {
        out->memory = mem;
        out->copy_key = reinterpret_cast<int64_t*>(mem);
        out->copy_slot = reinterpret_cast<int64_t*>(mem + o_cslot);
        out->copy_start = reinterpret_cast<int32_t*>(mem + o_cstart);
        out->out_slot = reinterpret_cast<int64_t*>(mem + o_oslot);
        out->out_jk = reinterpret_cast<int32_t*>(mem + o_ojk);
        out->out_start = reinterpret_cast<int32_t*>(mem + o_ostart);
        out->out_q = reinterpret_cast<int8_t*>(mem + o_oq);
    }
    auto sorted = [&](uint64_t* key, uint64_t max_key) {  // -> key2, slot2 (valid entries first)
        size_t b = tmp_bytes;
        cudaError_t x = cub::DeviceRadixSort::SortPairs(tmp, b, slot, slot1, key, key1, n, 0, slot_bits, st);
        b = tmp_bytes;
        // one bit more than the largest key: kNone keeps all its bits set within it
        if (x == cudaSuccess)
            x = cub::DeviceRadixSort::SortPairs(tmp, b, key1, key2, slot1, slot2, n, 0, bits_of(max_key) + 1, st);
        return x;
    };
    int h_runs[2] = {0, 0};
    int* run_len = reinterpret_cast<int*>(key1);
    if (e == cudaSuccess && nc > 0) {
        e = sorted(key_c, (uint64_t)Q << 32);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(const_cast<int64_t*>(out->copy_slot), slot2, sizeof(int64_t) * nc,
                                cudaMemcpyDeviceToDevice, st);
        size_t b = tmp_bytes;
        if (e == cudaSuccess)
            e = cub::DeviceRunLengthEncode::Encode(tmp, b, key2, reinterpret_cast<uint64_t*>(mem), run_len, runs,
                                                   (int)nc, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h_runs[0], runs, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        b = tmp_bytes;
        if (e == cudaSuccess)
            e = cub::DeviceScan::ExclusiveSum(tmp, b, run_len, const_cast<int32_t*>(out->copy_start), h_runs[0], st);
        if (e == cudaSuccess) k_close_csr<<<1, 1, 0, st>>>(const_cast<int32_t*>(out->copy_start), runs, (int32_t)nc);
    }
    if (e == cudaSuccess && no > 0) {
        e = sorted(key_o, (uint64_t)g.mn << 5 | 31u);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(const_cast<int64_t*>(out->out_slot), slot2, sizeof(int64_t) * no,
                                cudaMemcpyDeviceToDevice, st);
        if (e == cudaSuccess)
            k_outflow_q<<<(unsigned)((no + 255) / 256), 256, 0, st>>>(key2, (int64_t)no, const_cast<int8_t*>(out->out_q));
        size_t b = tmp_bytes;
        if (e == cudaSuccess)
            e = cub::DeviceRunLengthEncode::Encode(tmp, b, thrust::make_transform_iterator(key2, RowOf()),
                                                   const_cast<int32_t*>(out->out_jk), run_len, runs, (int)no, st);
        if (e == cudaSuccess) e = cudaMemcpyAsync(&h_runs[1], runs, sizeof(int), cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        b = tmp_bytes;
        if (e == cudaSuccess)
            e = cub::DeviceScan::ExclusiveSum(tmp, b, run_len, const_cast<int32_t*>(out->out_start), h_runs[1], st);
        if (e == cudaSuccess) k_close_csr<<<1, 1, 0, st>>>(const_cast<int32_t*>(out->out_start), runs, (int32_t)no);
    }
    if (e == cudaSuccess) e = cudaGetLastError();
    const cudaError_t es = cudaStreamSynchronize(st);
    if (e == cudaSuccess) e = es;
    cudaFree(scratch);
    out->ncopy = h_runs[0];
    out->nout = h_runs[1];
    if (e != cudaSuccess && mem) {
        cudaFree(mem);
        *out = HaloAdjointDevice{};
    }
    return e;
}

}  // namespace eup
