// Device side of the cell-pair layout of P1 tetrahedra (tetpair.cu), shared by the kernels on it.
#pragma once
#include <cuda_pipeline.h>

#include "domain_kernels.cuh"
#include "internal.hpp"

namespace plb {

constexpr int kPairThreads = 128;    // items (pairs or single cells) of a block at most
constexpr int kPairCells = 240;      // cells of a block at most: about 122 items
constexpr int kPairMaxNodes = 2 * kPairThreads;  // nodes of a block at most (two per thread)
constexpr int kPairSmallLd = 144;    // slots per block where all of a mesh's blocks fit (compact ones do; else
                                     // kPairMaxNodes: 35.0 and 35.1 us, see ensure_pair_layout in tetpair.cu)
constexpr uint32_t kPairShared = 0x80000000u;
constexpr uint32_t kNoNode = 0xffffffffu, kNoItem = 0xffffffffu;
constexpr int kCellBias = 0x8000;

// Per-block arrays have constant strides (LD slots per block), so their addresses need no loads.
struct PairArrays {
    const int32_t* nslots;      // [nblocks]
    const uint32_t* ids;        // [nblocks][LD] node id | kPairShared (kNoNode past the block's nodes)
    const double* coords;       // [nblocks][3][LD]
    const uint16_t* off;        // [nblocks][LD + 8] nslots + 1 incidence offsets
    const uint16_t* inc;        // [nblocks][5 * kPairThreads] staging offsets corner * 3 * threads + item
    const uint4* items;         // [nblocks][kPairThreads] (see PairPlan)
    double* partial;            // [nblocks][LD][3] deterministic partial sums
    int64_t nblocks;
};

// Shared memory for blocks of at most LD nodes: element vectors [15][threads], two node buffers
// (coordinates in FP64 and the field in T, component by component), two metadata buffers. LD is a
// compile-time multiple of 16, so a node's six values sit at constant offsets.
// W: field values per node and component (several right-hand sides).
template <int LD>
struct PairMeta {
    uint32_t ids[LD];
    uint16_t off[LD + 8];
    uint16_t inc[5 * kPairThreads];
};
template <typename T, int LD, int W = 1>
struct PairSmem {
    T E[15 * W * kPairThreads];
    struct Node {
        double x[3 * LD];
        T v[3 * W * LD];
    } node[2];
    PairMeta<LD> meta[2];
};

// This thread's slot ids of block b, and the block's slot count.
template <int LD>
PL_D void pair_load_ids(const PairArrays& A, int64_t b, uint32_t (&nd)[2], int& ns) {
    nd[0] = nd[1] = kNoNode;
    ns = 0;
    if (b >= A.nblocks) return;
    ns = A.nslots[b];
    nd[0] = A.ids[b * LD + threadIdx.x];
    if (threadIdx.x + kPairThreads < LD) nd[1] = A.ids[b * LD + threadIdx.x + kPairThreads];
}

// Asynchronous copies of block b (ids in nd and slot count ns read one block earlier): coordinates,
// ids, offsets and incidences as aligned 16-byte runs, and per node and component the W values of its
// field (one field: values 3 id + d; several: W of the row's stride, from `field` on).
template <int LD, int W, typename T, typename Smem>
PL_D void pair_stage(const T* __restrict__ field, int stride, const PairArrays& A, int64_t b, const uint32_t (&nd)[2], int ns,
                     Smem& S, int buf) {
    auto& node = S.node[buf];
    PairMeta<LD>& M = S.meta[buf];
#pragma unroll
    for (int k = 0; k < 2; ++k)
        if (nd[k] != kNoNode) {
            const T* f = field + 3 * (int64_t)(nd[k] & ~kPairShared) * stride;
#pragma unroll
            for (int d = 0; d < 3; ++d)
                __pipeline_memcpy_async(&node.v[W * (d * LD + threadIdx.x + k * kPairThreads)], f + d * stride, W * sizeof(T));
        }
    const double* x = A.coords + b * 3 * LD;
    if (2 * threadIdx.x < ns)
#pragma unroll
        for (int d = 0; d < 3; ++d) __pipeline_memcpy_async(&node.x[d * LD + 2 * threadIdx.x], x + d * LD + 2 * threadIdx.x, 16);
    if (4 * threadIdx.x < ns) __pipeline_memcpy_async(&M.ids[4 * threadIdx.x], &A.ids[b * LD + 4 * threadIdx.x], 16);
    if (8 * threadIdx.x <= ns) __pipeline_memcpy_async(&M.off[8 * threadIdx.x], &A.off[b * (LD + 8) + 8 * threadIdx.x], 16);
    if (threadIdx.x < 5 * kPairThreads / 8)
        __pipeline_memcpy_async(&M.inc[8 * threadIdx.x], &A.inc[b * 5 * kPairThreads + 8 * threadIdx.x], 16);
}

PL_D uint4 pair_load_item(const PairArrays& A, int64_t b) {
    return b < A.nblocks ? A.items[b * kPairThreads + threadIdx.x] : make_uint4(0, 0, 0, kNoItem);
}
PL_D bool pair_single(const uint4& it) { return it.z >> 16 == 0; }
// The item's per-cell inputs, on their way to L2 (cell B lies near cell A).
template <bool BF>
PL_D void pair_prefetch_cells(const DomainParams& p, const uint4& it) {
    if (it.w == kNoItem) return;
    prefetch_l2(&p.mu[it.w]);
    prefetch_l2(&p.K[it.w]);
    if (BF)
#pragma unroll
        for (int d = 0; d < 3; ++d) prefetch_l2(&p.body_force[d * p.ncells + it.w]);
}
// Per-cell inputs of the item's cells (a single cell's twice).
template <typename L>
PL_D void pair_load_cells(const DomainParams& p, const uint4& it, double (&aA)[L::size], double (&aB)[L::size]) {
    if (it.w == kNoItem) return;
    const int64_t cA = it.w, cB = pair_single(it) ? cA : cA + (int)(it.z >> 16) - kCellBias;
    L::load_cell(p, cA, aA);
    L::load_cell(p, cB, aB);
}

PL_D void cross3(const double (&a)[3], const double (&b)[3], double (&c)[3]) {
    c[0] = a[1] * b[2] - a[2] * b[1];
    c[1] = a[2] * b[0] - a[0] * b[2];
    c[2] = a[0] * b[1] - a[1] * b[0];
}

// Local nodes n0 .. n4 of an item, and the differences of their values (planes of LD) from n0's.
PL_D void pair_nodes(const uint4& it, int (&n)[5]) {
    n[0] = it.x & 0xffff, n[1] = it.x >> 16, n[2] = it.y & 0xffff, n[3] = it.y >> 16, n[4] = it.z & 0xffff;
}
template <int LD, typename T>
PL_D void pair_diffs(const int (&n)[5], const T* plane, T (&g)[4][3]) {
    T v0[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) v0[d] = plane[d * LD + n[0]];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int d = 0; d < 3; ++d) g[k][d] = plane[d * LD + n[k + 1]] - v0[d];
}

// The isotropic tangent (lambda, mu) of the item's cells (a single cell's twice): the solver's cache
// (p.lm32; CACHED) or the registered Jacobian kernel.
template <bool CACHED>
PL_D void pair_load_tangents(const DomainParams& p, const uint4& it, float2 (&lm)[2]) {
    if (it.w == kNoItem) return;
    const int64_t cells[2] = {(int64_t)it.w, pair_single(it) ? (int64_t)it.w : (int64_t)it.w + (int)(it.z >> 16) - kCellBias};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (CACHED) {
            lm[k] = reinterpret_cast<const float2*>(p.lm32)[cells[k]];
        } else {
            using L = AuxLayout<RHEO_ILE, false>;
            const AuxOffsets<RHEO_ILE, false> aoff;
            double a[L::size], x[3] = {0, 0, 0}, Jf3[81];
            L::load_cell(p, cells[k], a);
#pragma unroll
            for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
            call_jf3<RHEO_ILE>(L::numA, aoff.v, a, p, x, Jf3);
            lm[k] = make_float2((float)(-Jf3[((0 * 3 + 1) * 3 + 0) * 3 + 1]), (float)(-Jf3[((0 * 3 + 1) * 3 + 1) * 3 + 0]));
        }
    }
}

inline PairArrays pair_arrays_of(const PairLayout& L, double* partial, bool reduced) {
    PairArrays A;
    A.nslots = L.d_nslots;
    A.ids = reduced ? L.d_ids_red : L.d_ids;
    A.coords = L.d_coords;
    A.off = L.d_off;
    A.inc = L.d_inc;
    A.items = (const uint4*)L.d_items;
    A.partial = partial;
    A.nblocks = L.num_blocks;
    return A;
}

}  // namespace plb
