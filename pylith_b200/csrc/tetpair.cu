// P1 tetrahedra, residual and Jacobian actions: cell blocks of face-sharing pairs.
//
// As in blocked.cu a persistent CTA takes compact blocks of consecutive cells, stages the block's
// nodes (coordinates and field) in shared memory one block ahead, forms element vectors in one phase
// and sums them per node in the next; owned nodes are stored, shared ones reduced into the output.
// That scheme is bound by shared-memory traffic: a cell reads 24 node values and its 12-entry element
// vector is written and read again. Here a thread takes two tetrahedra that share a face: 30 node
// values, 15 entries, five incidences for the pair, 60 % of the traffic, and the shared edges and
// cross product are formed once. The host matches the cells of a block into pairs (98 % of them on
// Delaunay and structured meshes); a cell left over takes a thread by itself.
//
// Bound: shared memory still (79 % of its pipe on 1,218,746 cells), then HBM. Measured on B200 against the
// one-cell-per-thread kernel k_tet_pad2, residual or action, L2 warm: 1,296,000 structured cells FP64 53.8 ->
// 42.3 us and FP32 45.8 -> 33.3; 54,737 Delaunay cells FP64 9.5 -> 8.9, FP32 9.9 -> 8.7; 3,072 cells FP64 8.5
// -> 6.8. INSERT applications also start under their output's zeroing (zero_output).
//
// Sizes of a block: 240 cells in 128 items (threads), 4 CTAs per SM in FP64 (at most 128 registers), 6 in
// FP32. Others, residual and action of 1,179,648 cells, 80 us this way before the banks were planned by
// half-warps: 5 and 6 CTAs 80 to 92 (spills); 64, 96, 192 and 256 threads 82 to 98; two lanes per node in the
// sums 89. FP32 with 4, 5 and 6 CTAs: 45.6, 40.1 and 38.6 us.
#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <queue>
#include <thread>
#include <vector>

#include "bankplan.hpp"
#include "launch.hpp"
#include "tetpair.cuh"

namespace plb {

constexpr int kPairCtas = 4;    // resident CTAs per SM
constexpr int kPairCtas32 = 6;  // of the FP32 action

// One tetrahedron from its cofactor rows c0, c1, c2 (det J times the basis gradients of its corners
// 1, 2, 3), det and the field differences g0, g1, g2 of those corners: v[k] = |K| f1 . grad(phi_{k+1})
// (f1 C^T / 6), and, for the body force, bfw f0 (|K| / 4 times f0) in w.
template <int RHEO, bool BF, int OP>
PL_D void pair_tet(const DomainParams& p, const double* a, const double (&c0)[3], const double (&c1)[3], const double (&c2)[3],
                   double det, const double (&g0)[3], const double (&g1)[3], const double (&g2)[3], double (&v)[3][3],
                   double (&w)[3]) {
    using L = AuxLayout<RHEO, BF>;
    const AuxOffsets<RHEO, BF> aoff;
    if (!(det > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
    const double rdet = 1.0 / det;
    double s_x[9], x[3] = {0, 0, 0}, s[3] = {0, 0, 0};
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) s_x[c * 3 + d] = (g0[c] * c0[d] + g1[c] * c1[d] + g2[c] * c2[d]) * rdet;
    double f0[3] = {0, 0, 0}, f1[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const double sixth = 1.0 / 6.0;
    if (OP == OP_RESIDUAL) {
        if (BF) {
            const int sOff[1] = {0}, sOff_x[1] = {0};
            pw::g0v_bodyforce<double>(3, 1, L::numA, sOff, sOff_x, s, nullptr, s_x, aoff.v, nullptr, a, nullptr, nullptr, p.t, x,
                                      p.num_constants, p.constants, f0);
            const double bfw = det * sixth * 0.25;
#pragma unroll
            for (int c = 0; c < 3; ++c) w[c] = bfw * f0[c];
        }
        call_f1<RHEO>(L::numA, aoff.v, a, s, s_x, p, x, f1);
    } else {
        double Jf3[81];
#pragma unroll
        for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
        call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
        isotropic_jf3_contract<RHEO>(Jf3, s_x, f1);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        v[0][c] = (f1[3 * c] * c0[0] + f1[3 * c + 1] * c0[1] + f1[3 * c + 2] * c0[2]) * sixth;
        v[1][c] = (f1[3 * c] * c1[0] + f1[3 * c + 1] * c1[1] + f1[3 * c + 2] * c1[2]) * sixth;
        v[2][c] = (f1[3 * c] * c2[0] + f1[3 * c + 1] * c2[1] + f1[3 * c + 2] * c2[2]) * sixth;
    }
}

// The element vectors of one item into column E: tetrahedra (n0, n1, n2, n3) and, unless single,
// (n0, n2, n1, n4).
template <int RHEO, bool BF, int OP, int LD>
PL_D void pair_item(const DomainParams& p, const uint4& it, const double* aA, const double* aB,
                    const typename PairSmem<double, LD>::Node& node, double* E) {
    int n[5];
    double e[4][3], g[4][3];
    pair_nodes(it, n);
    pair_diffs<LD>(n, node.x, e);
    pair_diffs<LD>(n, node.v, g);
    double n12[3], c0[3], c1[3], v[3][3], w[3] = {0, 0, 0}, r0[3], r1[3], r2[3];
    cross3(e[0], e[1], n12);
    cross3(e[1], e[2], c0);
    cross3(e[2], e[0], c1);
    double det = e[0][0] * c0[0] + e[0][1] * c0[1] + e[0][2] * c0[2];
    pair_tet<RHEO, BF, OP>(p, aA, c0, c1, n12, det, g[0], g[1], g[2], v, w);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        r0[c] = w[c] - (v[0][c] + v[1][c] + v[2][c]);
        r1[c] = v[0][c] + w[c];
        r2[c] = v[1][c] + w[c];
        E[(9 + c) * kPairThreads] = v[2][c] + w[c];
    }
    if (!pair_single(it)) {
        double m[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) m[c] = -n12[c];
        cross3(e[0], e[3], c0);  // of corner n2
        cross3(e[3], e[1], c1);  // of corner n1
        det = e[1][0] * c0[0] + e[1][1] * c0[1] + e[1][2] * c0[2];
        pair_tet<RHEO, BF, OP>(p, aB, c0, c1, m, det, g[1], g[0], g[3], v, w);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            r0[c] += w[c] - (v[0][c] + v[1][c] + v[2][c]);
            r2[c] += v[0][c] + w[c];
            r1[c] += v[1][c] + w[c];
            E[(12 + c) * kPairThreads] = v[2][c] + w[c];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        E[c * kPairThreads] = r0[c];
        E[(3 + c) * kPairThreads] = r1[c];
        E[(6 + c) * kPairThreads] = r2[c];
    }
}

// One node's sum over its incidences j0 <= j < j1 of the staged element vectors.
template <typename T>
PL_D void pair_node_sum(const T* E, const uint16_t* inc, int j0, int j1, T (&r)[3]) {
    r[0] = r[1] = r[2] = T(0);
#pragma unroll 4
    for (int j = j0; j < j1; ++j) {
        const T* e = E + inc[j];
        r[0] += e[0];
        r[1] += e[kPairThreads];
        r[2] += e[2 * kPairThreads];
    }
}

// DET: a shared node's block sum goes to the partial-sum buffer for the fixup pass (bit-identical
// results run to run); otherwise it is added into the output with an FP64 reduction (the output was
// zeroed first for INSERT).
template <int RHEO, bool BF, int OP, bool INSERT, bool DET, int LD>
__global__ void __launch_bounds__(kPairThreads, kPairCtas) k_tet_pair(DomainParams p, PairArrays A) {
    using L = AuxLayout<RHEO, BF>;
    extern __shared__ __align__(16) char smem_raw[];
    PairSmem<double, LD>& S = *reinterpret_cast<PairSmem<double, LD>*>(smem_raw);
    const double* __restrict__ field = OP == OP_RESIDUAL ? p.u : p.v;
    const int64_t G = gridDim.x;
    int64_t b = blockIdx.x;
    if (b >= A.nblocks) return;
    uint32_t nd_next[2];
    int ns, ns_next;
    uint4 item = pair_load_item(A, b), item_next = pair_load_item(A, b + G);
    double aA[L::size], aB[L::size];
    {
        uint32_t nd0[2];
        pair_load_ids<LD>(A, b, nd0, ns);
        pair_stage<LD, 1>(field, 1, A, b, nd0, ns, S, 0);
        __pipeline_commit();
        pair_load_ids<LD>(A, b + G, nd_next, ns_next);
        pair_load_cells<L>(p, item, aA, aB);
        pair_prefetch_cells<BF>(p, item_next);
    }
    for (int it = 0; b < A.nblocks; b += G, ++it) {
        // what the next blocks need, so that no load of the loop waits for another or for HBM: the slot
        // ids and the item two blocks ahead (its cells' inputs then start for L2, and are read between
        // the two phases of the block before)
        uint32_t nd_after[2];
        int ns_after;
        pair_load_ids<LD>(A, b + 2 * G, nd_after, ns_after);
        const uint4 item_after = pair_load_item(A, b + 2 * G);
        __pipeline_wait_prior(0);
        // block b's copies have landed; every thread has finished the node sums of the previous block
        // (its buffers are free for block b + G)
        __syncthreads();
        if (b + G < A.nblocks) pair_stage<LD, 1>(field, 1, A, b + G, nd_next, ns_next, S, (it + 1) & 1);
        __pipeline_commit();
        nd_next[0] = nd_after[0], nd_next[1] = nd_after[1];
        if (item.w != kNoItem) pair_item<RHEO, BF, OP, LD>(p, item, aA, aB, S.node[it & 1], S.E + threadIdx.x);
        item = item_next, item_next = item_after;
        pair_load_cells<L>(p, item, aA, aB);
        pair_prefetch_cells<BF>(p, item_next);
        __syncthreads();
        wait_for_previous();
        const auto& M = S.meta[it & 1];
        for (int k = threadIdx.x; k < ns; k += kPairThreads) {
            const uint32_t id = M.ids[k];
            double* o = p.out + 3 * (int64_t)(id & ~kPairShared);
            double* pp = DET ? A.partial + 3 * (b * LD + k) : nullptr;
            double r[3], old[3] = {0.0, 0.0, 0.0};
            if (!INSERT && !(id & kPairShared))  // on its way while the sum runs (1 us of a 10 us launch)
#pragma unroll
                for (int d = 0; d < 3; ++d) old[d] = o[d];
            pair_node_sum(S.E, M.inc, M.off[k], M.off[k + 1], r);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if ((id & kPairShared) && DET) pp[d] = r[d];
                else if (id & kPairShared) red_add(o + d, r[d]);
                else o[d] = INSERT ? r[d] : old[d] + r[d];
            }
        }
        ns = ns_next, ns_next = ns_after;
    }
    __pipeline_wait_prior(0);
}

// ---- FP32 Jacobian action --------------------------------------------------------------------
// pair_tet of the FP32 action: cofactors and det in FP64, gradient, flux and vectors in FP32.
PL_D void pair_tet32(const DomainParams& p, float2 lm, const double (&c0)[3], const double (&c1)[3], const double (&c2)[3],
                     double det, const float (&g0)[3], const float (&g1)[3], const float (&g2)[3], float (&v)[3][3]) {
    if (!(det > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
    const double rdet = 1.0 / det;
    float inv[3][3], cf[3][3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
        inv[0][j] = (float)(c0[j] * rdet), cf[0][j] = (float)(c0[j] * (1.0 / 6.0));
        inv[1][j] = (float)(c1[j] * rdet), cf[1][j] = (float)(c1[j] * (1.0 / 6.0));
        inv[2][j] = (float)(c2[j] * rdet), cf[2][j] = (float)(c2[j] * (1.0 / 6.0));
    }
    float s[3][3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) s[c][d] = g0[c] * inv[0][d] + g1[c] * inv[1][d] + g2[c] * inv[2][d];
    // flux f1 = -(lambda tr(e) I + 2 mu e), e = sym grad v
    const float mu = lm.y, ltr = lm.x * (s[0][0] + s[1][1] + s[2][2]);
    const float xy = -mu * (s[0][1] + s[1][0]), yz = -mu * (s[1][2] + s[2][1]), xz = -mu * (s[0][2] + s[2][0]);
    const float f[3][3] = {{-(2.0f * mu * s[0][0] + ltr), xy, xz},
                           {xy, -(2.0f * mu * s[1][1] + ltr), yz},
                           {xz, yz, -(2.0f * mu * s[2][2] + ltr)}};
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int c = 0; c < 3; ++c) v[k][c] = f[c][0] * cf[k][0] + f[c][1] * cf[k][1] + f[c][2] * cf[k][2];
}

// FP32 Jacobian action of an isotropic tangent on the pairs (measured: head of the file), for the inner iterations of the
// mixed-precision solvers: as k_tet_pair, with FP64 geometry and FP32 field, flux, element vectors
// and sums. The output holds zero or the sum to add to.
template <bool CACHED, int LD>
__global__ void __launch_bounds__(kPairThreads, kPairCtas32) k_tet_pair_jv32(DomainParams p, PairArrays A) {
    extern __shared__ __align__(16) char smem_raw[];
    PairSmem<float, LD>& S = *reinterpret_cast<PairSmem<float, LD>*>(smem_raw);
    const int64_t G = gridDim.x;
    int64_t b = blockIdx.x;
    if (b >= A.nblocks) return;
    uint32_t nd_next[2];
    int ns, ns_next;
    uint4 item = pair_load_item(A, b), item_next = pair_load_item(A, b + G);
    float2 lm[2];
    {
        uint32_t nd0[2];
        pair_load_ids<LD>(A, b, nd0, ns);
        pair_stage<LD, 1>(p.v32, 1, A, b, nd0, ns, S, 0);
        __pipeline_commit();
        pair_load_ids<LD>(A, b + G, nd_next, ns_next);
        pair_load_tangents<CACHED>(p, item, lm);
        if (CACHED && item_next.w != kNoItem) prefetch_l2(&p.lm32[2 * (int64_t)item_next.w]);
    }
    for (int it = 0; b < A.nblocks; b += G, ++it) {
        uint32_t nd_after[2];
        int ns_after;
        pair_load_ids<LD>(A, b + 2 * G, nd_after, ns_after);
        const uint4 item_after = pair_load_item(A, b + 2 * G);
        __pipeline_wait_prior(0);
        // as in k_tet_pair: block b has landed, and the buffers of block b + G are free
        __syncthreads();
        if (b + G < A.nblocks) pair_stage<LD, 1>(p.v32, 1, A, b + G, nd_next, ns_next, S, (it + 1) & 1);
        __pipeline_commit();
        nd_next[0] = nd_after[0], nd_next[1] = nd_after[1];
        if (item.w != kNoItem) {
            float* E = S.E + threadIdx.x;
            double e[4][3], n12[3], c0[3], c1[3];
            float g[4][3], v[3][3], r0[3], r1[3], r2[3];
            int n[5];
            pair_nodes(item, n);
            pair_diffs<LD>(n, S.node[it & 1].x, e);
            pair_diffs<LD>(n, S.node[it & 1].v, g);
            cross3(e[0], e[1], n12);
            cross3(e[1], e[2], c0);
            cross3(e[2], e[0], c1);
            pair_tet32(p, lm[0], c0, c1, n12, e[0][0] * c0[0] + e[0][1] * c0[1] + e[0][2] * c0[2], g[0], g[1], g[2], v);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                r0[c] = -(v[0][c] + v[1][c] + v[2][c]);
                r1[c] = v[0][c];
                r2[c] = v[1][c];
                E[(9 + c) * kPairThreads] = v[2][c];
            }
            if (!pair_single(item)) {
                double m[3];
#pragma unroll
                for (int c = 0; c < 3; ++c) m[c] = -n12[c];
                cross3(e[0], e[3], c0);
                cross3(e[3], e[1], c1);
                pair_tet32(p, lm[1], c0, c1, m, e[1][0] * c0[0] + e[1][1] * c0[1] + e[1][2] * c0[2], g[1], g[0], g[3], v);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    r0[c] -= v[0][c] + v[1][c] + v[2][c];
                    r2[c] += v[0][c];
                    r1[c] += v[1][c];
                    E[(12 + c) * kPairThreads] = v[2][c];
                }
            }
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                E[c * kPairThreads] = r0[c];
                E[(3 + c) * kPairThreads] = r1[c];
                E[(6 + c) * kPairThreads] = r2[c];
            }
        }
        item = item_next, item_next = item_after;
        pair_load_tangents<CACHED>(p, item, lm);
        if (CACHED && item_next.w != kNoItem) prefetch_l2(&p.lm32[2 * (int64_t)item_next.w]);
        __syncthreads();
        wait_for_previous();
        const auto& M = S.meta[it & 1];
        for (int k = threadIdx.x; k < ns; k += kPairThreads) {
            const uint32_t id = M.ids[k];
            float* o = p.out32 + 3 * (int64_t)(id & ~kPairShared);
            float r[3], old[3] = {0.f, 0.f, 0.f};
            if (!(id & kPairShared))
#pragma unroll
                for (int d = 0; d < 3; ++d) old[d] = o[d];
            pair_node_sum(S.E, M.inc, M.off[k], M.off[k + 1], r);
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                if (id & kPairShared) red_add(o + d, r[d]);
                else o[d] = old[d] + r[d];
            }
        }
        ns = ns_next, ns_next = ns_after;
    }
    __pipeline_wait_prior(0);
}

// Second pass of the deterministic mode: every node that is not owned by exactly one block gets the
// sum of its blocks' partial sums, in block order (nodes in no cell get zero).
template <bool INSERT>
__global__ void k_pair_fixup(double* __restrict__ out, const double* __restrict__ partial, const int32_t* __restrict__ fix_node,
                             const int32_t* __restrict__ fix_off, const int32_t* __restrict__ fix_slot, int64_t nfix) {
    for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nfix; f += (int64_t)gridDim.x * blockDim.x) {
        double r[3] = {0.0, 0.0, 0.0};
        for (int j = fix_off[f]; j < fix_off[f + 1]; ++j)
#pragma unroll
            for (int d = 0; d < 3; ++d) r[d] += partial[3 * (int64_t)fix_slot[j] + d];
        double* o = out + 3 * (int64_t)fix_node[f];
#pragma unroll
        for (int d = 0; d < 3; ++d) o[d] = INSERT ? r[d] : o[d] + r[d];
    }
}

// ---- host: layout ------------------------------------------------------------------------------
namespace {

constexpr int kHalf = 16;       // lanes whose 64-bit reads go through together (bankplan.hpp)
// Steps of the numbering's search: 4,000 leave 2.7 cycles per gather of a warp (ideal 2; 3.7 when whole
// warps are planned), 16,000 leave 2.4 and plan more than twice as long: 43.3 and 42.3 us on 1,296,000 cells.
constexpr int kPlanSteps = 4000;

struct PairPlan {
    std::vector<int32_t> loc;       // global ids of the local nodes, by local index
    // {n0 | n1 << 16, n2 | n3 << 16, n4 | (B - A + kCellBias) << 16, A}: local node indices, cells A and
    // B (single cells: upper half of the third word 0)
    std::vector<uint32_t> items;    // [nitems][4]
    std::vector<uint16_t> off, inc;
};

struct Item {
    int a, b;       // cells of the block (b = -1: single)
    int32_t n[5];   // local node of each corner (n[4] = n[0] for a single)
};

// Corner order of cell v with corner k last that keeps its orientation.
void apex_last(const int* v, int k, int32_t (&out)[4]) {
    int m = 0;
    for (int i = 0; i < 4; ++i)
        if (i != k) out[m++] = v[i];
    out[3] = v[k];
    if ((3 - k) & 1) std::swap(out[0], out[1]);
}

// Face-sharing pairs of the block's cells (local connectivity lc): a maximal matching that takes the
// cells with the fewest free neighbours first. Pairs whose orientations do not fit (cells that are
// not consistently oriented across the face) stay single.
std::vector<Item> match_cells(const std::vector<int>& lc, int ncell) {
    static_assert(kPairMaxNodes <= 256 && kPairCells <= 256, "a face (three local nodes), its cell and corner in one word");
    std::vector<uint64_t> faces;
    faces.reserve(4 * (size_t)ncell);
    for (int c = 0; c < ncell; ++c)
        for (int k = 0; k < 4; ++k) {
            int f[3], m = 0;
            for (int i = 0; i < 4; ++i)
                if (i != k) f[m++] = lc[4 * c + i];
            if (f[0] > f[1]) std::swap(f[0], f[1]);
            if (f[1] > f[2]) std::swap(f[1], f[2]);
            if (f[0] > f[1]) std::swap(f[0], f[1]);
            faces.push_back((uint64_t)f[0] << 32 | (uint64_t)f[1] << 24 | (uint64_t)f[2] << 16 | (uint64_t)c << 2 | (uint64_t)k);
        }
    std::sort(faces.begin(), faces.end());
    struct Edge {
        int cell, k, k2;  // neighbour, this cell's and its corner off the face
    };
    struct Edges {
        int count = 0;
        Edge e[8];  // (a face that more than two cells share gives a cell two)
        const Edge* begin() const { return e; }
        const Edge* end() const { return e + count; }
        int size() const { return count; }
        void push_back(const Edge& x) { e[count++] = x; }
    };
    std::vector<Edges> adj(ncell);
    for (size_t i = 0; i + 1 < faces.size(); ++i) {
        const int c = (int)(faces[i] >> 2 & 0x3fff), d = (int)(faces[i + 1] >> 2 & 0x3fff);
        if (faces[i] >> 16 != faces[i + 1] >> 16 || c == d) continue;
        adj[c].push_back({d, (int)(faces[i] & 3), (int)(faces[i + 1] & 3)});
        adj[d].push_back({c, (int)(faces[i + 1] & 3), (int)(faces[i] & 3)});
    }
    std::vector<int> deg(ncell);
    std::vector<char> used(ncell, 0);
    using Q = std::pair<int, int>;
    std::priority_queue<Q, std::vector<Q>, std::greater<Q>> heap;
    for (int c = 0; c < ncell; ++c) heap.push({deg[c] = (int)adj[c].size(), c});
    std::vector<Item> items;
    auto drop = [&](int c) {
        used[c] = 1;
        for (const Edge& e : adj[c])
            if (!used[e.cell]) heap.push({--deg[e.cell], e.cell});
    };
    while (!heap.empty()) {
        const auto [d, c] = heap.top();
        heap.pop();
        if (used[c] || d != deg[c]) continue;
        const Edge* best = nullptr;
        int32_t A[4], B[4];
        for (const Edge& e : adj[c]) {
            if (used[e.cell] || (best && deg[e.cell] >= deg[best->cell])) continue;
            // cell c as (n0, n1, n2, n3); the other must be an even permutation of (n0, n2, n1, n4)
            int32_t x[4], y[4];
            apex_last(&lc[4 * c], e.k, x);
            apex_last(&lc[4 * e.cell], e.k2, y);
            bool fits = false;
            for (int r = 0; r < 3; ++r) fits = fits || (y[r] == x[0] && y[(r + 1) % 3] == x[2] && y[(r + 2) % 3] == x[1]);
            if (!fits) continue;
            best = &e;
            std::copy(x, x + 4, A);
            std::copy(y, y + 4, B);
        }
        Item it;
        it.a = c;
        if (best) {
            it.b = best->cell;
            for (int i = 0; i < 4; ++i) it.n[i] = A[i];
            it.n[4] = B[3];
            const int other = best->cell;
            drop(c);
            drop(other);
        } else {
            it.b = -1;
            for (int i = 0; i < 4; ++i) it.n[i] = lc[4 * c + i];
            it.n[4] = it.n[0];
            drop(c);
        }
        items.push_back(it);
    }
    std::sort(items.begin(), items.end(), [](const Item& x, const Item& y) { return x.a < y.a; });
    return items;
}

// A block: its cell count, its nodes in increasing order, and its items (local nodes: indices into them).
struct PairCut {
    int ncell;
    std::vector<int32_t> nodes;
    std::vector<Item> items;
};

// The block of the ncell cells bc[ncell][4]; returns 0, or where they need more items or nodes than a block
// has, how many cells fewer it must be at least (a cell less saves an item or four nodes at most).
int cut_pair_block(const int32_t* bc, int ncell, PairCut& cut) {
    cut.ncell = ncell;
    std::vector<uint64_t> at(4 * (size_t)ncell);  // (node, corner)
    for (int i = 0; i < 4 * ncell; ++i) at[i] = (uint64_t)bc[i] << 32 | (uint32_t)i;
    std::sort(at.begin(), at.end());
    cut.nodes.clear();
    std::vector<int> lc(4 * (size_t)ncell);
    for (uint64_t x : at) {
        const int32_t v = (int32_t)(x >> 32);
        if (cut.nodes.empty() || cut.nodes.back() != v) cut.nodes.push_back(v);
        lc[(uint32_t)x] = (int)cut.nodes.size() - 1;
    }
    const int nodes = (int)cut.nodes.size();
    if (nodes > kPairMaxNodes) return (nodes - kPairMaxNodes + 3) / 4;
    cut.items = match_cells(lc, ncell);
    return std::max(0, (int)cut.items.size() - kPairThreads);
}

// Blocks of the cells [begin, end): as even as kPairCells allows, a block that does not fit shrunk; false
// for scattered cells (see ensure_pair_layout). A few per cent of the planning: all of a mesh is cut
// before any of it is planned.
bool cut_pair_range(const int32_t* cells, int64_t begin, int64_t end, std::vector<PairCut>& out) {
    for (int64_t c = begin; c < end;) {
        const int64_t left = end - c, nb = (left + kPairCells - 1) / kPairCells;
        int n = (int)((left + nb - 1) / nb);
        PairCut cut;
        for (int fewer; (fewer = cut_pair_block(cells + 4 * c, n, cut)) > 0;) {
            for (const int most = n - fewer; n > most; n -= std::max(2, n / 16))
                if (n <= kPairCells / 2) return false;
        }
        out.push_back(std::move(cut));
        c += n;
    }
    return true;
}

// Numbers the nodes and orders the incidences of the block that starts at cell c0.
void plan_pair_block(int64_t c0, const PairCut& cut, PairPlan& P) {
    const std::vector<Item>& items = cut.items;
    const int nloc = (int)cut.nodes.size(), ni = (int)items.size();
    std::vector<std::vector<int>> groups(nloc);
    std::vector<int> deg(nloc, 0);
    for (int i = 0; i < ni; ++i)
        for (int k = 0; k < (items[i].b < 0 ? 4 : 5); ++k) {
            const int l = items[i].n[k], g = i / kHalf * 5 + k;
            deg[l]++;
            if (groups[l].empty() || std::find(groups[l].begin(), groups[l].end(), g) == groups[l].end()) groups[l].push_back(g);
        }
    std::vector<int32_t> perm;
    spread_nodes(groups, (ni + kHalf - 1) / kHalf * 5, deg, (uint64_t)c0, kPlanSteps, perm);
    P.loc.resize(nloc);
    for (int l = 0; l < nloc; ++l) P.loc[perm[l]] = cut.nodes[l];
    std::vector<std::vector<int>> lists(nloc);
    P.items.clear();
    for (int i = 0; i < ni; ++i) {
        uint32_t n[5];
        for (int k = 0; k < 5; ++k) {
            n[k] = (uint32_t)perm[items[i].n[k]];
            if (k < 4 || items[i].b >= 0) lists[n[k]].push_back(8 * i + k);
        }
        const uint32_t db = items[i].b < 0 ? 0u : (uint32_t)(items[i].b - items[i].a + kCellBias);
        for (uint32_t w : {n[0] | n[1] << 16, n[2] | n[3] << 16, n[4] | db << 16, (uint32_t)(c0 + items[i].a)}) P.items.push_back(w);
    }
    const auto ordered = order_for_banks(lists, (nloc + kWarp - 1) / kWarp, [](int k) { return k / kWarp; }, 3, kHalf);
    P.off.assign(1, 0);
    P.inc.clear();
    for (int k = 0; k < nloc; ++k) {
        for (int e : ordered[k]) P.inc.push_back((uint16_t)((e & 7) * 3 * kPairThreads + (e >> 3)));
        P.off.push_back((uint16_t)P.inc.size());
    }
}

int build_pair_layout(pl_mesh_s* m) {
    PairLayout* L = new PairLayout();
    m->pair = L;  // empty: not used for this mesh
    if (m->cell_type != PL_CELL_TET4 || m->nnodes >= (int64_t)kPairShared || m->ncells >= (int64_t)INT32_MAX) return PL_OK;
    // ranges of up to 16 blocks, planned in parallel (a range's plan depends only on its cells; the
    // calling thread takes ranges too, so the layout is complete even where no helper thread can be
    // started)
    const int64_t nc = m->ncells, want = (nc + kPairCells - 1) / kPairCells;
    const int64_t per = std::max<int64_t>(1, std::min<int64_t>(16, want / 64)), nr = (want + per - 1) / per;
    std::vector<std::vector<PairPlan>> plans(nr);
    std::atomic<bool> failed{false}, refused{false};
    auto all_ranges = [&](auto&& range) {  // range(r, first cell, last): false where the mesh is refused
        std::atomic<int64_t> next{0};
        auto work = [&]() noexcept {
            try {
                for (int64_t r; !failed.load() && !refused.load() && (r = next.fetch_add(1)) < nr;)
                    if (!range(r, r * nc / nr, (r + 1) * nc / nr)) refused.store(true);
            } catch (...) {
                failed.store(true);
            }
        };
        const int nth = (int)std::min<int64_t>(std::min(15u, std::thread::hardware_concurrency()), nr);
        std::vector<std::thread> th;
        try {
            for (int t = 1; t < nth; ++t) th.emplace_back(work);
        } catch (...) {
        }
        work();
        for (std::thread& x : th) x.join();
    };
    std::vector<std::vector<PairCut>> cuts(nr);
    all_ranges([&](int64_t r, int64_t c0, int64_t c1) { return cut_pair_range(m->h_cells.data(), c0, c1, cuts[r]); });
    if (!refused.load()) all_ranges([&](int64_t r, int64_t c, int64_t) {
        for (PairCut& cut : cuts[r]) {
            plans[r].emplace_back();
            plan_pair_block(c, cut, plans[r].back());
            c += cut.ncell;
            cut = PairCut();
        }
        return true;
    });
    if (failed.load()) return fail(PL_ERR_OUT_OF_MEMORY, "cell-pair layout planning ran out of host memory");
    if (refused.load()) return PL_OK;
    int maxloc = 0;
    int64_t nb = 0;
    for (const std::vector<PairPlan>& range : plans)
        for (const PairPlan& P : range) maxloc = std::max(maxloc, (int)P.loc.size()), ++nb;
    const size_t LD = maxloc <= kPairSmallLd ? kPairSmallLd : kPairMaxNodes;
    std::vector<int32_t> nslots(nb), nblocks_of(m->nnodes, 0);
    std::vector<uint32_t> ids(nb * LD, kNoNode), items((size_t)nb * 4 * kPairThreads, kNoItem);
    std::vector<double> coords(nb * 3 * LD, 0.0);
    std::vector<uint16_t> off(nb * (LD + 8), 0), inc((size_t)nb * 5 * kPairThreads, 0);
    size_t b = 0;
    for (std::vector<PairPlan>& range : plans)
        for (PairPlan& P : range) {
            nslots[b] = (int32_t)P.loc.size();
            for (int i = 0; i < nslots[b]; ++i) {
                ids[b * LD + i] = (uint32_t)P.loc[i];
                nblocks_of[P.loc[i]]++;
                for (int d = 0; d < 3; ++d) coords[(3 * b + d) * LD + i] = m->h_coords[3 * (size_t)P.loc[i] + d];
            }
            std::copy(P.off.begin(), P.off.end(), off.begin() + b * (LD + 8));
            std::copy(P.inc.begin(), P.inc.end(), inc.begin() + b * 5 * kPairThreads);
            std::copy(P.items.begin(), P.items.end(), items.begin() + b * 4 * kPairThreads);
            ++b;
            P = PairPlan();
        }
    // nodes not owned by exactly one block, with their slots in block order
    std::vector<int32_t> fix_node, fix_off(1, 0), fix_slot, first(m->nnodes + 1, 0);
    for (uint32_t& id : ids)
        if (id != kNoNode && nblocks_of[id] > 1) {
            first[id + 1]++;
            id |= kPairShared;
        }
    for (int64_t v = 0; v < m->nnodes; ++v) first[v + 1] += first[v];
    std::vector<int32_t> slots(first[m->nnodes]), pos(first.begin(), first.end() - 1);
    for (size_t at = 0; at < ids.size(); ++at)
        if (ids[at] != kNoNode && (ids[at] & kPairShared)) slots[pos[ids[at] & ~kPairShared]++] = (int32_t)at;
    for (int64_t v = 0; v < m->nnodes; ++v) {
        if (nblocks_of[v] == 1) continue;
        fix_node.push_back((int32_t)v);
        fix_slot.insert(fix_slot.end(), slots.begin() + first[v], slots.begin() + first[v + 1]);
        fix_off.push_back((int32_t)fix_slot.size());
    }
    cudaStream_t s = m->ctx->stream;
    cudaError_t e = cudaSuccess;
    auto up = [&](auto** dst, const auto& v) {
        if (e != cudaSuccess || v.empty()) return;
        const size_t bytes = v.size() * sizeof(v[0]);
        e = dev_alloc((void**)dst, bytes);
        if (e == cudaSuccess) e = cudaMemcpyAsync(*dst, v.data(), bytes, cudaMemcpyHostToDevice, s);
    };
    up(&L->d_nslots, nslots);
    up(&L->d_ids, ids);
    up(&L->d_coords, coords);
    up(&L->d_off, off);
    up(&L->d_inc, inc);
    up(&L->d_items, items);
    up(&L->d_fix_node, fix_node);
    up(&L->d_fix_off, fix_off);
    up(&L->d_fix_slot, fix_slot);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return cuda_fail(e, "cell-pair layout upload");
    L->num_slots = (int64_t)ids.size();
    L->num_fix = (int64_t)fix_node.size();
    L->ld = (int)LD;
    L->h_ids.swap(ids);
    L->num_blocks = nb;
    return PL_OK;
}

template <typename T, int LD, typename Kernel>
void launch_pairs(Kernel kern, const DomainParams& p, const PairArrays& A, cudaStream_t s) {
    constexpr size_t smem = sizeof(PairSmem<T, LD>);
    ensure_kernel_smem((const void*)kern, smem);
    launch_domain(kern, std::min<int64_t>(A.nblocks, (int64_t)sm_count() * (sizeof(T) == 4 ? kPairCtas32 : kPairCtas)), kPairThreads, smem, s, p, A);
}

template <bool BF, int OP, bool INSERT, bool DET>
void launch_one(const DomainParams& p, const PairLayout& L, const PairArrays& A, cudaStream_t s) {
    if (L.ld == kPairSmallLd) launch_pairs<double, kPairSmallLd>(k_tet_pair<RHEO_ILE, BF, OP, INSERT, DET, kPairSmallLd>, p, A, s);
    else launch_pairs<double, kPairMaxNodes>(k_tet_pair<RHEO_ILE, BF, OP, INSERT, DET, kPairMaxNodes>, p, A, s);
}

template <bool CACHED>
void launch_jv32(const DomainParams& p, const PairLayout& L, const PairArrays& A, cudaStream_t s) {
    if (L.ld == kPairSmallLd) launch_pairs<float, kPairSmallLd>(k_tet_pair_jv32<CACHED, kPairSmallLd>, p, A, s);
    else launch_pairs<float, kPairMaxNodes>(k_tet_pair_jv32<CACHED, kPairMaxNodes>, p, A, s);
}

template <bool BF, int OP>
void launch_op(const DomainParams& p, const PairLayout& L, bool insert, double* partial, bool reduced, cudaStream_t s) {
    const PairArrays A = pair_arrays_of(L, partial, reduced);
    if (partial && insert) launch_one<BF, OP, true, true>(p, L, A, s);
    else if (partial) launch_one<BF, OP, false, true>(p, L, A, s);
    else if (insert) launch_one<BF, OP, true, false>(p, L, A, s);
    else launch_one<BF, OP, false, false>(p, L, A, s);
    if (partial && L.num_fix > 0) {
        const int g = (int)std::min<int64_t>((L.num_fix + 255) / 256, 148 * 8);
        if (insert) k_pair_fixup<true><<<g, 256, 0, s>>>(p.out, partial, L.d_fix_node, L.d_fix_off, L.d_fix_slot, L.num_fix);
        else k_pair_fixup<false><<<g, 256, 0, s>>>(p.out, partial, L.d_fix_node, L.d_fix_off, L.d_fix_slot, L.num_fix);
        count_launch();
    }
}

}  // namespace

// PYLITH_B200_TET_KERNEL, read once per process: "pair" (the default) or a cell-block kernel of
// blocked.cu.
static bool tet_pairs_selected() {
    static const bool on = [] {
        const char* v = std::getenv("PYLITH_B200_TET_KERNEL");
        return !v || (std::strcmp(v, "pad2") != 0 && std::strcmp(v, "pipe") != 0 && std::strcmp(v, "twophase") != 0);
    }();
    return on;
}

// The mesh's pair layout (num_blocks 0: not usable). Meshes whose consecutive cells are scattered, so
// that a block of kPairCells / 2 of them does not fit, keep the layout of single cells; the blocks are cut
// before any is planned, so that such a mesh pays little for the attempt. Residual here and there, first
// call in brackets, in us (ms):
//   1,179,648 structured cells along a Morton curve 35.0 and 48.4 (253 and 597), in grid order, with
//     kPairMaxNodes slots per block, 35.1 and 47.4 (198 and 432)
//   394,718 Delaunay cells along a Morton curve 16.5 and 21.7 (90 and 210), in Qhull's order 18.7 and 31.9
//     (89 and 186)
//   384,000 cells shuffled within windows of 480 21.5 and 29.8 (121 to 170 and 231); of 10,000, refused,
//     44.4 either way (207 and 202 without the attempt); shuffled throughout, if forced, 52.2 and 48.0
int ensure_pair_layout(pl_mesh_s* m) {
    if (m->pair) return PL_OK;
    int rc;
    try {
        rc = build_pair_layout(m);
    } catch (const std::bad_alloc&) {
        rc = fail(PL_ERR_OUT_OF_MEMORY, "cell-pair layout: out of host memory");
    } catch (...) {
        rc = fail(PL_ERR_INVALID_ARG, "cell-pair layout failed");
    }
    if (rc) {
        free_pair_layout(m->pair, m->ctx->stream);
        m->pair = nullptr;
    }
    return rc;
}

int ensure_pair_reduced_ids(pl_mesh_s* m) {
    PairLayout* L = m->pair;
    if (!L || L->num_blocks == 0) return fail(PL_ERR_UNSUPPORTED, "no cell-pair layout");
    if (L->d_ids_red) return PL_OK;
    if (m->h_node_red.size() != (size_t)m->nnodes) return fail(PL_ERR_UNSUPPORTED, "no reduced fault space");
    // a node of the reduced space is owned by its block only if it has one slot in all blocks
    std::vector<uint32_t> ids(L->h_ids.size(), 0u);
    std::vector<int32_t> slots(m->nnodes, 0);
    for (size_t at = 0; at < ids.size(); ++at)
        ids[at] = L->h_ids[at] == kNoNode ? kNoNode : (uint32_t)m->h_node_red[L->h_ids[at] & ~kPairShared];
    for (uint32_t id : ids)
        if (id != kNoNode) slots[id]++;
    for (uint32_t& id : ids)
        if (id != kNoNode && slots[id] > 1) id |= kPairShared;
    uint32_t* d = nullptr;
    PLB_CUDA(dev_alloc(&d, ids.size()));
    cudaError_t e = cudaMemcpyAsync(d, ids.data(), ids.size() * sizeof(uint32_t), cudaMemcpyHostToDevice, m->ctx->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(m->ctx->stream);
    if (e != cudaSuccess) {
        dev_free(d, m->ctx->stream);
        return cuda_fail(e, "reduced slot ids");
    }
    L->d_ids_red = d;
    return PL_OK;
}

// Whether the mesh's cell-block kernels run on pairs (after prepare_tet_layout).
bool uses_pairs(const pl_mesh_s* m) { return m->pair && m->pair->num_blocks > 0; }

int prepare_tet_layout(pl_mesh_s* m) {
    int rc = PL_OK;
    if (tet_pairs_selected() && (rc = ensure_pair_layout(m)) != PL_OK) return rc;
    return uses_pairs(m) ? PL_OK : ensure_blocked_layout(m);
}

int ensure_cell_ids_reduced(pl_mesh_s* m) { return uses_pairs(m) ? ensure_pair_reduced_ids(m) : ensure_reduced_ids(m); }

bool launch_domain_apply_pair(const DomainParams& p, const PairLayout& L, int rheo, bool bf, int op, bool insert, int64_t nnodes,
                              double* partial, cudaStream_t s, bool reduced) {
    if (rheo != RHEO_ILE || L.num_blocks == 0 || (reduced && (insert || partial || !L.d_ids_red))) return false;
    // INSERT without partial sums: shared nodes are reduced into zeros
    DomainParams q = p;
    q.after_zeros = insert && !partial && L.num_fix > 0 && zero_output(p.out, 3 * nnodes, true, true, s);
    if (op != OP_RESIDUAL) launch_op<false, OP_JACOBIAN_ACTION>(q, L, insert, partial, reduced, s);
    else if (bf) launch_op<true, OP_RESIDUAL>(q, L, insert, partial, reduced, s);
    else launch_op<false, OP_RESIDUAL>(q, L, insert, partial, reduced, s);
    return true;
}

// The FP32 action; with the solver's cached tangent any isotropic rheology.
bool launch_domain_jv32_pair(const DomainParams& p, const PairLayout& L, int rheo, cudaStream_t s, bool reduced) {
    if ((rheo != RHEO_ILE && !p.lm32) || L.num_blocks == 0 || (reduced && !L.d_ids_red)) return false;
    const PairArrays A = pair_arrays_of(L, nullptr, reduced);
    if (p.lm32) launch_jv32<true>(p, L, A, s);
    else launch_jv32<false>(p, L, A, s);
    return true;
}

void free_pair_layout(PairLayout* L, cudaStream_t after) {
    if (!L) return;
    for (void* p : {(void*)L->d_nslots, (void*)L->d_ids, (void*)L->d_ids_red,
                    (void*)L->d_coords, (void*)L->d_off, (void*)L->d_inc, (void*)L->d_items, (void*)L->d_fix_node,
                    (void*)L->d_fix_off, (void*)L->d_fix_slot})
        dev_free(p, after);
    delete L;
}

}  // namespace plb
