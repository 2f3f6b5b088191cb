// Q2 hexahedra (27 nodes, 3x3x3 Gauss points) by sum factorisation with a plane of nodes per lane:
// FP64 residual and Jacobian action (small meshes: hex27lines.cu).
//
// Three lanes share a cell, ten cells a warp. The Q2 basis is a tensor product of the 1-D quadratic
// basis, so the reference gradient at the points is three 1-D contractions. Lane m takes the nodes
// of the plane zeta = node m through the x and y contractions in its registers (27 values per
// component), the planes are exchanged through shared memory, and the lane takes the z-lines
// (i = m, j) of points one after the other: z contraction, geometry, pointwise function and the
// transposed z contraction in registers, written back where they were read. The x and y
// transposes run on planes again. A value so crosses shared memory twice each way (972 accesses
// per cell) instead of at every change of direction. Field and result cross between global and
// shared memory with consecutive lanes on consecutive doubles of the cells' rows of nodes, the loads
// as cp.async (10 warps per multiprocessor do not cover plain ones: 468 us), and sums of nodes that
// consecutive cells share are handed on before they are added.
//
// Bound: latency at 2.5 warps per scheduler, the L1 pipe at 60 % and FP64 (2,180 operations per lane
// and cell) at 45 %; registers and shared memory both stop at 10 warps. 64^3 cells (262,144): 465 us
// with a line of points per lane (nine lanes per cell, L1 pipe 94 %), 230 us this way. Measured and
// not kept: a persistent loop that loads the next pass's node ids during this one (344 us, 200
// bytes of spills); 8 warps without spills (245 us); node ids prefetched a wave ahead (no change).
#include <cuda_pipeline.h>

#include <algorithm>

#include "domain_kernels.cuh"
#include "internal.hpp"
#include "launch.hpp"

namespace plb {

namespace q2 {
// Gauss points -a, 0, a (a^2 = 3/5), weights 5/9, 8/9, 5/9; half of a. Basis values at a: kB0, 0.4,
// kB2; derivatives at a: a - 1/2, -2 a, a + 1/2; at -a mirrored; at 0 the middle node.
constexpr double kA = 0.77459666924148337704, kHalfA = 0.5 * kA;
constexpr double kB0 = 0.3 - kHalfA, kB2 = 0.3 + kHalfA, kD0 = kA - 0.5, kD2 = kA + 0.5;

// Values B u and derivatives D u at the points of a line with node values u0, u1, u2.
PL_D void fwd_b(double u0, double u1, double u2, double& b0, double& b1, double& b2) {
    b0 = kB2 * u0 + 0.4 * u1 + kB0 * u2;
    b1 = u1;
    b2 = kB0 * u0 + 0.4 * u1 + kB2 * u2;
}
PL_D void fwd_d(double u0, double u1, double u2, double& d0, double& d1, double& d2) {
    d0 = 2.0 * kA * u1 - kD2 * u0 - kD0 * u2;
    d1 = 0.5 * (u2 - u0);
    d2 = kD0 * u0 + kD2 * u2 - 2.0 * kA * u1;
}
// The transposes, set or added to n0, n1, n2.
PL_D void rev_b(double p0, double p1, double p2, double (&n)[3]) {
    n[0] = kB2 * p0 + kB0 * p2;
    n[1] = 0.4 * (p0 + p2) + p1;
    n[2] = kB0 * p0 + kB2 * p2;
}
PL_D void rev_b_add(double p0, double p1, double p2, double (&n)[3]) {
    n[0] = fma(kB2, p0, fma(kB0, p2, n[0]));
    n[1] = fma(0.4, p0 + p2, n[1] + p1);
    n[2] = fma(kB0, p0, fma(kB2, p2, n[2]));
}
PL_D void rev_d(double q0, double q1, double q2, double (&n)[3]) {
    n[0] = fma(kD0, q2, fma(-kD2, q0, -0.5 * q1));
    n[1] = 2.0 * kA * (q0 - q2);
    n[2] = fma(kD2, q2, fma(-kD0, q0, 0.5 * q1));
}
PL_D void rev_d_add(double q0, double q1, double q2, double (&n)[3]) {
    n[0] = fma(kD0, q2, fma(-kD2, q0, fma(-0.5, q1, n[0])));
    n[1] = fma(2.0 * kA, q0 - q2, n[1]);
    n[2] = fma(kD2, q2, fma(-kD0, q0, fma(0.5, q1, n[2])));
}

constexpr int WARPS = 2, CELLS = 10;  // cells per warp: lanes 3 g + m, m = 0 .. 2
// Per cell: [plane 3][component 3][channel 3][point 9] doubles, channels BB, BD (d/dy), DB (d/dx).
// 81 doubles per lane, 1 modulo the 16 eight-byte bank pairs: a warp's accesses, whether each lane
// reads its own plane or its own line i = m, fall on distinct pairs.
constexpr int CELL = 243, O_ID = CELLS * CELL;
constexpr int PER_WARP = O_ID + CELLS * 27 / 2;
constexpr size_t smem_bytes() { return sizeof(double) * (size_t)WARPS * PER_WARP; }

// The 81 field values of each of a warp's cells in the order (row of 3 nodes, cell, node,
// component), packed: byte offset in S (bits 0-14), byte offset in sId (16-27), component (28-29).
// A table, because the divisions by 3 and 10 of each entry took as many issue slots as half of the
// arithmetic.
constexpr int ENTRIES = 81 * CELLS;
struct EntryTable {
    uint32_t e[ENTRIES];
};
constexpr EntryTable make_entries() {
    EntryTable t{};
    for (int i = 0; i < ENTRIES; ++i) {
        const int d = i % 3, a = i / 3 % 3, cell = i / 9 % CELLS, row = i / (9 * CELLS);
        const int at = CELL * cell + 81 * (row / 3) + 27 * d + 3 * (row % 3) + a;
        t.e[i] = (uint32_t)(8 * at) | (uint32_t)(4 * (27 * cell + 3 * row + a)) << 16 | (uint32_t)d << 28;
    }
    return t;
}
__device__ const EntryTable kEntries = make_entries();
constexpr int BATCH = 9;  // entries of a lane in flight: three batches
PL_D int id_offset(uint32_t e) { return e >> 16 & 0xfff; }
PL_D int value_offset(uint32_t e) { return e & 0x7fff; }
PL_D int64_t dof(int id, uint32_t e) { return 3 * (int64_t)id + (e >> 28); }
}  // namespace q2

template <int RHEO, bool BF, int OP>
__global__ void __launch_bounds__(q2::WARPS * 32, RHEO == RHEO_ILE ? 5 : 4) k_hex27_planes(DomainParams p) {
    using namespace q2;
    using L = AuxLayout<RHEO, BF>;
    constexpr bool BODY = BF && OP == OP_RESIDUAL;
    const AuxOffsets<RHEO, BF> aoff;
    extern __shared__ __align__(16) double q2_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* S = q2_smem + warp * PER_WARP;
    int32_t* sId = reinterpret_cast<int32_t*>(S + O_ID);
    const double* __restrict__ field = OP == OP_RESIDUAL ? p.u : p.v;
    const int64_t c0 = ((int64_t)blockIdx.x * WARPS + warp) * CELLS;
    if (c0 >= p.ncells) return;  // whole warps
    const int nc = (int)min((int64_t)CELLS, p.ncells - c0);
    const int g = lane / 3, m = lane - 3 * g;
    const bool live = g < nc;  // lanes 30, 31: g = 10
    {
        constexpr int N = (27 * CELLS + 31) / 32;
        int id[N];
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int t = lane + 32 * i, k = t / 27;
            id[i] = -1;
            if (t < 27 * nc) id[i] = p.cells[(p.cell_ids ? (int64_t)p.cell_ids[c0 + k] : c0 + k) * 27 + (t - 27 * k)];
        }
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (lane + 32 * i < 27 * CELLS) sId[lane + 32 * i] = id[i];  // -1: no cell
    }
    __syncwarp();
    // the field of node a + 3 row, component d, at channel BB of its plane: rows of all cells together,
    // so cells consecutive along x read consecutive nodes
#pragma unroll 1
    for (int i0 = lane; i0 < ENTRIES; i0 += 32 * BATCH) {
        uint32_t e[BATCH];
        int id[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) e[i] = i0 + 32 * i < ENTRIES ? kEntries.e[i0 + 32 * i] : 0u;
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
            id[i] = i0 + 32 * i < ENTRIES ? *reinterpret_cast<const int*>(reinterpret_cast<const char*>(sId) + id_offset(e[i])) : -1;
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
            if (id[i] >= 0)
                __pipeline_memcpy_async(reinterpret_cast<char*>(S) + value_offset(e[i]), field + dof(id[i], e[i]), sizeof(double));
    }
    // the corners' coordinates on their way to L2
    if (live)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            if (m + 3 * k < 8) prefetch_l2(&p.coords[3 * (int64_t)sId[27 * g + Elem<HEX27>::corner(m + 3 * k)]]);
    __pipeline_commit();
    __pipeline_wait_prior(0);
    __syncwarp();
    if (live) {
        // x and y contractions of this lane's plane
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            double* R = S + 81 * lane + 27 * d;
            double xb[3][3], xd[3][3];  // [b][i]
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const double u0 = R[3 * b], u1 = R[3 * b + 1], u2 = R[3 * b + 2];
                fwd_b(u0, u1, u2, xb[b][0], xb[b][1], xb[b][2]);
                fwd_d(u0, u1, u2, xd[b][0], xd[b][1], xd[b][2]);
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                double v[3];
                fwd_b(xb[0][i], xb[1][i], xb[2][i], v[0], v[1], v[2]);
#pragma unroll
                for (int j = 0; j < 3; ++j) R[i + 3 * j] = v[j];
                fwd_d(xb[0][i], xb[1][i], xb[2][i], v[0], v[1], v[2]);
#pragma unroll
                for (int j = 0; j < 3; ++j) R[9 + i + 3 * j] = v[j];
                fwd_b(xd[0][i], xd[1][i], xd[2][i], v[0], v[1], v[2]);
#pragma unroll
                for (int j = 0; j < 3; ++j) R[18 + i + 3 * j] = v[j];
            }
        }
    }
    __syncwarp();
    if (live) {
        const int64_t c = c0 + g;
        double a[L::size] = {};
        double x[3] = {0, 0, 0}, s3[3] = {0, 0, 0};
        L::load_cell(p, c, a);
        double lam = 0.0, mu = 0.0;
        if (OP == OP_JACOBIAN_ACTION) {  // the tangents read no state: one evaluation per lane
            double Jf3[81];
#pragma unroll
            for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
            call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
            lam = -Jf3[((0 * 3 + 1) * 3 + 0) * 3 + 1];
            mu = -Jf3[((0 * 3 + 1) * 3 + 1) * 3 + 0];
        }
        double X[24];  // corner coordinates [8][3]
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
            for (int d = 0; d < 3; ++d) X[3 * k + d] = p.coords[3 * (int64_t)sId[27 * g + Elem<HEX27>::corner(k)] + d];
        const double wi = 0.5 + kHalfA * (m - 1);  // xi of this lane's lines on [0, 1]
        // trilinear geometry on [0, 1]^3 (the Jacobian is twice the one on [-1, 1]^3)
        double yb[3], ys[3], e0[3], es[3];  // d/deta at the bottom and its slope in zeta; vertical edge at y = 0, slope in eta
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double* x8 = X + d;
            const double y0 = x8[9] - x8[0], y1 = x8[6] - x8[3], t0 = x8[21] - x8[12], t1 = x8[18] - x8[15];
            yb[d] = y0 + wi * (y1 - y0);
            ys[d] = (t0 + wi * (t1 - t0)) - yb[d];
            const double z0 = x8[12] - x8[0], z1 = x8[15] - x8[3], z2 = x8[18] - x8[6], z3 = x8[21] - x8[9];
            e0[d] = z0 + wi * (z1 - z0);
            es[d] = (z3 + wi * (z2 - z3)) - e0[d];
        }
        const double wij0 = m == 1 ? 8.0 / 9.0 : 5.0 / 9.0;
#pragma unroll 1
        for (int j = 0; j < 3; ++j) {
            const double wj = 0.5 + kHalfA * (j - 1);
            double* R = S + CELL * g + m + 3 * j;  // + 81 plane + 27 component + 9 channel
            double G[3][3][3];                     // [k][component][direction]
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                fwd_b(R[27 * d + 18], R[81 + 27 * d + 18], R[162 + 27 * d + 18], G[0][d][0], G[1][d][0], G[2][d][0]);
                fwd_b(R[27 * d + 9], R[81 + 27 * d + 9], R[162 + 27 * d + 9], G[0][d][1], G[1][d][1], G[2][d][1]);
                fwd_d(R[27 * d], R[81 + 27 * d], R[162 + 27 * d], G[0][d][2], G[1][d][2], G[2][d][2]);
            }
            double xb[3], xs[3], jz[3];
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const double* x8 = X + d;
                const double b0 = x8[3] - x8[0], b1 = x8[6] - x8[9], t0 = x8[15] - x8[12], t1 = x8[18] - x8[21];
                xb[d] = b0 + wj * (b1 - b0);
                xs[d] = (t0 + wj * (t1 - t0)) - xb[d];
                jz[d] = e0[d] + wj * es[d];
            }
            const double wij = wij0 * (j == 1 ? 8.0 / 9.0 : 5.0 / 9.0) * 0.25;  // C on [-1, 1]^3 is a quarter
            double F0[3][3];  // [k][component] body-force weights
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double wk = 0.5 + kHalfA * (k - 1);
                double J[3][3], C[3][3];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    J[d][0] = xb[d] + wk * xs[d];
                    J[d][1] = yb[d] + wk * ys[d];
                    J[d][2] = jz[d];
                }
                C[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
                C[0][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
                C[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
                C[1][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
                C[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
                C[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
                C[2][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
                C[2][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
                C[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
                const double det = J[0][0] * C[0][0] + J[0][1] * C[1][0] + J[0][2] * C[2][0];
                if (!(det > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
                const double rdet = 2.0 / det;  // C / det on [-1, 1]^3
                const double w = wij * (k == 1 ? 8.0 / 9.0 : 5.0 / 9.0);
                double s_x[9], f1[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int e = 0; e < 3; ++e)
                        s_x[f * 3 + e] = G[k][f][0] * C[0][e] + G[k][f][1] * C[1][e] + G[k][f][2] * C[2][e];
                if (OP == OP_JACOBIAN_ACTION) {
                    const double r = rdet * w;
                    isotropic_contract<double>(lam * r, mu * r, s_x, f1);  // linear in the gradient
                } else {
#pragma unroll
                    for (int f = 0; f < 9; ++f) s_x[f] *= rdet;
                    L::load_qp(p, c, m + 3 * j + 9 * k, 27, a);
                    if constexpr (BODY) {
                        const int sOff[1] = {0}, sOff_x[1] = {0};
                        double f0[3] = {0, 0, 0};
                        pw::g0v_bodyforce<double>(3, 1, L::numA, sOff, sOff_x, s3, nullptr, s_x, aoff.v, nullptr, a, nullptr,
                                                  nullptr, p.t, x, p.num_constants, p.constants, f0);
#pragma unroll
                        for (int d = 0; d < 3; ++d) F0[k][d] = (0.5 * w * det) * f0[d];
                    }
                    call_f1<RHEO>(L::numA, aoff.v, a, s3, s_x, p, x, f1);
#pragma unroll
                    for (int f = 0; f < 9; ++f) f1[f] *= w;
                }
                // test weights w C f1 in place of the gradient
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        G[k][f][d] = C[d][0] * f1[f * 3 + 0] + C[d][1] * f1[f * 3 + 1] + C[d][2] * f1[f * 3 + 2];
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                double n[3];
                rev_b(G[0][d][0], G[1][d][0], G[2][d][0], n);
                R[27 * d + 18] = n[0], R[81 + 27 * d + 18] = n[1], R[162 + 27 * d + 18] = n[2];
                rev_b(G[0][d][1], G[1][d][1], G[2][d][1], n);
                R[27 * d + 9] = n[0], R[81 + 27 * d + 9] = n[1], R[162 + 27 * d + 9] = n[2];
                rev_d(G[0][d][2], G[1][d][2], G[2][d][2], n);
                if (BODY) rev_b_add(F0[0][d], F0[1][d], F0[2][d], n);
                R[27 * d] = n[0], R[81 + 27 * d] = n[1], R[162 + 27 * d] = n[2];
            }
        }
    }
    __syncwarp();
    // y and x transposes of this lane's plane; the node sums at channel BB. Where the next cell (lane
    // + 3) starts with this cell's last nodes (its a = 0 are this one's a = 2, as in boxes numbered
    // along x), it takes over their sums and this cell's entries are dropped.
    {
        const unsigned full = 0xffffffffu;
        int32_t* id = sId + 9 * (live ? lane : 0);  // this lane's plane
        bool give[3], take[3];
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            const int first = live ? id[3 * b] : -1, last = live ? id[3 * b + 2] : -2;
            give[b] = __shfl_down_sync(full, first, 3) == last && lane + 3 < 3 * nc;
            take[b] = __shfl_up_sync(full, (int)give[b], 3) && lane >= 3;
        }
        __syncwarp();
#pragma unroll
        for (int b = 0; b < 3; ++b)
            if (give[b]) id[3 * b + 2] = -1;
#pragma unroll 1
        for (int d = 0; d < 3; ++d) {
            double* R = S + 81 * (live ? lane : 0) + 27 * d;
            double nb[3][3], nd[3][3];  // [i][b]: value and x-derivative channels
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                rev_b(R[i], R[i + 3], R[i + 6], nb[i]);
                rev_d_add(R[9 + i], R[12 + i], R[15 + i], nb[i]);
                rev_b(R[18 + i], R[21 + i], R[24 + i], nd[i]);
            }
            __syncwarp();  // lanes without a plane have read lane 0's: it is overwritten only now
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                double n[3];
                rev_b(nb[0][b], nb[1][b], nb[2][b], n);
                rev_d_add(nd[0][b], nd[1][b], nd[2][b], n);
                const double prev = __shfl_up_sync(full, n[2], 3);
                if (take[b]) n[0] += prev;
                if (live) R[3 * b] = n[0], R[3 * b + 1] = n[1], R[3 * b + 2] = n[2];
            }
        }
        __syncwarp();
    }
    wait_for_previous();
#pragma unroll 1
    for (int i0 = lane; i0 < ENTRIES; i0 += 32 * BATCH) {
        uint32_t e[BATCH];
        int id[BATCH];
        double v[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; ++i) e[i] = i0 + 32 * i < ENTRIES ? kEntries.e[i0 + 32 * i] : 0u;
#pragma unroll
        for (int i = 0; i < BATCH; ++i) {
            id[i] = i0 + 32 * i < ENTRIES ? *reinterpret_cast<const int*>(reinterpret_cast<const char*>(sId) + id_offset(e[i])) : -1;
            v[i] = *reinterpret_cast<const double*>(reinterpret_cast<const char*>(S) + value_offset(e[i]));
        }
#pragma unroll
        for (int i = 0; i < BATCH; ++i)
            if (id[i] >= 0) red_add(p.out + dof(id[i], e[i]), v[i]);
    }
}

template <int RHEO, bool BF, int OP>
static void launch_t(const DomainParams& p, cudaStream_t s) {
    auto kern = k_hex27_planes<RHEO, BF, OP>;
    ensure_kernel_smem((const void*)kern, q2::smem_bytes());
    const int64_t per = q2::WARPS * q2::CELLS;
    launch_domain(kern, (p.ncells + per - 1) / per, q2::WARPS * 32, q2::smem_bytes(), s, p);
}

template <int RHEO>
static void launch_r(const DomainParams& p, bool bf, int op, cudaStream_t s) {
    if (op != OP_RESIDUAL) launch_t<RHEO, false, OP_JACOBIAN_ACTION>(p, s);
    else if (bf) launch_t<RHEO, true, OP_RESIDUAL>(p, s);
    else launch_t<RHEO, false, OP_RESIDUAL>(p, s);
}

void launch_hex27(const DomainParams& p, int rheo, bool bf, int op, cudaStream_t s) {
    if (rheo == RHEO_ILE) launch_r<RHEO_ILE>(p, bf, op, s);
    else launch_r<RHEO_GENMAXWELL>(p, bf, op, s);
}

}  // namespace plb
