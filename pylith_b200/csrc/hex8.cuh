// Q1 hexahedra with one thread per cell: the trilinear geometry, the field gradient at the 2x2x2
// Gauss points and the test-function contraction by edge differences, all in registers.
//
// With P(a, b) = V0 + w_k (V1 - V0) the nodes of the plane zeta = point k (V0, V1: bottom and top
// nodes), the reference gradient at point (i, j, k) is
//     d/dxi   = x0 + w_j c,  x0 = P10 - P00,          d/deta = y0 + w_i c,  y0 = P01 - P00,
//     d/dzeta = bilinear in the vertical edges V1 - V0,       c = P11 - P10 - P01 + P00
// (reference cell [0, 1]^3, so every entry is twice the one on [-1, 1]^3), 42 operations per
// component for the 8 points, and the reverse contraction is its transpose. With C = det(J) J^{-1}
// the gradient is G C / det and the test weights are C f1, so each point takes one reciprocal. On
// [0, 1]^3 a Gauss weight is 1/8, applied to the node sums at the end.
#pragma once

#include <cuda_pipeline.h>

#include <type_traits>

#include "domain_kernels.cuh"

namespace plb {

// Coordinate of 2-point Gauss point p on [0, 1].
template <typename T>
PL_D T hex8_w(int p) {
    return p == 0 ? T(0.21132486540518711775) : T(0.78867513459481288225);
}

// Position in the lattice of the bottom nodes, index a + 2 b, of corner c in {0, 1, 2, 3}.
PL_D constexpr int hex8_ab(int c) { return c == 0 ? 0 : (c == 1 ? 1 : (c == 2 ? 3 : 2)); }

// The cell's nodes as the sweep reads them: bottom nodes V0[a + 2 b] relative to corner 0 (V0[0] is
// zero and not read) and vertical edges Dz, 6 components each (0-2 coordinates, differenced in
// FP64, 3-5 field). Only differences enter, so no large coordinates or displacements cancel.
template <typename T>
struct Hex8Nodes {
    T V0[4][6], Dz[4][6];
};

PL_D void hex8_nodes(const DomainParams& p, int64_t c, int (&nodes)[8]) {
    const int4* cn = reinterpret_cast<const int4*>(p.cells + 8 * (p.cell_ids ? (int64_t)p.cell_ids[c] : c));
    const int4 lo = cn[0], hi = cn[1];
    nodes[0] = lo.x, nodes[1] = lo.y, nodes[2] = lo.z, nodes[3] = lo.w;
    nodes[4] = hi.x, nodes[5] = hi.y, nodes[6] = hi.z, nodes[7] = hi.w;
}

template <typename T, typename F>
PL_D void hex8_load(const double* __restrict__ coords, const F* __restrict__ field, const int (&nodes)[8], Hex8Nodes<T>& h) {
    double X[8][3];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) X[c][d] = coords[3 * (int64_t)nodes[c] + d];
    T U[8][3];
#pragma unroll
    for (int c = 0; c < 8; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) U[c][d] = (T)field[3 * (int64_t)nodes[c] + d];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const int ab = hex8_ab(c);
            h.V0[ab][d] = (T)(X[c][d] - X[0][d]);
            h.Dz[ab][d] = (T)(X[c + 4][d] - X[c][d]);
            h.V0[ab][3 + d] = U[c][d] - U[0][d];
            h.Dz[ab][3 + d] = U[c + 4][d] - U[c][d];
        }
}

// Visits the 8 Gauss points (q = i + 2 j + 4 k): pt(q, G, C, det, W) gets the reference gradient
// of the field G[component][direction], the cofactors C = det J^{-1} and det > 0 (on [0, 1]^3), and
// sets the test weights W[component][direction] = sum_e C[direction][e] f1[component][e] (unread
// unless REVERSE) and, with VALUE, W0[component], the weight of the basis values. g[8 corners][3]:
// the node sums, before the factor 1/8.
template <bool REVERSE, bool VALUE, typename T, typename Point>
PL_D void hex8_sweep(const Hex8Nodes<T>& h, unsigned int* err, T (&g)[8][3], Point pt) {
    // d/dP summed over the planes, its w_k-weighted sum, d/dzeta weights
    T g0[4][3], gz[4][3], az[2][2][3];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const T wk = hex8_w<T>(k);
        T x0[6], y0[6], cc[6];
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            const T p00 = wk * h.Dz[0][f], p10 = h.V0[1][f] + wk * h.Dz[1][f];
            const T p01 = h.V0[2][f] + wk * h.Dz[2][f], p11 = h.V0[3][f] + wk * h.Dz[3][f];
            x0[f] = p10 - p00;
            y0[f] = p01 - p00;
            cc[f] = (p11 - p01) - x0[f];
        }
        T ax[2][3], ay[2][3], av[4][3];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const T wj = hex8_w<T>(j);
            T xj[6], z0[6], z1[6];
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                xj[f] = x0[f] + wj * cc[f];
                z0[f] = h.Dz[0][f] + wj * (h.Dz[2][f] - h.Dz[0][f]);
                z1[f] = h.Dz[1][f] + wj * (h.Dz[3][f] - h.Dz[1][f]);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const T wi = hex8_w<T>(i);
                T J[3][3], G[3][3];  // [component][direction]
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    J[d][0] = xj[d];
                    J[d][1] = y0[d] + wi * cc[d];
                    J[d][2] = z0[d] + wi * (z1[d] - z0[d]);
                    G[d][0] = xj[3 + d];
                    G[d][1] = y0[3 + d] + wi * cc[3 + d];
                    G[d][2] = z0[3 + d] + wi * (z1[3 + d] - z0[3 + d]);
                }
                T C[3][3];
                C[0][0] = J[1][1] * J[2][2] - J[1][2] * J[2][1];
                C[0][1] = J[0][2] * J[2][1] - J[0][1] * J[2][2];
                C[0][2] = J[0][1] * J[1][2] - J[0][2] * J[1][1];
                C[1][0] = J[1][2] * J[2][0] - J[1][0] * J[2][2];
                C[1][1] = J[0][0] * J[2][2] - J[0][2] * J[2][0];
                C[1][2] = J[0][2] * J[1][0] - J[0][0] * J[1][2];
                C[2][0] = J[1][0] * J[2][1] - J[1][1] * J[2][0];
                C[2][1] = J[0][1] * J[2][0] - J[0][0] * J[2][1];
                C[2][2] = J[0][0] * J[1][1] - J[0][1] * J[1][0];
                const T det = J[0][0] * C[0][0] + J[0][1] * C[1][0] + J[0][2] * C[2][0];
                if (!(det > T(0))) flag_error(err, CHECK_NONPOSITIVE_DETJ);
                T W[3][3], W0[3];
                pt(i + 2 * j + 4 * k, G, C, det, W, W0);
                if (!REVERSE) continue;
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    ax[j][d] = i == 0 ? W[d][0] : ax[j][d] + W[d][0];
                    ay[i][d] = j == 0 ? W[d][1] : ay[i][d] + W[d][1];
                    az[j][i][d] = k == 0 ? W[d][2] : az[j][i][d] + W[d][2];
                    if (VALUE) {
                        const T u1 = wi * W0[d], u0 = W0[d] - u1;
                        const T v10 = wj * u0, v11 = wj * u1;
                        const bool first = i == 0 && j == 0;
                        av[0][d] = first ? u0 - v10 : av[0][d] + (u0 - v10);
                        av[1][d] = first ? u1 - v11 : av[1][d] + (u1 - v11);
                        av[2][d] = first ? v10 : av[2][d] + v10;
                        av[3][d] = first ? v11 : av[3][d] + v11;
                    }
                }
            }
        }
        if (!REVERSE) continue;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const T gx = ax[0][d] + ax[1][d], gy = ay[0][d] + ay[1][d];
            const T gc = hex8_w<T>(0) * (ax[0][d] + ay[0][d]) + hex8_w<T>(1) * (ax[1][d] + ay[1][d]);
            T gp[4] = {gc - gx - gy, gx - gc, gy - gc, gc};
#pragma unroll
            for (int ab = 0; ab < 4; ++ab) {
                if (VALUE) gp[ab] += av[ab][d];
                g0[ab][d] = k == 0 ? gp[ab] : g0[ab][d] + gp[ab];
                gz[ab][d] = k == 0 ? wk * gp[ab] : gz[ab][d] + wk * gp[ab];
            }
        }
    }
    if (!REVERSE) return;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const T w0 = hex8_w<T>(0), w1 = hex8_w<T>(1);
        // transpose of the bilinear interpolation of the vertical edges: along i, then along j
        T e[2][2];  // [j][a]
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            e[j][1] = w0 * az[j][0][d] + w1 * az[j][1][d];
            e[j][0] = w1 * az[j][0][d] + w0 * az[j][1][d];
        }
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            gz[a][d] += w1 * e[0][a] + w0 * e[1][a];
            gz[2 + a][d] += w0 * e[0][a] + w1 * e[1][a];
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            g[c][d] = g0[hex8_ab(c)][d] - gz[hex8_ab(c)][d];
            g[c + 4][d] = gz[hex8_ab(c)][d];
        }
    }
}

// Adds the node sums g of the calling lane's cell into out. Where the next lane's cell continues
// this one along xi (its corners 0, 3, 4, 7 are this one's 1, 2, 5, 6, as in boxes numbered along
// x), the shared face's sums travel there by shuffle and are added once: up to half of the
// reductions into L2 less. Every lane of the warp calls it (dead cells with nodes -1).
template <typename T>
PL_D void hex8_scatter(const int (&nodes)[8], T (&g)[8][3], T* out) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    bool skip[8] = {};
    constexpr int from[4] = {1, 2, 5, 6}, to[4] = {0, 3, 4, 7};
#pragma unroll
    for (int f = 0; f < 4; ++f) {
        const int nb = __shfl_down_sync(full, nodes[to[f]], 1);
        const bool give = lane < 31 && nb == nodes[from[f]];
        const bool take = __shfl_up_sync(full, (int)give, 1) && lane > 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const T v = __shfl_up_sync(full, g[from[f]][d], 1);
            if (take) g[to[f]][d] += v;
        }
        skip[from[f]] = give;
    }
#pragma unroll
    for (int c = 0; c < 8; ++c)
        if (nodes[c] >= 0 && !skip[c])
#pragma unroll
            for (int d = 0; d < 3; ++d) red_add(out + 3 * (int64_t)nodes[c] + d, g[c][d]);
}

// The generalized-Maxwell state of a thread's own cell, point by point (18 viscous strains, 6 total
// strains), copied three points ahead into the thread's row of shared memory: 192 doubles per cell
// are the bulk of what these kernels read, and at 8 warps per multiprocessor only copies that hold
// no registers keep enough of them in flight. A slot is filled again one point after it was read.
constexpr int kHex8Slots = 4, kHex8Row = 25;  // odd: a warp's accesses fall on distinct banks
constexpr size_t hex8_state_bytes(int threads) { return sizeof(double) * kHex8Row * kHex8Slots * threads; }
struct Hex8State {
    double* row;  // [kHex8Slots][blockDim.x][kHex8Row], this thread's row
    const DomainParams& p;
    int64_t c;
    PL_D Hex8State(double* smem, const DomainParams& params, int64_t cell) : row(smem + threadIdx.x * kHex8Row), p(params), c(cell) {
#pragma unroll
        for (int q = 0; q < kHex8Slots - 1; ++q) fetch(q);
    }
    PL_D double* slot(int q) { return row + (q % kHex8Slots) * blockDim.x * kHex8Row; }
    PL_D void fetch(int q) {
        if (q < 8) {
            double* dst = slot(q);
            const double* v = p.visc + q * p.ncells + c;
            const double* t = p.total + q * p.ncells + c;
#pragma unroll
            for (int k = 0; k < 18; ++k) __pipeline_memcpy_async(dst + k, v + (int64_t)k * 8 * p.ncells, sizeof(double));
#pragma unroll
            for (int k = 0; k < 6; ++k) __pipeline_memcpy_async(dst + 18 + k, t + (int64_t)k * 8 * p.ncells, sizeof(double));
        }
        __pipeline_commit();  // (empty at the end: the wait counts groups)
    }
    // The state of point q, visited in order 0 .. 7.
    PL_D const double* take(int q) {
        fetch(q + kHex8Slots - 1);
        __pipeline_wait_prior(kHex8Slots - 1);
        return slot(q);
    }
};
struct Hex8NoState {
    PL_D Hex8NoState(double*, const DomainParams&, int64_t) {}
};

// Residual or Jacobian action of cell c (p.ncells <= c: no cell) into p.out / p.out32; every lane
// of the warp calls it. stage: shared memory of hex8_state_bytes (generalized-Maxwell residual).
template <int RHEO, bool BF, int OP, typename T>
PL_D void hex8_cell(const DomainParams& p, int64_t c, double* stage = nullptr) {
    using L = AuxLayout<RHEO, BF>;
    constexpr bool F32 = sizeof(T) == 4;
    const AuxOffsets<RHEO, BF> aoff;
    int nodes[8];
    T g[8][3];
    const bool live = c < p.ncells;
#pragma unroll
    for (int n = 0; n < 8; ++n) nodes[n] = -1;
    if (live) {
        constexpr bool STATE = RHEO == RHEO_GENMAXWELL && OP == OP_RESIDUAL;  // the tangents read no state
        [[maybe_unused]] std::conditional_t<STATE, Hex8State, Hex8NoState> state(stage, p, c);
        hex8_nodes(p, c, nodes);
        Hex8Nodes<T> h;
        if constexpr (F32) hex8_load(p.coords, p.v32, nodes, h);
        else hex8_load(p.coords, OP == OP_RESIDUAL ? p.u : p.v, nodes, h);
        double a[L::size] = {};
        double x[3] = {0, 0, 0}, s[3] = {0, 0, 0};
        T lam = 0, mu = 0;
        if (OP == OP_JACOBIAN_ACTION && F32 && p.lm32) {
            const float2 lm = reinterpret_cast<const float2*>(p.lm32)[c];
            lam = lm.x, mu = lm.y;
        } else {
            L::load_cell(p, c, a);
            if (OP == OP_JACOBIAN_ACTION) {  // the tangents read no state: one evaluation per cell
                double Jf3[81];
#pragma unroll
                for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
                call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
                lam = (T)(-Jf3[((0 * 3 + 1) * 3 + 0) * 3 + 1]);
                mu = (T)(-Jf3[((0 * 3 + 1) * 3 + 1) * 3 + 0]);
            }
        }
        T scale = T(0.125);
        if constexpr (F32) {
            // the moduli as multiples of a power of two, applied to the node sums: modulus / det would leave
            // FP32's range where a cell is smaller than about 1e-9 m with moduli in Pa
            const unsigned e = min(max(__float_as_uint(fabsf(lam) + 2.0f * fabsf(mu)) >> 23 & 0xffu, 1u), 253u);
            const float to_one = __uint_as_float((254u - e) << 23);
            lam *= to_one, mu *= to_one;
            scale *= __uint_as_float(e << 23);
        }
        [[maybe_unused]] pw::MaxwellFactors<double> mf;
        // once per cell: evaluated at each point, the exponentials made the unrolled code overflow the
        // instruction cache (69 us against 44 for the residual of 48x48x36 cells)
        if constexpr (STATE) mf = pw::maxwell_factors(a + L::base + 2, p.constants[0]);
        hex8_sweep<true, BF && OP == OP_RESIDUAL, T>(
            h, p.err, g, [&](int q, const T(&G)[3][3], const T(&C)[3][3], T det, T(&W)[3][3], T(&W0)[3]) {
                const T rdet = T(1) / det;
                T s_x[9], f1[9] = {};
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int e = 0; e < 3; ++e)
                        s_x[f * 3 + e] = G[f][0] * C[0][e] + G[f][1] * C[1][e] + G[f][2] * C[2][e];
                if constexpr (OP == OP_JACOBIAN_ACTION) {
                    isotropic_contract<T>(lam * rdet, mu * rdet, s_x, f1);  // linear in the gradient
                } else {
#pragma unroll
                    for (int f = 0; f < 9; ++f) s_x[f] *= rdet;
                    if constexpr (BF) {
                        const int sOff[1] = {0}, sOff_x[1] = {0};
                        double f0[3] = {0, 0, 0};
                        pw::g0v_bodyforce<double>(3, 1, L::numA, sOff, sOff_x, s, nullptr, s_x, aoff.v, nullptr, a, nullptr,
                                                  nullptr, p.t, x, p.num_constants, p.constants, f0);
#pragma unroll
                        for (int d = 0; d < 3; ++d) W0[d] = det * f0[d];
                    }
                    if constexpr (STATE) {  // gm3d_f1v with the cell's factors
                        const double* st = state.take(q);
                        pw::f1_minus_stress(pw::genmaxwell_stress(a[L::base], a[L::base + 1], a + L::base + 5, st,
                                                                  pw::sym_from_vector(st + 18), mf, pw::strain(s_x)),
                                            f1);
                    } else {
                        call_f1<RHEO>(L::numA, aoff.v, a, s, s_x, p, x, f1);
                    }
                }
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        W[f][d] = C[d][0] * f1[f * 3 + 0] + C[d][1] * f1[f * 3 + 1] + C[d][2] * f1[f * 3 + 2];
            });
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
            for (int d = 0; d < 3; ++d) g[n][d] *= scale;
    }
    __syncwarp();
    wait_for_previous();  // see zero_output
    if constexpr (F32) hex8_scatter<T>(nodes, g, p.out32);
    else hex8_scatter<T>(nodes, g, p.out);
}

}  // namespace plb
