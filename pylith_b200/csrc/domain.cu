// Domain cell-loop kernels (thread per cell, atomic scatter) and their launchers.
#include <algorithm>
#include <atomic>

#include "domain_kernels.cuh"
#include "internal.hpp"
#include "launch.hpp"

namespace plb {

// Residual (OP_RESIDUAL) or matrix-free Jacobian action (OP_JACOBIAN_ACTION) of one
// domain integrator; FP64 throughout.
template <int CELL, int RHEO, bool BF, int OP>
__global__ void __launch_bounds__(128) k_domain_apply(DomainParams p) {
    using E = Elem<CELL>;
    using L = AuxLayout<RHEO, BF>;
    const AuxOffsets<RHEO, BF> aoff;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < p.ncells;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t mc = p.cell_ids ? p.cell_ids[c] : c;
        const int32_t* cn = p.cells + mc * E::nen;
        int nodes[E::nen];
#pragma unroll
        for (int n = 0; n < E::nen; ++n) nodes[n] = cn[n];
        double X[E::ngeom][3];
#pragma unroll
        for (int k = 0; k < E::ngeom; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * (int64_t)nodes[E::corner(k)] + i];
        const double* field = OP == OP_RESIDUAL ? p.u : p.v;
        double a[L::size] = {};
        L::load_cell(p, c, a);
        double acc[E::nen * 3];
#pragma unroll
        for (int i = 0; i < E::nen * 3; ++i) acc[i] = 0.0;
#pragma unroll 1
        for (int q = 0; q < E::nq; ++q) {
            Geom g;
            E::geom(X, q, &g);
            if (!(g.detJ > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
            double s[3] = {0, 0, 0}, s_x[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            for (int n = 0; n < E::nen; ++n) {
                double gr[3];
                E::grad(g, q, n, gr);
                const double* un = field + 3 * (int64_t)nodes[n];
                const double u0 = un[0], u1 = un[1], u2 = un[2];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    s_x[0 + d] += u0 * gr[d];
                    s_x[3 + d] += u1 * gr[d];
                    s_x[6 + d] += u2 * gr[d];
                }
            }
            if (OP == OP_RESIDUAL) L::load_qp(p, c, q, E::nq, a);  // the tangents read no state
            double x[3] = {0, 0, 0};
            double f0[3] = {0, 0, 0}, f1[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            if (OP == OP_RESIDUAL) {
                if (BF) {
                    const int sOff[1] = {0}, sOff_x[1] = {0};
                    pw::g0v_bodyforce<double>(3, 1, L::numA, sOff, sOff_x, s, nullptr, s_x, aoff.v,
                                              nullptr, a, nullptr, nullptr, p.t, x,
                                              p.num_constants, p.constants, f0);
                }
                call_f1<RHEO>(L::numA, aoff.v, a, s, s_x, p, x, f1);
            } else {
                double Jf3[81];
#pragma unroll
                for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
                call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
                // f1[f][df] = sum_{g,dg} Jf3[f][g][df][dg] dv_g/dx_dg
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int df = 0; df < 3; ++df) {
                        double acc1 = 0.0;
#pragma unroll
                        for (int gg = 0; gg < 3; ++gg)
#pragma unroll
                            for (int dg = 0; dg < 3; ++dg)
                                acc1 += Jf3[((f * 3 + gg) * 3 + df) * 3 + dg] * s_x[gg * 3 + dg];
                        f1[f * 3 + df] = acc1;
                    }
            }
#pragma unroll
            for (int n = 0; n < E::nen; ++n) {
                double gr[3];
                E::grad(g, q, n, gr);
                const double ph = BF && OP == OP_RESIDUAL ? E::phi(q, n) : 0.0;
#pragma unroll
                for (int cc = 0; cc < 3; ++cc)
                    acc[n * 3 + cc] += g.wdetJ * (f0[cc] * ph + f1[cc * 3 + 0] * gr[0] +
                                                  f1[cc * 3 + 1] * gr[1] + f1[cc * 3 + 2] * gr[2]);
            }
        }
#pragma unroll
        for (int n = 0; n < E::nen; ++n)
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) red_add(&p.out[3 * (int64_t)nodes[n] + cc], acc[n * 3 + cc]);
    }
}

// FP32 Jacobian action: FP64 geometry per cell, FP32 operand/accumulation.
template <int CELL, int RHEO>
__global__ void __launch_bounds__(128) k_domain_jv_f32(DomainParams p) {
    using E = Elem<CELL>;
    using L = AuxLayout<RHEO, false>;
    const AuxOffsets<RHEO, false> aoff;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < p.ncells;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t mc = p.cell_ids ? p.cell_ids[c] : c;
        const int32_t* cn = p.cells + mc * E::nen;
        int nodes[E::nen];
#pragma unroll
        for (int n = 0; n < E::nen; ++n) nodes[n] = cn[n];
        double X[E::ngeom][3];
#pragma unroll
        for (int k = 0; k < E::ngeom; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * (int64_t)nodes[E::corner(k)] + i];
        double a[L::size] = {};
        L::load_cell(p, c, a);
        float acc[E::nen * 3];
#pragma unroll
        for (int i = 0; i < E::nen * 3; ++i) acc[i] = 0.0f;
#pragma unroll 1
        for (int q = 0; q < E::nq; ++q) {
            Geom g;
            E::geom(X, q, &g);
            float s_x[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            for (int n = 0; n < E::nen; ++n) {
                double grd[3];
                E::grad(g, q, n, grd);
                const float gr[3] = {(float)grd[0], (float)grd[1], (float)grd[2]};
                const float* vn = p.v32 + 3 * (int64_t)nodes[n];
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    s_x[0 + d] += vn[0] * gr[d];
                    s_x[3 + d] += vn[1] * gr[d];
                    s_x[6 + d] += vn[2] * gr[d];
                }
            }
            // the tangents (Jf3vu of both rheologies) read no per-point state
            double x[3] = {0, 0, 0};
            double Jf3d[81];
#pragma unroll
            for (int i = 0; i < 81; ++i) Jf3d[i] = 0.0;
            call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3d);
            float f1[9];
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int df = 0; df < 3; ++df) {
                    float acc1 = 0.0f;
#pragma unroll
                    for (int gg = 0; gg < 3; ++gg)
#pragma unroll
                        for (int dg = 0; dg < 3; ++dg)
                            acc1 += (float)Jf3d[((f * 3 + gg) * 3 + df) * 3 + dg] * s_x[gg * 3 + dg];
                    f1[f * 3 + df] = acc1;
                }
            const float w = (float)g.wdetJ;
#pragma unroll
            for (int n = 0; n < E::nen; ++n) {
                double grd[3];
                E::grad(g, q, n, grd);
#pragma unroll
                for (int cc = 0; cc < 3; ++cc)
                    acc[n * 3 + cc] += w * (f1[cc * 3 + 0] * (float)grd[0] + f1[cc * 3 + 1] * (float)grd[1] +
                                            f1[cc * 3 + 2] * (float)grd[2]);
            }
        }
#pragma unroll
        for (int n = 0; n < E::nen; ++n)
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) red_add(&p.out32[3 * (int64_t)nodes[n] + cc], acc[n * 3 + cc]);
    }
}

// DMProjectFieldLocal at quadrature points for the generalized Maxwell state: new viscous
// strain from the previous viscous and total strain, then the new total strain; both kernels
// see the previous state (IntegratorDomain.cc:555-590), written back in place.
template <int CELL>
__global__ void __launch_bounds__(128) k_domain_update_state(DomainParams p) {
    using E = Elem<CELL>;
    using L = AuxLayout<RHEO_GENMAXWELL, false>;
    const AuxOffsets<RHEO_GENMAXWELL, false> aoff;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < p.ncells;
         c += (int64_t)gridDim.x * blockDim.x) {
        const int64_t mc = p.cell_ids ? p.cell_ids[c] : c;
        const int32_t* cn = p.cells + mc * E::nen;
        int nodes[E::nen];
#pragma unroll
        for (int n = 0; n < E::nen; ++n) nodes[n] = cn[n];
        double X[E::ngeom][3];
#pragma unroll
        for (int k = 0; k < E::ngeom; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * (int64_t)nodes[E::corner(k)] + i];
        // Q1: coordinates and field relative to the first corner, as in hex8.cu (the basis gradients sum to
        // zero), so that no large coordinates or displacements cancel
        double u0[3] = {0, 0, 0};
        if (CELL == HEX8) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                u0[i] = p.u[3 * (int64_t)nodes[0] + i];
#pragma unroll
                for (int k = E::ngeom - 1; k >= 0; --k) X[k][i] -= X[0][i];
            }
        }
        double a[L::size] = {};
        L::load_cell(p, c, a);
#pragma unroll 1
        for (int q = 0; q < E::nq; ++q) {
            Geom g;
            E::geom(X, q, &g);
            double s_x[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            for (int n = 0; n < E::nen; ++n) {
                double gr[3];
                E::grad(g, q, n, gr);
                const double* un = p.u + 3 * (int64_t)nodes[n];
                const double u[3] = {un[0] - u0[0], un[1] - u0[1], un[2] - u0[2]};
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    s_x[0 + d] += u[0] * gr[d];
                    s_x[3 + d] += u[1] * gr[d];
                    s_x[6 + d] += u[2] * gr[d];
                }
            }
            L::load_qp(p, c, q, E::nq, a);
            const int sOff[1] = {0}, sOff_x[1] = {0};
            double x[3] = {0, 0, 0};
            double visc[18], tot[6];
            pw::gm3d_viscous_strain<double>(3, 1, L::numA, sOff, sOff_x, nullptr, nullptr, s_x,
                                            aoff.v, nullptr, a, nullptr, nullptr, p.t, x,
                                            p.num_constants, p.constants, visc);
            pw::el3d_strain_vector<double>(3, 1, L::numA, sOff, sOff_x, nullptr, nullptr, s_x,
                                           aoff.v, nullptr, a, nullptr, nullptr, p.t, x,
                                           p.num_constants, p.constants, tot);
#pragma unroll
            for (int k = 0; k < 18; ++k) p.visc[((int64_t)k * E::nq + q) * p.ncells + c] = visc[k];
#pragma unroll
            for (int k = 0; k < 6; ++k) p.total[((int64_t)k * E::nq + q) * p.ncells + c] = tot[k];
        }
    }
}

// One project kernel at a point with gradient s_x and aux a.
template <int RHEO>
PL_D void derived_point(const DomainParams& p, int kind, const double* s_x, const double* a, double (&o)[6]) {
    using L = AuxLayout<RHEO, false>;
    const AuxOffsets<RHEO, false> aoff;
    const int sOff[1] = {0}, sOff_x[1] = {0};
    double x[3] = {0, 0, 0};
    if (kind == K_EL_STRAIN_VECTOR)
        pw::el3d_strain_vector<double>(3, 1, L::numA, sOff, sOff_x, nullptr, nullptr, s_x, aoff.v, nullptr, a, nullptr, nullptr, p.t,
                                       x, p.num_constants, p.constants, o);
    else if (RHEO == RHEO_ILE && kind == K_ILE_STRESS_VECTOR)
        pw::ile3d_stress_vector<double>(3, 1, L::numA, sOff, sOff_x, nullptr, nullptr, s_x, aoff.v, nullptr, a, nullptr, nullptr, p.t,
                                        x, p.num_constants, p.constants, o);
    else if (RHEO == RHEO_GENMAXWELL && kind == K_GM_STRESS_VECTOR)
        pw::gm3d_stress_vector<double>(3, 1, L::numA, sOff, sOff_x, nullptr, nullptr, s_x, aoff.v, nullptr, a, nullptr, nullptr, p.t,
                                       x, p.num_constants, p.constants, o);
}

// Derived fields of basis order 0 (IntegratorDomain::_computeDerivedField,
// IntegratorDomain.cc:596-630, with PyLith's default basis order 0 for cauchy_stress and
// cauchy_strain, DerivedSubfieldsElasticity.py:42-44): each registered project kernel evaluated
// at the cell centroid, out[c][6 * k + i] for kernel k. A generalized-Maxwell stress reads the
// state of the cell's single quadrature point (P1 tetrahedra only).
//
// Bound: L2, at first by the stores: a thread's six values per kernel lie in a row of its own, so a
// warp's store touched 32 sectors. Rows are staged in shared memory and a warp stores its cells' rows
// with consecutive lanes on consecutive doubles; node ids, coordinates and field are read before
// they are used: stress and strain of 100,345 Q1 hexahedra 12.9 -> 8.2 us with the nodes in L2; with L2
// cold 36,720 cells 11.5 -> 9.9, 196,608 24.6 -> 18.4.
constexpr int kDerivedThreads = 128;
constexpr int kDerivedRow = 6 * 4 + 1;  // values of a cell at most; odd, so a warp's accesses spread over the banks
template <int CELL, int RHEO>
__global__ void __launch_bounds__(kDerivedThreads) k_domain_derived(DomainParams p, DerivedSpec spec) {
    using E = Elem<CELL>;
    using L = AuxLayout<RHEO, false>;
    constexpr int AHEAD = E::nen <= 8 ? E::nen : 1;  // nodes held in registers
    __shared__ double rows[kDerivedThreads * kDerivedRow];
    const int nout = 6 * spec.n, lane = threadIdx.x & 31;
    double* const wrow = rows + (threadIdx.x - lane) * kDerivedRow;  // the warp's rows
    for (int64_t c0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; c0 < p.ncells;
         c0 += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = c0 + lane;
        if (c < p.ncells) {
            const int64_t mc = p.cell_ids ? p.cell_ids[c] : c;
            const int32_t* cn = p.cells + mc * E::nen;
            int nd[AHEAD];
            double U[AHEAD][3];
            if (E::nen <= 8) {
#pragma unroll
                for (int n = 0; n < AHEAD; ++n) nd[n] = cn[n];
#pragma unroll
                for (int n = 0; n < AHEAD; ++n)
#pragma unroll
                    for (int i = 0; i < 3; ++i) U[n][i] = p.u[3 * (int64_t)nd[n] + i];
            }
            double X[E::ngeom][3];
#pragma unroll
            for (int k = 0; k < E::ngeom; ++k) {
                const int64_t node = E::nen <= 8 ? nd[k < AHEAD ? k : 0] : cn[E::corner(k)];
#pragma unroll
                for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * node + i];
            }
            double a[L::size] = {};
            L::load_cell(p, c, a);
            L::load_qp(p, c, 0, E::nq, a);
            Geom g;
            E::centre_geom(X, &g);
            if (!(g.detJ > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
            double s_x[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
            auto add = [&](int n, const double* un) {
                double gr[3];
                E::centre_grad(g, n, gr);
#pragma unroll
                for (int d = 0; d < 3; ++d) {
                    s_x[0 + d] += un[0] * gr[d];
                    s_x[3 + d] += un[1] * gr[d];
                    s_x[6 + d] += un[2] * gr[d];
                }
            };
            if (E::nen <= 8) {
#pragma unroll
                for (int n = 0; n < AHEAD; ++n) add(n, U[n]);
            } else {
                for (int n = 0; n < E::nen; ++n) add(n, p.u + 3 * (int64_t)cn[n]);
            }
            for (int k = 0; k < spec.n; ++k) {
                double o[6] = {0, 0, 0, 0, 0, 0};
                derived_point<RHEO>(p, spec.kind[k], s_x, a, o);
#pragma unroll
                for (int i = 0; i < 6; ++i) wrow[lane * kDerivedRow + 6 * k + i] = o[i];
            }
        }
        __syncwarp();
        const int count = (int)min((int64_t)32, p.ncells - c0) * nout;
        double* out = p.out + c0 * nout;
        int row = lane / nout, col = lane - row * nout;  // of entry e
        const int drow = 32 / nout, dcol = 32 - drow * nout;
        for (int e = lane; e < count; e += 32) {
            out[e] = wrow[row * kDerivedRow + col];
            row += drow, col += dcol;
            if (col >= nout) ++row, col -= nout;
        }
        __syncwarp();
    }
}

// The same without staging, for Q2 meshes of up to a block per multiprocessor, where the row stores do not
// count and the shorter code does: 384 to 11,520 cells, L2 cold, 12.3 us and 14.3 staged; 24,576 cells and
// four kernels 10.5 us and 8.3 staged.
template <int CELL, int RHEO>
__global__ void __launch_bounds__(kDerivedThreads) k_domain_derived_direct(DomainParams p, DerivedSpec spec) {
    using E = Elem<CELL>;
    using L = AuxLayout<RHEO, false>;
    const int nout = 6 * spec.n;
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= p.ncells) return;
    const int32_t* cn = p.cells + (p.cell_ids ? p.cell_ids[c] : c) * E::nen;
    double X[E::ngeom][3];
#pragma unroll
    for (int k = 0; k < E::ngeom; ++k)
#pragma unroll
        for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * (int64_t)cn[E::corner(k)] + i];
    Geom g;
    E::centre_geom(X, &g);
    if (!(g.detJ > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
    double s_x[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    for (int n = 0; n < E::nen; ++n) {
        double gr[3];
        E::centre_grad(g, n, gr);
        const double* un = p.u + 3 * (int64_t)cn[n];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            s_x[0 + d] += un[0] * gr[d];
            s_x[3 + d] += un[1] * gr[d];
            s_x[6 + d] += un[2] * gr[d];
        }
    }
    double a[L::size] = {};
    L::load_cell(p, c, a);
    L::load_qp(p, c, 0, E::nq, a);
    for (int k = 0; k < spec.n; ++k) {
        double o[6] = {0, 0, 0, 0, 0, 0};
        derived_point<RHEO>(p, spec.kind[k], s_x, a, o);
#pragma unroll
        for (int i = 0; i < 6; ++i) p.out[c * nout + 6 * k + i] = o[i];
    }
}

static int grid_for(int64_t n, int threads) {
    const int64_t blocks = (n + threads - 1) / threads;
    return (int)(blocks < 148 * 64 ? (blocks > 0 ? blocks : 1) : 148 * 64);
}

template <int CELL, int RHEO, bool BF>
static void launch_apply_t(const DomainParams& p, int op, cudaStream_t s) {
    const int th = 128;
    if (op == OP_RESIDUAL)
        k_domain_apply<CELL, RHEO, BF, OP_RESIDUAL><<<grid_for(p.ncells, th), th, 0, s>>>(p);
    else
        k_domain_apply<CELL, RHEO, false, OP_JACOBIAN_ACTION><<<grid_for(p.ncells, th), th, 0, s>>>(p);
    count_launch();
}

template <int CELL>
static void launch_apply_cell(const DomainParams& p, int rheo, bool bf, int op, cudaStream_t s) {
    if (rheo == RHEO_ILE) {
        if (bf) launch_apply_t<CELL, RHEO_ILE, true>(p, op, s);
        else launch_apply_t<CELL, RHEO_ILE, false>(p, op, s);
    } else {
        if (bf) launch_apply_t<CELL, RHEO_GENMAXWELL, true>(p, op, s);
        else launch_apply_t<CELL, RHEO_GENMAXWELL, false>(p, op, s);
    }
}

// Zeros ahead of a cell kernel that starts while they are written, so that neither the launch nor the
// kernel's staging and arithmetic wait for a memset. A multiprocessor keeps its split of L1 and shared
// memory while it is busy, so the next kernel's blocks start under this kernel's: SHARED asks for the
// most shared memory. Measured on B200 against a memset in between: residual and action of 1,179,648
// tetrahedra 75.8 -> 70.5 us (73.9 without SHARED), with the FP32 action of 54,737 tetrahedra 24.6 -> 21.5
// and of 663,552 Q1 hexahedra 220 -> 209, of 4,096 Q1 hexahedra 16.4 -> 14.5, of 262,144 Q2 hexahedra
// 458 -> 450. The generalized-Maxwell residual keeps the memset: with the state update and the fault
// 124 us on 82,944 cells, 137 this way whatever the split (cause not found).
template <typename T, bool SHARED>
static __global__ void k_zero_output(T* __restrict__ out, int64_t n) {
    asm volatile("griddepcontrol.launch_dependents;");
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) out[i] = T(0);
}
template <typename T, bool SHARED>
static void zero_output_t(T* out, int64_t n, cudaStream_t s) {
    if (SHARED) {  // once per device (a 64-bit word holds them all)
        static std::atomic<uint64_t> done{0};
        int dev = 0;
        cudaGetDevice(&dev);
        if (!(done.load() >> (dev & 63) & 1)) {
            cudaFuncSetAttribute((const void*)k_zero_output<T, SHARED>, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 cudaSharedmemCarveoutMaxShared);
            done.fetch_or((uint64_t)1 << (dev & 63));
        }
    }
    k_zero_output<T, SHARED><<<(unsigned)std::min<int64_t>((n + 255) / 256, (int64_t)sm_count() * 8), 256, 0, s>>>(out, n);
    count_launch();
}
template <typename T>
static bool zero_any(T* out, int64_t n, bool early, bool shared, cudaStream_t s) {
    // A memset where nothing starts under it (a launch of its own then costs 0.5 to 1 us more: atomic
    // scatter on 2,652 tetrahedra 6.6 and 7.2 us, FP32 action of 1,188 Q2 hexahedra 12.4 and 13.4) and
    // for outputs of one block, ready before the next launch either way (FP32 action of 6 tetrahedra 6.3
    // and 6.8 us; of 750, 648 values, 8.2 and 6.6).
    early = early && n > 256;
    if (!early) cudaMemsetAsync(out, 0, n * sizeof(T), s);
    else if (shared) zero_output_t<T, true>(out, n, s);
    else zero_output_t<T, false>(out, n, s);
    return early;
}
bool zero_output(double* out, int64_t n, bool early, bool shared, cudaStream_t s) { return zero_any(out, n, early, shared, s); }
bool zero_output(float* out, int64_t n, bool early, bool shared, cudaStream_t s) { return zero_any(out, n, early, shared, s); }

void launch_domain_apply_atomic(const DomainParams& p, int cell, int rheo, bool bf, int op,
                                cudaStream_t s) {
    if (p.ncells == 0) return;
    if (cell == TET4) launch_apply_cell<TET4>(p, rheo, bf, op, s);
    else if (cell == HEX8) launch_apply_cell<HEX8>(p, rheo, bf, op, s);
    else launch_apply_cell<HEX27>(p, rheo, bf, op, s);
}

void launch_domain_jv_f32_atomic(const DomainParams& p, int cell, int rheo, cudaStream_t s) {
    if (p.ncells == 0) return;
    const int th = 128;
    const int gr = grid_for(p.ncells, th);
#define PLB_F32(C, R) k_domain_jv_f32<C, R><<<gr, th, 0, s>>>(p)
    if (cell == TET4) { if (rheo == RHEO_ILE) PLB_F32(TET4, RHEO_ILE); else PLB_F32(TET4, RHEO_GENMAXWELL); }
    else if (cell == HEX8) { if (rheo == RHEO_ILE) PLB_F32(HEX8, RHEO_ILE); else PLB_F32(HEX8, RHEO_GENMAXWELL); }
    else { if (rheo == RHEO_ILE) PLB_F32(HEX27, RHEO_ILE); else PLB_F32(HEX27, RHEO_GENMAXWELL); }
#undef PLB_F32
    count_launch();
}

void launch_domain_update_state(const DomainParams& p, int cell, cudaStream_t s) {
    if (p.ncells == 0) return;
    const int th = 128;
    const int gr = grid_for(p.ncells, th);
    // Q1: a thread per cell with the state copied ahead (hex8.cu) while the state (192 doubles a cell) fits
    // L2, where latency counts; larger meshes stream it from HBM and the loop over the points is the
    // faster one: 10.5 and 14.5 us at 9,384 cells, 16.6 and 18.7 at 36,720; 76.0 and 71.7 at 104,000, 264
    // and 244 at 384,000.
    if (cell == HEX8 && p.ncells * 192 * (int64_t)sizeof(double) <= ((int64_t)128 << 20)) {
        launch_hex8_update_state(p, s);
        return;
    }
    if (cell == TET4) k_domain_update_state<TET4><<<gr, th, 0, s>>>(p);
    else if (cell == HEX8) k_domain_update_state<HEX8><<<gr, th, 0, s>>>(p);
    else k_domain_update_state<HEX27><<<gr, th, 0, s>>>(p);
    count_launch();
}

void launch_domain_derived(const DomainParams& p, int cell, int rheo, const DerivedSpec& spec, cudaStream_t s) {
    if (p.ncells == 0) return;
    const int th = kDerivedThreads;
    const int gr = grid_for(p.ncells, th);
    if (cell == HEX27 && p.ncells <= (int64_t)th * sm_count()) {
        const int blocks = (int)((p.ncells + th - 1) / th);
        if (rheo == RHEO_GENMAXWELL) k_domain_derived_direct<HEX27, RHEO_GENMAXWELL><<<blocks, th, 0, s>>>(p, spec);
        else k_domain_derived_direct<HEX27, RHEO_ILE><<<blocks, th, 0, s>>>(p, spec);
    } else if (rheo == RHEO_GENMAXWELL) {
        if (cell == TET4) k_domain_derived<TET4, RHEO_GENMAXWELL><<<gr, th, 0, s>>>(p, spec);
        else if (cell == HEX8) k_domain_derived<HEX8, RHEO_GENMAXWELL><<<gr, th, 0, s>>>(p, spec);
        else k_domain_derived<HEX27, RHEO_GENMAXWELL><<<gr, th, 0, s>>>(p, spec);
    } else {
        if (cell == TET4) k_domain_derived<TET4, RHEO_ILE><<<gr, th, 0, s>>>(p, spec);
        else if (cell == HEX8) k_domain_derived<HEX8, RHEO_ILE><<<gr, th, 0, s>>>(p, spec);
        else k_domain_derived<HEX27, RHEO_ILE><<<gr, th, 0, s>>>(p, spec);
    }
    count_launch();
}

}  // namespace plb
