// Hexahedral cells with a group of lanes per cell: the generalized-Maxwell residual of small Q1 meshes and
// the FP32 action of Q2; and the dispatch of all hexahedral kernels (Q1: hex8.cu, Q2 in FP64: hex27.cu,
// hex27lines.cu).
//
// A warp shares one Q2 cell (27 lanes busy) or four Q1 cells (8 lanes each). Lane q owns quadrature
// point q: it forms the trilinear geometry, the solution gradient from the cell's node values staged in
// shared memory, calls the registered pointwise kernel and stages its test-function weights
// wdetJ f1 J^{-T} (and wdetJ f0). Lane n then owns node n: it contracts the staged weights with the
// reference basis gradients of node n over all quadrature points and adds the result into the output
// (reductions; nodes are shared with neighbouring cells). The reference basis tables (gradients and
// values at the quadrature points, and the trilinear geometry gradients) are built once per block in
// shared memory. The FP32 action (inner iterations of the refined solver) keeps the geometry and the
// tangent in FP64 and stages the field, the weights and the sums in FP32.
#include "domain_kernels.cuh"
#include "internal.hpp"
#include "launch.hpp"

namespace plb {

template <int CELL, typename T = double>
struct HexGroup {
    using E = Elem<CELL>;
    static constexpr int NEN = E::nen;
    static constexpr int NQ = E::nq;
    static constexpr int G = CELL == HEX27 ? 32 : 8;   // lanes per cell
    static constexpr int CPW = 32 / G;                 // cells per warp
    static constexpr int LDB = (NEN * 3) | 1;          // odd row stride: lanes q spread over banks
    static constexpr int WARPS = 8;
    // FP64 tables (bytes from the start): geometry gradients [NQ][25], weights [NQ]
    static constexpr int T_W = NQ * 25;
    static constexpr int T_END64 = T_W + NQ;
    // T tables after them: field-basis gradients [NQ][LDB], basis values [NQ][NEN]
    static constexpr int T_PHI = NQ * LDB;
    static constexpr int T_ENDT = T_PHI + NQ * NEN;
    // per-group staging: corner coordinates [8][3] FP64; node field [NEN][3], test-function
    // weights [NQ][9] and body-force weights [NQ][3] in T; odd stride between groups
    static constexpr int OFF_F = NEN * 3;
    static constexpr int OFF_F0 = OFF_F + NQ * 9;
    static constexpr int PER_GROUP_T = (OFF_F0 + NQ * 3) | 1;
    static constexpr int PER_GROUP_X = 25;
    static constexpr int GROUPS = WARPS * CPW;
    static constexpr size_t bytes64() { return sizeof(double) * ((size_t)T_END64 + (size_t)GROUPS * PER_GROUP_X); }
    static constexpr size_t smem_bytes() {
        return bytes64() + sizeof(T) * ((size_t)T_ENDT + (size_t)GROUPS * PER_GROUP_T);
    }
};

template <int CELL, typename T>
PL_D void fill_tables(double* t64, T* tt) {
    using H = HexGroup<CELL, T>;
    for (int i = threadIdx.x; i < H::NQ * H::NEN; i += blockDim.x) {
        const int q = i / H::NEN, n = i % H::NEN;
        double d[3];
        if (CELL == HEX8) {
            hex_corner_dN<2>(n, q & 1, (q >> 1) & 1, q >> 2, d);
        } else {
            const double x = gauss3_x(q % 3), y = gauss3_x((q / 3) % 3), z = gauss3_x(q / 9);
            const int a = n % 3, b = (n / 3) % 3, c = n / 9;
            d[0] = quad_d(a, x) * quad_v(b, y) * quad_v(c, z);
            d[1] = quad_v(a, x) * quad_d(b, y) * quad_v(c, z);
            d[2] = quad_v(a, x) * quad_v(b, y) * quad_d(c, z);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) tt[q * H::LDB + n * 3 + k] = (T)d[k];
        tt[H::T_PHI + q * H::NEN + n] = (T)Elem<CELL>::phi(q, n);
    }
    for (int i = threadIdx.x; i < H::NQ * 8; i += blockDim.x) {
        const int q = i / 8, c = i % 8;
        double d[3];
        if (CELL == HEX8) hex_corner_dN<2>(c, q & 1, (q >> 1) & 1, q >> 2, d);
        else hex_corner_dN<3>(c, q % 3, (q / 3) % 3, q / 9, d);
#pragma unroll
        for (int k = 0; k < 3; ++k) t64[q * 25 + c * 3 + k] = d[k];
    }
    for (int q = threadIdx.x; q < H::NQ; q += blockDim.x)
        t64[H::T_W + q] = CELL == HEX8 ? 1.0 : gauss3_w(q % 3) * gauss3_w((q / 3) % 3) * gauss3_w(q / 9);
}

// Per-block tables and per-group staging of the group-of-lanes hexahedral kernels.
template <int CELL, typename T>
struct HexGroupSmem {
    const double* tN;  // geometry gradients [NQ][25]
    const double* tW;  // quadrature weights
    const T* tB;       // field-basis gradients [NQ][LDB]
    const T* tPhi;     // basis values [NQ][NEN]
    double* sX;        // this group's corner coordinates
    T* su;             // this group's node field
    T* sF;             // test-function weights
    T* sF0;            // body-force weights
    int grp, l;        // group of this lane within its warp, lane within the group
};

template <int CELL, typename T>
PL_D HexGroupSmem<CELL, T> hex_group_smem(double* hsm) {
    using H = HexGroup<CELL, T>;
    HexGroupSmem<CELL, T> g;
    double* t64 = hsm;
    T* tt = reinterpret_cast<T*>(hsm + H::T_END64 + H::GROUPS * H::PER_GROUP_X);
    g.tN = t64;
    g.tW = t64 + H::T_W;
    g.tB = tt;
    g.tPhi = tt + H::T_PHI;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    g.grp = lane / H::G;
    g.l = lane % H::G;
    const int gid = warp * H::CPW + g.grp;
    g.sX = hsm + H::T_END64 + gid * H::PER_GROUP_X;
    T* sg = tt + H::T_ENDT + gid * H::PER_GROUP_T;
    g.su = sg;
    g.sF = sg + H::OFF_F;
    g.sF0 = sg + H::OFF_F0;
    return g;
}

// The CPW cells base .. base + CPW - 1 of p, one per group of lanes of the calling warp (every
// lane of the warp calls it: it synchronises the warp).
template <int CELL, int RHEO, bool BF, int OP, typename T>
PL_D void hex_group_cells(const DomainParams& p, int64_t base, const HexGroupSmem<CELL, T>& g) {
    using H = HexGroup<CELL, T>;
    using L = AuxLayout<RHEO, BF>;
    const AuxOffsets<RHEO, BF> aoff;
    const double* tN = g.tN;
    const double* tW = g.tW;
    const T* tB = g.tB;
    const T* tPhi = g.tPhi;
    double* sX = g.sX;
    T* su = g.su;
    T* sF = g.sF;
    T* sF0 = g.sF0;
    const int grp = g.grp, l = g.l;
    constexpr bool f32 = sizeof(T) == 4;
    {
        const int64_t c = base + grp;
        const bool live = c < p.ncells;
        const int64_t mc = live ? (p.cell_ids ? p.cell_ids[c] : c) : 0;
        int node = 0;
        if (CELL == HEX8 && live) {
            // field and coordinates relative to the first corner (the basis gradients sum to zero), so that no
            // large coordinates or displacements cancel
            static_assert(CELL != HEX8 || (!f32 && OP == OP_RESIDUAL), "the Q1 instantiation is the FP64 residual's");
            node = p.cells[mc * 8 + l];
            const int64_t first = p.cells[mc * 8];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                su[l * 3 + k] = p.u[3 * (int64_t)node + k] - p.u[3 * first + k];
                sX[l * 3 + k] = p.coords[3 * (int64_t)node + k] - p.coords[3 * first + k];
            }
        } else if (live && l < H::NEN) {
            node = p.cells[mc * H::NEN + l];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                if (f32) su[l * 3 + k] = (T)p.v32[3 * (int64_t)node + k];
                else su[l * 3 + k] = (T)(OP == OP_RESIDUAL ? p.u : p.v)[3 * (int64_t)node + k];
            }
        }
        if (CELL != HEX8 && live && l < 8) {
            const int cn = p.cells[mc * H::NEN + Elem<CELL>::corner(l)];
#pragma unroll
            for (int k = 0; k < 3; ++k) sX[l * 3 + k] = p.coords[3 * (int64_t)cn + k];
        }
        __syncwarp();
        if (live && l < H::NQ) {
            const int q = l;
            T inv[3][3];
            T wdetJ;
            {
                double J[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll
                for (int k = 0; k < 8; ++k)
#pragma unroll
                    for (int i = 0; i < 3; ++i)
#pragma unroll
                        for (int j = 0; j < 3; ++j) J[i][j] += sX[k * 3 + i] * tN[q * 25 + k * 3 + j];
                double inv64[3][3];
                const double detJ = invert3(J, inv64);
                if (!(detJ > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
                wdetJ = (T)(tW[q] * detJ);
#pragma unroll
                for (int i = 0; i < 3; ++i)
#pragma unroll
                    for (int j = 0; j < 3; ++j) inv[i][j] = (T)inv64[i][j];
            }
            // reference gradient of the field, then s_x = Gref J^{-1}
            T Gr[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
#pragma unroll 9
            for (int n = 0; n < H::NEN; ++n) {
                const T b0 = tB[q * H::LDB + n * 3], b1 = tB[q * H::LDB + n * 3 + 1], b2 = tB[q * H::LDB + n * 3 + 2];
#pragma unroll
                for (int cc = 0; cc < 3; ++cc) {
                    const T un = su[n * 3 + cc];
                    Gr[cc][0] += un * b0;
                    Gr[cc][1] += un * b1;
                    Gr[cc][2] += un * b2;
                }
            }
            T s_x[9];
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
#pragma unroll
                for (int e = 0; e < 3; ++e)
                    s_x[cc * 3 + e] = Gr[cc][0] * inv[0][e] + Gr[cc][1] * inv[1][e] + Gr[cc][2] * inv[2][e];
            double a[L::size] = {};
            const bool cached = f32 && OP == OP_JACOBIAN_ACTION && p.lm32;
            if (!cached) L::load_cell(p, c, a);
            if (OP == OP_RESIDUAL) L::load_qp(p, c, q, H::NQ, a);  // the tangents read no state
            double x[3] = {0, 0, 0}, s[3] = {0, 0, 0};
            double f0[3] = {0, 0, 0};
            T f1[9];
            if (cached) {
                isotropic_contract<T>((T)p.lm32[2 * c], (T)p.lm32[2 * c + 1], s_x, f1);
            } else if (OP == OP_RESIDUAL) {
                double s_x64[9], f164[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
                for (int i = 0; i < 9; ++i) s_x64[i] = (double)s_x[i];
                if (BF) {
                    const int sOff[1] = {0}, sOff_x[1] = {0};
                    pw::g0v_bodyforce<double>(3, 1, L::numA, sOff, sOff_x, s, nullptr, s_x64, aoff.v, nullptr, a,
                                              nullptr, nullptr, p.t, x, p.num_constants, p.constants, f0);
                }
                call_f1<RHEO>(L::numA, aoff.v, a, s, s_x64, p, x, f164);
#pragma unroll
                for (int i = 0; i < 9; ++i) f1[i] = (T)f164[i];
            } else {
                double Jf3[81];
#pragma unroll
                for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
                call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
                isotropic_jf3_contract<RHEO>(Jf3, s_x, f1);
            }
            // test-function weights: grad(phi_n) . f1 = tB_n . (J^{-1} f1^T), so stage
            // W[cc][d] = wdetJ sum_e inv[d][e] f1[cc][e]
#pragma unroll
            for (int cc = 0; cc < 3; ++cc)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    sF[q * 9 + cc * 3 + d] =
                        wdetJ * (inv[d][0] * f1[cc * 3 + 0] + inv[d][1] * f1[cc * 3 + 1] + inv[d][2] * f1[cc * 3 + 2]);
            if (BF && OP == OP_RESIDUAL)
#pragma unroll
                for (int cc = 0; cc < 3; ++cc) sF0[q * 3 + cc] = wdetJ * (T)f0[cc];
        }
        __syncwarp();
        if (live && l < H::NEN) {
            const int n = l;
            T r0 = 0, r1 = 0, r2 = 0;
#pragma unroll 9
            for (int q = 0; q < H::NQ; ++q) {
                const T b0 = tB[q * H::LDB + n * 3], b1 = tB[q * H::LDB + n * 3 + 1], b2 = tB[q * H::LDB + n * 3 + 2];
                const T* w = sF + q * 9;
                r0 += b0 * w[0] + b1 * w[1] + b2 * w[2];
                r1 += b0 * w[3] + b1 * w[4] + b2 * w[5];
                r2 += b0 * w[6] + b1 * w[7] + b2 * w[8];
                if (BF && OP == OP_RESIDUAL) {
                    const T ph = tPhi[q * H::NEN + n];
                    r0 += ph * sF0[q * 3 + 0];
                    r1 += ph * sF0[q * 3 + 1];
                    r2 += ph * sF0[q * 3 + 2];
                }
            }
            if (f32) {
                float* o = p.out32 + 3 * (int64_t)node;
                red_add(o, (float)r0);
                red_add(o + 1, (float)r1);
                red_add(o + 2, (float)r2);
            } else {
                double* o = p.out + 3 * (int64_t)node;
                red_add(o, (double)r0);
                red_add(o + 1, (double)r1);
                red_add(o + 2, (double)r2);
            }
        }
        __syncwarp();
    }
}

// T = double: residual (OP_RESIDUAL) or Jacobian action into p.out from p.u / p.v;
// T = float: Jacobian action into p.out32 from p.v32.
template <int CELL, int RHEO, bool BF, int OP, typename T>
__global__ void __launch_bounds__(HexGroup<CELL, T>::WARPS * 32) k_hex_group(DomainParams p) {
    using H = HexGroup<CELL, T>;
    extern __shared__ __align__(16) double hsm[];
    fill_tables<CELL, T>(hsm, reinterpret_cast<T*>(hsm + H::T_END64 + H::GROUPS * H::PER_GROUP_X));
    __syncthreads();
    const HexGroupSmem<CELL, T> g = hex_group_smem<CELL, T>(hsm);
    const int warp = threadIdx.x >> 5;
    const int64_t cells_per_pass = (int64_t)gridDim.x * H::WARPS * H::CPW;
    // every lane of a warp runs the same number of passes (the __syncwarp calls need them all)
    for (int64_t base = ((int64_t)blockIdx.x * H::WARPS + warp) * H::CPW; base < p.ncells; base += cells_per_pass)
        hex_group_cells<CELL, RHEO, BF, OP, T>(p, base, g);
}

template <int CELL, int RHEO, bool BF, int OP, typename T = double>
static void launch_group_t(const DomainParams& p, cudaStream_t s) {
    using H = HexGroup<CELL, T>;
    auto kern = k_hex_group<CELL, RHEO, BF, OP, T>;
    const size_t smem = H::smem_bytes();
    ensure_kernel_smem((const void*)kern, smem);
    const int nsm = sm_count();
    static int per_sm = 0;  // occupancy of this instantiation (the same on every B200)
    if (!per_sm) {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, H::WARPS * 32, smem);
        per_sm = std::max(per_sm, 1);
    }
    const int64_t groups = (p.ncells + H::WARPS * H::CPW - 1) / (H::WARPS * H::CPW);
    const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(groups, (int64_t)nsm * std::max(per_sm, 1)));
    kern<<<grid, H::WARPS * 32, smem, s>>>(p);
    count_launch();
}

// Q2 hexahedra: a line of points per lane (hex27lines.cu) while the mesh is a wave or so of its blocks,
// a plane of nodes per lane (hex27.cu) beyond. Cells per multiprocessor at which they cross, with the
// two measured below and above (us, ADD): isotropic 10.4 and 12.4 at 2,912 cells, 14.5 and 12.5 at 5,508;
// generalized-Maxwell residual 20.7 and 22.7 at 5,202, 26.9 and 22.7 at 6,000; its action 14.5 and 17.0
// at 5,184, 20.6 and 19.6 at 7,200. One cell to a few hundred: 6.3 and 10.4, residual 8.4 and 18.6.
static bool hex27_by_lines(const DomainParams& p, int rheo, int op) {
    const int per_sm = rheo != RHEO_GENMAXWELL ? 26 : (op == OP_RESIDUAL ? 36 : 44);
    return p.ncells <= per_sm * (int64_t)sm_count();
}

// Generalized-Maxwell residual of Q1: a lane per point (this file) while that is at most one block of 32
// cells per multiprocessor, a thread per cell (hex8.cu) beyond: the points' exponentials and state, one
// after the other, are a longer chain. ADD: 8.4 and 10.4 us at 336 to 2,912 cells, 8.3 and 10.6 at 3,978,
// 12.5 and 10.4 at 5,760.
static bool hex8_by_points(const DomainParams& p, int rheo, int op) {
    return rheo == RHEO_GENMAXWELL && op == OP_RESIDUAL && p.ncells <= 32 * (int64_t)sm_count();
}

bool launch_domain_apply_hexgroup(const DomainParams& p, int cell, int rheo, bool bf, int op, cudaStream_t s) {
    if (p.ncells == 0) return true;
    if (cell == HEX8 && hex8_by_points(p, rheo, op)) {
        if (bf) launch_group_t<HEX8, RHEO_GENMAXWELL, true, OP_RESIDUAL>(p, s);
        else launch_group_t<HEX8, RHEO_GENMAXWELL, false, OP_RESIDUAL>(p, s);
    } else if (cell == HEX8) launch_hex8(p, rheo, bf, op, s);
    else if (cell == HEX27 && hex27_by_lines(p, rheo, op)) launch_hex27_lines(p, rheo, bf, op, s);
    else if (cell == HEX27) launch_hex27(p, rheo, bf, op, s);
    else return false;
    return true;
}

// (lambda, mu) of the isotropic tangent per integrator cell at p.t, p.dt, from the registered
// Jacobian kernel: the FP32 Jacobian action of hexahedra reads them instead of evaluating the
// tangent (for generalized Maxwell, three exponentials in FP64) at each quadrature point.
template <int RHEO>
__global__ void k_tangent_lm32(DomainParams p, float* __restrict__ out) {
    using L = AuxLayout<RHEO, false>;
    const AuxOffsets<RHEO, false> aoff;
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < p.ncells; c += (int64_t)gridDim.x * blockDim.x) {
        double a[L::size] = {};
        L::load_cell(p, c, a);
        double x[3] = {0, 0, 0}, Jf3[81];
#pragma unroll
        for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
        call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
        out[2 * c] = (float)(-Jf3[((0 * 3 + 1) * 3 + 0) * 3 + 1]);
        out[2 * c + 1] = (float)(-Jf3[((0 * 3 + 1) * 3 + 1) * 3 + 0]);
    }
}

bool launch_tangent_lm32(const DomainParams& p, int rheo, float* out, cudaStream_t s) {
    if (rheo != RHEO_ILE && rheo != RHEO_GENMAXWELL) return false;
    if (p.ncells == 0) return true;
    const int grid = (int)std::min<int64_t>((p.ncells + 255) / 256, 148 * 16);
    if (rheo == RHEO_GENMAXWELL) k_tangent_lm32<RHEO_GENMAXWELL><<<grid, 256, 0, s>>>(p, out);
    else k_tangent_lm32<RHEO_ILE><<<grid, 256, 0, s>>>(p, out);
    count_launch();
    return true;
}

bool launch_domain_jv32_hexgroup(const DomainParams& p, int cell, int rheo, cudaStream_t s) {
    if (p.ncells == 0) return true;
    const bool gm = rheo == RHEO_GENMAXWELL;
    if (cell == HEX8) {
        launch_hex8_jv32(p, rheo, s);
    } else if (cell == HEX27) {
        if (gm) launch_group_t<HEX27, RHEO_GENMAXWELL, false, OP_JACOBIAN_ACTION, float>(p, s);
        else launch_group_t<HEX27, RHEO_ILE, false, OP_JACOBIAN_ACTION, float>(p, s);
    } else {
        return false;
    }
    return true;
}

}  // namespace plb
