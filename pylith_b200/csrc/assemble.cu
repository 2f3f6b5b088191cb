// Assembled Jacobian: element matrices from the registered Jf3, added into the 3x3-block CSR values
// at precomputed block positions (DMPlexComputeJacobianByKey + MatSetClosure).
//
// Bound: the reductions into L2. An L2 slice takes a 32-byte sector of a reduction at a time,
// whether one of its four doubles or all of them change (about 200 G sectors/s on this GPU), so
// what counts is sectors, not values. A warp therefore sums a cell's blocks over the quadrature
// points first, stages them in shared memory and adds them with consecutive lanes on consecutive
// doubles: 2.3 to 4 sectors per 3x3 block. The tangents on this path read no per-point state and
// are isotropic (domain_kernels.cuh), so with H = sum_q w det grad(phi_a) grad(phi_b)^T
//     K_ab = -(lambda H + mu (tr(H) I + H^T)).
#include <algorithm>

#include "domain_kernels.cuh"
#include "internal.hpp"
#include "launch.hpp"

namespace plb {

// (lambda, mu) of integrator cell c's tangent at p.t, p.dt.
template <int RHEO>
PL_D double2 cell_tangent(const DomainParams& p, int64_t c) {
    using L = AuxLayout<RHEO, false>;
    const AuxOffsets<RHEO, false> aoff;
    double a[L::size] = {};
    L::load_cell(p, c, a);
    double x[3] = {0, 0, 0}, Jf3[81];
#pragma unroll
    for (int i = 0; i < 81; ++i) Jf3[i] = 0.0;
    call_jf3<RHEO>(L::numA, aoff.v, a, p, x, Jf3);
    return make_double2(-Jf3[((0 * 3 + 1) * 3 + 0) * 3 + 1], -Jf3[((0 * 3 + 1) * 3 + 1) * 3 + 0]);
}

template <int CELL>
struct AssembleHex {
    using E = Elem<CELL>;
    static constexpr int NEN = E::nen, NQ = E::nq;
    static constexpr int CPW = CELL == HEX8 ? 4 : 1;  // cells per warp and pass
    static constexpr int WARPS = 2;
    static constexpr int TA = CELL == HEX8 ? 2 : 3, TB = TA;  // blocks of a lane: TA rows x TB columns
    static constexpr int TILE = TA * TB, NTB = NEN / TB;
    static constexpr int TILES = NEN / TA * NTB;  // of a cell
    static constexpr int LDG = (NEN * 3) | 1;   // odd stride between the points' gradients
    static constexpr int LDT = (TILE * 9) | 1;  // odd stride between the lanes' staged blocks
    // per warp: gradients [CPW][NQ][LDG], weights [CPW][NQ], (lambda, mu) [CPW], staged blocks
    // [32][LDT] (doubles), then the staged blocks' positions [32][TILE] as int32
    static constexpr int O_W = CPW * NQ * LDG, O_T = O_W + CPW * NQ, O_S = O_T + 2 * CPW, O_P = O_S + 32 * LDT;
    static constexpr int PER_WARP = O_P + 32 * TILE / 2;
    static constexpr size_t smem_bytes() { return sizeof(double) * (size_t)WARPS * PER_WARP; }
};

// Hexahedra: lanes (cell, point) form the gradients of a warp's CPW cells in shared memory; then
// each lane sums a tile of a cell's blocks over the points (Q1: 2 x 2 of its 8 x 8 blocks; Q2: 3 x 3
// of 27 x 27), so a point's 12 (18) loaded gradient entries make 36 (81) multiply-adds. 32x32x24 Q1 cells: 794 us with a thread per cell and 9
// reductions per block and point, 51 us with two blocks of one row per lane (bound by the
// shared-memory pipe), 45 us with 2 x 4 blocks (7 warps per multiprocessor), 43 us with 2 x 2 (11
// warps; L1 pipe 76 %, most of it the reductions).
template <int CELL, int RHEO>
__global__ void __launch_bounds__(AssembleHex<CELL>::WARPS * 32) k_assemble_hex(DomainParams p, const int32_t* __restrict__ pos,
                                                                                double* __restrict__ vals) {
    using A = AssembleHex<CELL>;
    using E = Elem<CELL>;
    extern __shared__ __align__(16) double asm_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* sG = asm_smem + warp * A::PER_WARP;
    double* sW = sG + A::O_W;
    double* sT = sG + A::O_T;
    double* sS = sG + A::O_S;
    int32_t* sP = reinterpret_cast<int32_t*>(sG + A::O_P);
    const int64_t stride = (int64_t)gridDim.x * A::WARPS * A::CPW;
    for (int64_t c0 = ((int64_t)blockIdx.x * A::WARPS + warp) * A::CPW; c0 < p.ncells; c0 += stride) {
        const int ncell = (int)min((int64_t)A::CPW, p.ncells - c0);
        constexpr int LPC = 32 / A::CPW;  // lanes per cell of the geometry
        const int gc = lane / LPC, gl = lane % LPC;
        if (gc < ncell && gl < A::NQ) {
            const int64_t c = c0 + gc;
            const int32_t* cn = p.cells + (p.cell_ids ? p.cell_ids[c] : c) * A::NEN;
            double X[8][3];
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
                for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * (int64_t)cn[E::corner(k)] + i];
            Geom g;
            E::geom(X, gl, &g);
            if (!(g.detJ > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
            sW[gc * A::NQ + gl] = g.wdetJ;
            double* out = sG + (gc * A::NQ + gl) * A::LDG;
#pragma unroll 9
            for (int n = 0; n < A::NEN; ++n) {
                double gr[3];
                E::grad(g, gl, n, gr);
#pragma unroll
                for (int k = 0; k < 3; ++k) out[3 * n + k] = gr[k];
            }
            if (gl == 0) {
                const double2 lm = cell_tangent<RHEO>(p, c);
                sT[2 * gc] = lm.x;
                sT[2 * gc + 1] = lm.y;
            }
        }
        __syncwarp();
#pragma unroll 1
        for (int t0 = 0; t0 < ncell * A::TILES; t0 += 32) {
            if (t0 + lane < ncell * A::TILES) {
                const int k = (t0 + lane) / A::TILES, tile = (t0 + lane) % A::TILES;
                const int a0 = tile / A::NTB * A::TA, b0 = tile % A::NTB * A::TB;
                double H[A::TILE][9] = {};
                const double* ga = sG + k * A::NQ * A::LDG + 3 * a0;
                const double* gb = sG + k * A::NQ * A::LDG + 3 * b0;
#pragma unroll 1
                for (int q = 0; q < A::NQ; ++q, ga += A::LDG, gb += A::LDG) {
                    const double w = sW[k * A::NQ + q];
                    double wa[A::TA][3];
#pragma unroll
                    for (int i = 0; i < A::TA; ++i)
#pragma unroll
                        for (int f = 0; f < 3; ++f) wa[i][f] = w * ga[3 * i + f];
#pragma unroll
                    for (int j = 0; j < A::TB; ++j)
#pragma unroll
                        for (int gg = 0; gg < 3; ++gg) {
                            const double b = gb[3 * j + gg];
#pragma unroll
                            for (int i = 0; i < A::TA; ++i)
#pragma unroll
                                for (int f = 0; f < 3; ++f) H[i * A::TB + j][3 * f + gg] += wa[i][f] * b;
                        }
                }
                const double lam = sT[2 * k], mu = sT[2 * k + 1];
                const int64_t c = c0 + k;
                const int32_t* cpos = pos + (p.cell_ids ? p.cell_ids[c] : c) * A::NEN * A::NEN + a0 * A::NEN + b0;
#pragma unroll
                for (int m = 0; m < A::TILE; ++m) {
                    sP[lane * A::TILE + m] = cpos[m / A::TB * A::NEN + m % A::TB];
                    const double tr = mu * (H[m][0] + H[m][4] + H[m][8]);
#pragma unroll
                    for (int f = 0; f < 3; ++f)
#pragma unroll
                        for (int gg = 0; gg < 3; ++gg)
                            sS[lane * A::LDT + 9 * m + 3 * f + gg] =
                                -(lam * H[m][3 * f + gg] + mu * H[m][3 * gg + f] + (f == gg ? tr : 0.0));
                }
            }
            __syncwarp();
            const int n = min(32, ncell * A::TILES - t0);  // staging lanes
#pragma unroll 2
            for (int t = lane; t < n * A::TILE * 9; t += 32) {
                const int l = t / (A::TILE * 9), blk = t / 9;
                red_add(vals + 9 * (int64_t)sP[blk] + (t - 9 * blk), sS[t + l * (A::LDT - A::TILE * 9)]);
            }
            __syncwarp();
        }
    }
}

// Tetrahedra: one gradient per corner and cell. Lanes form the gradients of a warp's 8 cells, then
// take the cells two at a time, a block per lane, staged and added as above. 54,737 cells: 51 us
// with a thread per cell and unstaged reductions, 29 us with a value per lane formed on the fly
// (L1 pipe 84 %), 24 us this way (63 %).
struct AssembleTet {
    static constexpr int WARPS = 4;
    static constexpr int CELLS = 8;  // per warp and pass
    static constexpr int LDC = 15;  // per cell: gradients [4][3], lambda |K|, mu |K| (odd stride)
    static constexpr size_t smem_bytes() { return (sizeof(double) * (LDC * CELLS + 9 * 32) + sizeof(int32_t) * 32) * WARPS; }
};

template <int RHEO>
__global__ void __launch_bounds__(AssembleTet::WARPS * 32) k_assemble_tet(DomainParams p, const int32_t* __restrict__ pos,
                                                                          double* __restrict__ vals) {
    using A = AssembleTet;
    extern __shared__ __align__(16) double asm_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* sC = asm_smem + warp * A::CELLS * A::LDC;
    double* sS = asm_smem + A::WARPS * A::CELLS * A::LDC + warp * 9 * 32;
    int32_t* sP = reinterpret_cast<int32_t*>(asm_smem + A::WARPS * (A::CELLS * A::LDC + 9 * 32)) + warp * 32;
    const int64_t stride = (int64_t)gridDim.x * A::WARPS * A::CELLS;
    for (int64_t c0 = ((int64_t)blockIdx.x * A::WARPS + warp) * A::CELLS; c0 < p.ncells; c0 += stride) {
        const int n = (int)min((int64_t)A::CELLS, p.ncells - c0);
        if (lane < n) {
            const int64_t c = c0 + lane;
            const int4 cn = reinterpret_cast<const int4*>(p.cells)[p.cell_ids ? p.cell_ids[c] : c];
            const int nd[4] = {cn.x, cn.y, cn.z, cn.w};
            double X[4][3];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int i = 0; i < 3; ++i) X[k][i] = p.coords[3 * (int64_t)nd[k] + i];
            Geom g;
            tet_geometry(X, &g);
            if (!(g.detJ > 0.0)) flag_error(p.err, CHECK_NONPOSITIVE_DETJ);
            double* out = sC + lane * A::LDC;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                double gr[3];
                tet_grad(g, k, gr);
#pragma unroll
                for (int i = 0; i < 3; ++i) out[3 * k + i] = gr[i];
            }
            const double2 t = cell_tangent<RHEO>(p, c);
            out[12] = -g.wdetJ * t.x;
            out[13] = -g.wdetJ * t.y;
        }
        __syncwarp();
#pragma unroll 1
        for (int b0 = 0; b0 < 16 * n; b0 += 32) {
            const int e = b0 + lane;  // block 16 cell + 4 a + b
            if (e < 16 * n) {
                const int64_t c = c0 + (e >> 4);
                sP[lane] = pos[16 * (p.cell_ids ? (int64_t)p.cell_ids[c] : c) + (e & 15)];
                const double* C = sC + (e >> 4) * A::LDC;
                double ga[3], gb[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    ga[i] = C[3 * ((e >> 2) & 3) + i];
                    gb[i] = C[3 * (e & 3) + i];
                }
                const double lam = C[12], mu = C[13];
                const double tr = mu * (ga[0] * gb[0] + ga[1] * gb[1] + ga[2] * gb[2]);
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int g = 0; g < 3; ++g)
                        sS[9 * lane + 3 * f + g] = lam * (ga[f] * gb[g]) + mu * (ga[g] * gb[f]) + (f == g ? tr : 0.0);
            }
            __syncwarp();
            const int nv = 9 * min(32, 16 * n - b0);
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const int t = lane + 32 * i, blk = t / 9;
                if (t < nv) red_add(vals + 9 * (int64_t)sP[blk] + (t - 9 * blk), sS[t]);
            }
            __syncwarp();
        }
    }
}

template <int CELL, int RHEO>
static void launch_hex_t(const DomainParams& p, const int32_t* pos, double* vals, cudaStream_t s) {
    using A = AssembleHex<CELL>;
    auto kern = k_assemble_hex<CELL, RHEO>;
    ensure_kernel_smem((const void*)kern, A::smem_bytes());
    const int64_t per = A::WARPS * A::CPW;
    kern<<<(unsigned)std::min<int64_t>((p.ncells + per - 1) / per, 1 << 20), A::WARPS * 32, A::smem_bytes(), s>>>(p, pos, vals);
    count_launch();
}

template <int RHEO>
static void launch_tet_t(const DomainParams& p, const int32_t* pos, double* vals, cudaStream_t s) {
    using A = AssembleTet;
    auto kern = k_assemble_tet<RHEO>;
    const int64_t per = A::WARPS * A::CELLS;
    kern<<<(unsigned)std::min<int64_t>((p.ncells + per - 1) / per, 1 << 20), A::WARPS * 32, A::smem_bytes(), s>>>(p, pos, vals);
    count_launch();
}

void launch_domain_jacobian(const DomainParams& p, int cell, int rheo, const int32_t* pos, double* vals, cudaStream_t s) {
    if (p.ncells == 0) return;
    const bool gm = rheo == RHEO_GENMAXWELL;
    if (cell == TET4) gm ? launch_tet_t<RHEO_GENMAXWELL>(p, pos, vals, s) : launch_tet_t<RHEO_ILE>(p, pos, vals, s);
    else if (cell == HEX8) gm ? launch_hex_t<HEX8, RHEO_GENMAXWELL>(p, pos, vals, s) : launch_hex_t<HEX8, RHEO_ILE>(p, pos, vals, s);
    else gm ? launch_hex_t<HEX27, RHEO_GENMAXWELL>(p, pos, vals, s) : launch_hex_t<HEX27, RHEO_ILE>(p, pos, vals, s);
}

}  // namespace plb
