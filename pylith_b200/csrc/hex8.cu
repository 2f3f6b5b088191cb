// Q1 hexahedra, one thread per cell (hex8.cuh): residual, FP64 and FP32 Jacobian action.
//
// Bound: FP64 arithmetic, about 1,350 operations per cell (65 % of the FP64 pipe busy at 8 warps per
// multiprocessor, DRAM 13 %); FP32, instruction issue and latency. One thread per cell takes the
// whole sweep into registers (254 in FP64), where 8 lanes per cell staged every contraction through
// shared memory: on the 96x96x72 box (663,552 cells), numbered along x, the FP64 residual went from 275
// to 78 us, the FP64 action from 275 to 74 us and the FP32 action from 192 to 45 us; numbered along a
// Morton curve 264, 264, 185 -> 94, 90, 60; shuffled 293, 293, 212 -> 131, 127, 115. The reductions alone, 16 M
// on that box, take 58 us in FP64 when each cell adds its own 24 sums and 31 us when consecutive
// cells hand on their shared face (hex8_scatter). FP32 with 6 blocks of 64 threads per
// multiprocessor (145 registers) was slower than with 8 (128): 62 against 55 us when measured.
#include <algorithm>

#include "hex8.cuh"
#include "internal.hpp"
#include "launch.hpp"

namespace plb {

template <int RHEO, bool BF, int OP, typename T>
__global__ void __launch_bounds__(64, sizeof(T) == 4 ? 8 : 4) k_hex8(DomainParams p) {
    extern __shared__ __align__(16) double h8_smem[];
    hex8_cell<RHEO, BF, OP, T>(p, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, h8_smem);
}

// State update of generalized-Maxwell cells (domain.cu, k_domain_update_state) with the gradient by
// edge differences and the state copied ahead; written back in place. Bound: HBM (4.5 TB/s of state
// read and written). 48x48x36 cells: 60 us with a thread per cell in a loop over the points, 56 us
// this way; 12 or 16 warps per multiprocessor (456 bytes of spills and more) measured 66 and 73 us.
__global__ void __launch_bounds__(64, 4) k_hex8_update_state(DomainParams p) {
    using L = AuxLayout<RHEO_GENMAXWELL, false>;
    extern __shared__ __align__(16) double h8_smem[];
    const int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (c >= p.ncells) return;
    Hex8State state(h8_smem, p, c);
    int nodes[8];
    hex8_nodes(p, c, nodes);
    Hex8Nodes<double> h;
    hex8_load(p.coords, p.u, nodes, h);
    double a[L::size] = {}, g[8][3];
    L::load_cell(p, c, a);
    const pw::MaxwellFactors<double> mf = pw::maxwell_factors(a + L::base + 2, p.constants[0]);
    hex8_sweep<false, false, double>(
        h, nullptr, g, [&](int q, const double(&G)[3][3], const double(&C)[3][3], double det, double(&)[3][3], double(&)[3]) {
            const double rdet = 1.0 / det;
            double s_x[9], visc[18];
#pragma unroll
            for (int f = 0; f < 3; ++f)
#pragma unroll
                for (int e = 0; e < 3; ++e)
                    s_x[f * 3 + e] = (G[f][0] * C[0][e] + G[f][1] * C[1][e] + G[f][2] * C[2][e]) * rdet;
            const double* st = state.take(q);
            const pw::Sym<double> e = pw::strain(s_x);
            pw::genmaxwell_viscous_strain(st, pw::sym_from_vector(st + 18), mf, e, visc);
            double* pv = p.visc + q * p.ncells + c;
            double* pt = p.total + q * p.ncells + c;
#pragma unroll
            for (int k = 0; k < 18; ++k) pv[(int64_t)k * 8 * p.ncells] = visc[k];
            const double tot[6] = {e.xx, e.yy, e.zz, e.xy, e.yz, e.xz};
#pragma unroll
            for (int k = 0; k < 6; ++k) pt[(int64_t)k * 8 * p.ncells] = tot[k];
        });
}

// Threads per block: warps spread over the multiprocessors while there are fewer than two per
// multiprocessor.
static int hex8_threads(int64_t ncells) { return ncells <= (int64_t)sm_count() * 64 ? 32 : 64; }

template <int RHEO, bool BF, int OP, typename T>
static void launch_t(const DomainParams& p, cudaStream_t s) {
    const int th = hex8_threads(p.ncells);
    auto kern = k_hex8<RHEO, BF, OP, T>;
    const size_t smem = RHEO == RHEO_GENMAXWELL && OP == OP_RESIDUAL ? hex8_state_bytes(th) : 0;
    if (smem) ensure_kernel_smem((const void*)kern, smem);
    launch_domain(kern, (p.ncells + th - 1) / th, th, smem, s, p);
}

void launch_hex8_update_state(const DomainParams& p, cudaStream_t s) {
    const int th = hex8_threads(p.ncells);
    ensure_kernel_smem((const void*)k_hex8_update_state, hex8_state_bytes(th));
    k_hex8_update_state<<<(unsigned)((p.ncells + th - 1) / th), th, hex8_state_bytes(th), s>>>(p);
    count_launch();
}

template <int RHEO>
static void launch_r(const DomainParams& p, bool bf, int op, cudaStream_t s) {
    if (op != OP_RESIDUAL) launch_t<RHEO, false, OP_JACOBIAN_ACTION, double>(p, s);
    else if (bf) launch_t<RHEO, true, OP_RESIDUAL, double>(p, s);
    else launch_t<RHEO, false, OP_RESIDUAL, double>(p, s);
}

void launch_hex8(const DomainParams& p, int rheo, bool bf, int op, cudaStream_t s) {
    if (rheo == RHEO_ILE) launch_r<RHEO_ILE>(p, bf, op, s);
    else launch_r<RHEO_GENMAXWELL>(p, bf, op, s);
}

void launch_hex8_jv32(const DomainParams& p, int rheo, cudaStream_t s) {
    if (rheo == RHEO_ILE) launch_t<RHEO_ILE, false, OP_JACOBIAN_ACTION, float>(p, s);
    else launch_t<RHEO_GENMAXWELL, false, OP_JACOBIAN_ACTION, float>(p, s);
}

// FP32 Jacobian action over the cells of many meshes in one launch (the ragged batch of solvers,
// ragged.cu): member m's cells form warp chunks chunk0[m] .. chunk0[m + 1] - 1 of one index space
// (kHex8ChunkCells cells per chunk), so a warp never mixes members; ops[m] holds member m's operator
// arguments (its own cells, coordinates, cached per-cell tangent, input and output). Members must
// have the cached isotropic tangent (lm32).
static_assert(kHex8ChunkCells == 32, "one cell per lane");
__global__ void __launch_bounds__(64, 8)
    k_hex8_jv32_ragged(const DomainParams* __restrict__ ops, const int64_t* __restrict__ chunk0,
                       const int* __restrict__ active, const int* __restrict__ nmembers) {
    const int M = *nmembers;
    const int64_t total = chunk0[M];
    const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; w < total; w += warps) {
        int lo = 0, hi = M;  // the member of chunk w: largest m with chunk0[m] <= w
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (chunk0[mid] <= w) lo = mid;
            else hi = mid;
        }
        if (!active[lo]) continue;  // the whole warp shares w
        hex8_cell<RHEO_ILE, false, OP_JACOBIAN_ACTION, float>(ops[lo], (w - chunk0[lo]) * kHex8ChunkCells + (threadIdx.x & 31));
    }
}

void launch_hex8_jv32_ragged(const DomainParams* ops, const int64_t* chunk0, const int* active, const int* nmembers,
                             cudaStream_t s) {
    k_hex8_jv32_ragged<<<sm_count() * 8, 64, 0, s>>>(ops, chunk0, active, nmembers);
}

}  // namespace plb
