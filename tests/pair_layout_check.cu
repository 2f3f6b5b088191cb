// Host check of the cell-pair planner (match_cells, cut_pair_range and plan_pair_block in
// pylith_b200/csrc/tetpair.cu), built by tests/test_pair_layout.py: a Kuhn-split grid whose cells are
// shuffled within windows, and every seventh turned inside out, is cut into blocks and planned. The
// program prints one JSON line. ok: every cell is in one item, as an even permutation of its corners;
// every (item, corner) is in one node's list, at its staging offset; no block exceeds its limits; a
// block's cells follow the one before.
// usage: pair_layout_check GRID WINDOW (0: cells in order)
#include <cstdio>
#include <cstdlib>

#include "../pylith_b200/csrc/tetpair.cu"

namespace plb {
void count_launch(int) {}
void ensure_kernel_smem(const void*, size_t) {}
int sm_count() { return 148; }
int cuda_fail(cudaError_t, const char*) { return PL_ERR_CUDA; }
int fail(int code, const std::string&) { return code; }
cudaError_t dev_alloc(void**, size_t) { return cudaErrorNotSupported; }
void dev_free(void*, cudaStream_t) {}
bool zero_output(double*, int64_t, bool, bool, cudaStream_t) { return false; }
int ensure_blocked_layout(pl_mesh_s*) { return PL_ERR_UNSUPPORTED; }
int ensure_reduced_ids(pl_mesh_s*) { return PL_ERR_UNSUPPORTED; }
}  // namespace plb

using namespace plb;

// Whether the corners p are an even permutation of the corners q.
static bool even(const int32_t* p, const int32_t* q) {
    int at[4], swaps = 0;
    for (int i = 0; i < 4; ++i) {
        at[i] = -1;
        for (int j = 0; j < 4; ++j)
            if (p[i] == q[j]) at[i] = j;
        if (at[i] < 0) return false;
    }
    for (int i = 0; i < 4; ++i)
        for (int j = i + 1; j < 4; ++j) {
            if (at[i] == at[j]) return false;
            swaps += at[i] > at[j];
        }
    return swaps % 2 == 0;
}

int main(int argc, char** argv) {
    const int n = argc > 1 ? atoi(argv[1]) : 6, window = argc > 2 ? atoi(argv[2]) : 0;
    auto id = [&](int i, int j, int k) { return (i * (n + 1) + j) * (n + 1) + k; };
    const int perm[6][3] = {{0, 1, 2}, {0, 2, 1}, {1, 0, 2}, {1, 2, 0}, {2, 0, 1}, {2, 1, 0}};
    std::vector<int32_t> cells;
    for (int i = 0; i < n; ++i)
        for (int j = 0; j < n; ++j)
            for (int k = 0; k < n; ++k)
                for (int q = 0; q < 6; ++q) {
                    int x[3] = {i, j, k};
                    cells.push_back(id(x[0], x[1], x[2]));
                    for (int s = 0; s < 3; ++s) {
                        x[perm[q][s]]++;
                        cells.push_back(id(x[0], x[1], x[2]));
                    }
                    int inv = 0;  // one orientation for all
                    for (int a = 0; a < 3; ++a)
                        for (int b = a + 1; b < 3; ++b) inv += perm[q][a] > perm[q][b];
                    if (inv % 2) std::swap(cells[cells.size() - 1], cells[cells.size() - 2]);
                }
    const int64_t nc = (int64_t)cells.size() / 4;
    for (int64_t c = 0; c < nc; c += 7) std::swap(cells[4 * c], cells[4 * c + 1]);
    uint64_t rs = 1;
    for (int64_t w = 0; window > 0 && w < nc; w += window) {
        const int64_t m = std::min<int64_t>(window, nc - w);
        for (int64_t i = m - 1; i > 0; --i) {
            const int64_t j = (int64_t)(splitmix64(rs) % (uint64_t)(i + 1));
            for (int k = 0; k < 4; ++k) std::swap(cells[4 * (w + i) + k], cells[4 * (w + j) + k]);
        }
    }
    std::vector<PairCut> cuts;
    const bool planned = cut_pair_range(cells.data(), 0, nc, cuts);
    if (!planned) cuts.clear();
    bool ok = true;
    int64_t c0 = 0, pairs = 0;
    int most = 0;
    for (const PairCut& cut : cuts) {
        PairPlan P;
        plan_pair_block(c0, cut, P);
        const int nloc = (int)P.loc.size(), ni = (int)P.items.size() / 4;
        most = std::max(most, nloc);
        ok = ok && nloc <= kPairMaxNodes && ni >= 1 && ni <= kPairThreads && (int)P.off.size() == nloc + 1 && P.inc.size() <= 5 * kPairThreads;
        std::vector<int> used(kPairCells, 0);
        std::vector<int32_t> node(5 * (size_t)ni, -1);  // of each (item, corner)
        int ncell = 0;
        for (int i = 0; ok && i < ni; ++i) {
            const uint32_t* w = &P.items[4 * i];
            const uint32_t l[5] = {w[0] & 0xffff, w[0] >> 16, w[1] & 0xffff, w[1] >> 16, w[2] & 0xffff};
            const bool single = w[2] >> 16 == 0;
            for (int k = 0; k < 5; ++k) {
                ok = ok && (int)l[k] < nloc;
                if (ok && (k < 4 || !single)) node[5 * i + k] = P.loc[l[k]];
            }
            if (!ok) break;
            const int64_t a = w[3], b = single ? a : a + (int)(w[2] >> 16) - kCellBias;
            const int32_t A[4] = {P.loc[l[0]], P.loc[l[1]], P.loc[l[2]], P.loc[l[3]]}, B[4] = {P.loc[l[0]], P.loc[l[2]], P.loc[l[1]], P.loc[l[4]]};
            for (int64_t c : {a, b}) ok = ok && c >= c0 && c < c0 + kPairCells && c < nc;
            if (!ok) break;
            ok = even(A, &cells[4 * a]) && used[a - c0]++ == 0;
            if (!single) ok = ok && even(B, &cells[4 * b]) && used[b - c0]++ == 0;
            ncell += single ? 1 : 2;
            pairs += !single;
        }
        for (int i = 0; ok && i < ncell; ++i) ok = used[i] == 1;  // the block's cells are consecutive
        std::vector<int> hit(5 * (size_t)ni, 0);
        for (int v = 0; ok && v < nloc; ++v)
            for (int j = P.off[v]; j < P.off[v + 1]; ++j) {
                const int q = P.inc[j], k = q / (3 * kPairThreads), i = q % (3 * kPairThreads);
                ok = ok && k < 5 && i < ni && node[5 * i + k] == P.loc[v] && hit[5 * i + k]++ == 0;
            }
        for (int i = 0; ok && i < 5 * ni; ++i) ok = hit[i] == (node[i] >= 0);
        c0 += ncell;
    }
    ok = ok && c0 == (planned ? nc : 0);
    printf("{\"ok\": %s, \"planned\": %s, \"cells\": %lld, \"blocks\": %zu, \"pairs\": %lld, \"most_nodes\": %d}\n", ok ? "true" : "false",
           planned ? "true" : "false", (long long)nc, cuts.size(), (long long)pairs, most);
    return ok ? 0 : 1;
}
