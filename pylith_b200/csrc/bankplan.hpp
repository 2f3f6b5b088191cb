// Host: numbering a cell block's local nodes and ordering its incidences for shared-memory banks.
//
// The cell-block kernels keep node values component-major in shared memory, so the bank pair of node
// i in an FP64 array is i mod 16 (and the 16-byte bank group of an FP32 row of 28 floats is 7 i mod
// 8): the reads of one corner by a warp conflict when distinct nodes share an index residue. A warp's
// 64-bit reads go through in two halves of 16 lanes, whose conflicts add up (measured: two-way conflicts
// within each half cost 3.9 cycles, although no bank pair is read more than twice by the warp).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace plb {

constexpr int kBankPairs = 16, kWarp = 32;

inline uint64_t splitmix64(uint64_t& x) {
    uint64_t z = (x += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

// perm[l]: the new index of node l. node_groups[l]: the (lanes that read together, corner)
// reads that touch node l, ng in all. Starting from perm = identity, a local search over swaps of two nodes' indices (deterministic,
// `iters` steps seeded by `seed`) lowers the sum over groups of the largest number of distinct nodes on
// one residue. Within each residue class the nodes are then placed by decreasing deg (incidence count),
// so each warp of the per-node sums gets nodes of similar counts and runs fewer steps.
inline void spread_nodes(const std::vector<std::vector<int>>& node_groups, int ng, const std::vector<int>& deg, uint64_t seed,
                         int iters, std::vector<int32_t>& perm) {
    constexpr int R = kBankPairs;
    const int nloc = (int)node_groups.size();
    perm.resize(nloc);
    for (int l = 0; l < nloc; ++l) perm[l] = l;
    std::vector<uint8_t> cnt((size_t)ng * R, 0);  // (a group holds at most 32 distinct nodes)
    for (int l = 0; l < nloc; ++l)
        for (int g : node_groups[l]) cnt[(size_t)g * R + (perm[l] & (R - 1))]++;
    auto gmax = [&](int g) {
        const uint8_t* c = &cnt[(size_t)g * R];
        uint8_t m = 0;
        for (int r = 0; r < R; ++r) m = m > c[r] ? m : c[r];
        return (int)m;
    };
    auto move = [&](int l, int from, int to) {
        for (int g : node_groups[l]) {
            cnt[(size_t)g * R + from]--;
            cnt[(size_t)g * R + to]++;
        }
    };
    std::vector<int> mark(ng, -1), aff;
    uint64_t rs = seed;
    for (int it = 0; it < iters && nloc > 1; ++it) {
        const int a = (int)(splitmix64(rs) % (uint64_t)nloc), b = (int)(splitmix64(rs) % (uint64_t)nloc);
        const int ra = perm[a] & (R - 1), rb = perm[b] & (R - 1);
        if (ra == rb) continue;
        aff.clear();
        for (int g : node_groups[a])
            if (mark[g] != it) mark[g] = it, aff.push_back(g);
        for (int g : node_groups[b])
            if (mark[g] != it) mark[g] = it, aff.push_back(g);
        int before = 0, after = 0;
        for (int g : aff) before += gmax(g);
        move(a, ra, rb);
        move(b, rb, ra);
        for (int g : aff) after += gmax(g);
        if (after <= before) {
            std::swap(perm[a], perm[b]);
        } else {
            move(a, rb, ra);
            move(b, ra, rb);
        }
    }
    for (int r = 0; r < R; ++r) {
        std::vector<int> nodes, slots;
        for (int l = 0; l < nloc; ++l)
            if ((perm[l] & (R - 1)) == r) nodes.push_back(l), slots.push_back(perm[l]);
        std::sort(slots.begin(), slots.end());
        std::stable_sort(nodes.begin(), nodes.end(), [&](int x, int y) { return deg[x] > deg[y]; });
        for (size_t i = 0; i < nodes.size(); ++i) perm[nodes[i]] = slots[i];
    }
}

// Orders each node's incidences (lists[k], entries (item << shift) + corner) so that the entries that
// lanes_per_read neighbouring lanes read in one step (bank pair = item mod 16) spread over the banks:
// step by step, lanes are matched with banks one to one as far as possible, and a lane left over takes
// the least used bank. The warp of node k is group(k) and its lanes run the group's nodes in increasing
// k. Returns the per-node ordered lists. Any fixed order keeps the sums identical from run to run.
template <typename Group>
std::vector<std::vector<int>> order_for_banks(std::vector<std::vector<int>> lists, int ngroups, Group group, int shift = 2,
                                              int lanes_per_read = kWarp) {
    constexpr int R = kBankPairs;
    const int nloc = (int)lists.size();
    std::vector<std::vector<int>> members(ngroups), ordered(nloc);
    for (int k = 0; k < nloc; ++k) members[group(k)].push_back(k);
    for (const std::vector<int>& mem : members) {
        const int nl = (int)mem.size();
        if (nl == 0) continue;
        int left[kWarp][R] = {};
        for (int i = 0; i < nl; ++i)
            for (int e : lists[mem[i]]) left[i % kWarp / lanes_per_read][(e >> shift) & (R - 1)]++;
        std::vector<int> lanes(nl);
        int depth = 0;
        for (int k : mem) depth = std::max(depth, (int)lists[k].size());
        for (int j = 0; j < depth; ++j) {
            int count[kWarp][R] = {};
            for (int i = 0; i < nl; ++i) lanes[i] = i;
            std::stable_sort(lanes.begin(), lanes.end(),
                             [&](int x, int y) { return lists[mem[x]].size() > lists[mem[y]].size(); });
            // augmenting paths, longest lists first, the banks with the most entries left first
            int owner[kWarp][R], take[kWarp];
            std::fill(&owner[0][0], &owner[0][0] + kWarp * R, -1);
            bool seen[R];
            auto bank = [&](int e) { return (e >> shift) & (R - 1); };
            auto augment = [&](auto&& self, int i) -> bool {
                const int h = i % kWarp / lanes_per_read;
                std::vector<int>& L = lists[mem[i]];
                for (;;) {
                    int best = -1;
                    for (int t = 0; t < (int)L.size(); ++t)
                        if (!seen[bank(L[t])] && (best < 0 || left[h][bank(L[t])] > left[h][bank(L[best])])) best = t;
                    if (best < 0) return false;
                    const int r = bank(L[best]), before = owner[h][r];
                    seen[r] = true;
                    if (before >= 0 && !self(self, before)) continue;
                    owner[h][r] = i;
                    take[i] = L[best];
                    return true;
                }
            };
            for (int i : lanes) {
                take[i] = -1;
                std::fill(seen, seen + R, false);
                augment(augment, i);
            }
            for (int i : lanes)
                if (take[i] >= 0) count[i % kWarp / lanes_per_read][bank(take[i])]++;
            for (int i : lanes) {
                std::vector<int>& L = lists[mem[i]];
                if (L.empty()) continue;
                const int h = i % kWarp / lanes_per_read;
                if (take[i] < 0) {
                    take[i] = *std::min_element(L.begin(), L.end(), [&](int x, int y) { return count[h][bank(x)] < count[h][bank(y)]; });
                    count[h][bank(take[i])]++;
                }
                left[h][bank(take[i])]--;
                ordered[mem[i]].push_back(take[i]);
                L.erase(std::find(L.begin(), L.end(), take[i]));
            }
        }
    }
    return ordered;
}

}  // namespace plb
