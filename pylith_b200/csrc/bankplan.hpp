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
    std::vector<int> cnt((size_t)ng * R, 0);
    for (int l = 0; l < nloc; ++l)
        for (int g : node_groups[l]) cnt[(size_t)g * R + (perm[l] & (R - 1))]++;
    auto gmax = [&](int g) {
        const int* c = &cnt[(size_t)g * R];
        int m = 0;
        for (int r = 0; r < R; ++r) m = m > c[r] ? m : c[r];
        return m;
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
std::vector<std::vector<int>> order_for_banks(const std::vector<std::vector<int>>& lists, int ngroups, Group group, int shift = 2,
                                              int lanes_per_read = kWarp) {
    constexpr int R = kBankPairs, H = 2;  // a warp's reads go through in H groups of lanes at most
    const int nloc = (int)lists.size();
    std::vector<std::vector<int>> members(ngroups), ordered(nloc);
    for (int k = 0; k < nloc; ++k) members[group(k)].push_back(k);
    // a lane's entries by bank: those of bank r that are left are entries[at[r]] .. entries[end[r]]
    struct Lane {
        int at[R], end[R], left;
        uint32_t banks;  // with entries left
    };
    std::vector<int> entries, lanes, take, first;
    std::vector<Lane> lane;
    for (const std::vector<int>& mem : members) {
        const int nl = (int)mem.size();
        if (nl == 0) continue;
        int left[H][R] = {};  // entries left of all lanes
        lane.resize(nl);
        entries.clear();
        int depth = 0;
        for (int i = 0; i < nl; ++i) {
            Lane& L = lane[i];
            const std::vector<int>& list = lists[mem[i]];
            L.left = (int)list.size();
            L.banks = 0;
            depth = std::max(depth, L.left);
            int n[R] = {}, at = (int)entries.size();
            for (int e : list) n[(e >> shift) & (R - 1)]++;
            for (int r = 0; r < R; ++r) {
                L.at[r] = L.end[r] = at;
                at += n[r];
                L.banks |= (uint32_t)(n[r] > 0) << r;
                left[i % kWarp / lanes_per_read][r] += n[r];
            }
            entries.resize(at);
            for (int e : list) entries[L.end[(e >> shift) & (R - 1)]++] = e;
            ordered[mem[i]].reserve(list.size());
        }
        lanes.resize(nl);
        take.resize(nl);
        first.resize(depth + 2);
        for (int j = 0; j < depth; ++j) {
            // lanes with the longest lists first
            std::fill(first.begin(), first.end(), 0);
            for (int i = 0; i < nl; ++i) first[depth - lane[i].left + 1]++, take[i] = -1;
            for (int d = 0; d < depth; ++d) first[d + 1] += first[d];
            for (int i = 0; i < nl; ++i) lanes[first[depth - lane[i].left]++] = i;
            // augmenting paths, longest lists first, the banks with the most entries left first
            int owner[H][R], count[H][R] = {};
            std::fill(&owner[0][0], &owner[0][0] + H * R, -1);
            uint32_t seen;
            auto augment = [&](auto&& self, int i) -> bool {
                const int h = i % kWarp / lanes_per_read;
                while (const uint32_t open = lane[i].banks & ~seen) {
                    int best = __builtin_ctz(open);
                    for (uint32_t o = open & (open - 1); o; o &= o - 1)
                        if (left[h][__builtin_ctz(o)] > left[h][best]) best = __builtin_ctz(o);
                    seen |= 1u << best;
                    const int before = owner[h][best];
                    if (before >= 0 && !self(self, before)) continue;
                    owner[h][best] = i;
                    take[i] = best;
                    return true;
                }
                return false;
            };
            int unowned[H] = {};  // banks with entries left and no owner
            for (int h = 0; h < H; ++h)
                for (int r = 0; r < R; ++r) unowned[h] += left[h][r] > 0;
            for (int i : lanes) {
                const int h = i % kWarp / lanes_per_read;
                if (lane[i].left == 0) break;
                seen = 0;
                if (unowned[h] > 0 && augment(augment, i)) unowned[h]--;
            }
            for (int i : lanes)
                if (take[i] >= 0) count[i % kWarp / lanes_per_read][take[i]]++;
            for (int i : lanes) {
                Lane& L = lane[i];
                if (L.left == 0) break;
                const int h = i % kWarp / lanes_per_read;
                if (take[i] < 0) {
                    for (int r = 0; r < R; ++r)
                        if (L.banks >> r & 1 && (take[i] < 0 || count[h][r] < count[h][take[i]])) take[i] = r;
                    count[h][take[i]]++;
                }
                const int r = take[i];
                left[h][r]--;
                L.left--;
                ordered[mem[i]].push_back(entries[L.at[r]++]);
                if (L.at[r] == L.end[r]) L.banks &= ~(1u << r);
            }
        }
    }
    return ordered;
}

}  // namespace plb
