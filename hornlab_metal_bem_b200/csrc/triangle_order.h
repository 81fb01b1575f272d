// Host-side triangle order of the tiled assembly (no CUDA: also compiled by
// itself in the tests).
#pragma once
#include <algorithm>
#include <vector>

namespace hbem {

constexpr int kOrderScan = 64;   // open triangles of a dof looked at per step

// Triangle order of the tiled assembly.  Chunks of chunk_len and tiles of
// tile_len consecutive triangles should touch few distinct dofs, and a
// triangle should share an edge with the one before it.  Grown greedily over
// the mesh: the next triangle touches the chunk (else the tile, the previous
// tile, or comes first in `seed`) and brings the fewest new dofs to the chunk,
// then to the tile, shares most dofs with the last triangle and leaves the
// fewest open neighbours.  A dof offers at most `scan` of its open triangles
// (each step would otherwise look at every triangle about an apex: 20 000
// around one took 4.1 s; its rim vertices offer the neighbours in any case).
// On the quarter horn of 1950 triangles: 29 dofs a tile and 9.9 a chunk,
// against 35 and 14 in Morton order alone.
inline void cluster_order(const std::vector<int> &l2g, int n_dof, const std::vector<int> &seed, int chunk_len,
                          int tile_len, int scan, std::vector<int> &order) {
    const int T = (int)seed.size();
    std::vector<int> start(n_dof + 1, 0), end, inc(3 * (size_t)T), rank(T), open(n_dof, 0);
    for (int v : l2g) { ++start[v + 1]; ++open[v]; }
    for (int v = 0; v < n_dof; ++v) start[v + 1] += start[v];
    // inc[start[v] .. end[v]): triangles with dof v; used ones leave when they are met
    end.assign(start.begin(), start.end() - 1);
    for (int t = 0; t < T; ++t)
        for (int l = 0; l < 3; ++l) inc[end[l2g[3 * t + l]]++] = t;
    for (int i = 0; i < T; ++i) rank[seed[i]] = i;
    std::vector<char> used(T, 0);
    // stamps: the chunk, tile and previous tile a dof belongs to last
    std::vector<int> chunk_of(n_dof, -1), tile_of(n_dof, -1);
    // last_of: the position of the last triangle with that dof; seen: the last
    // position a triangle was a candidate for
    std::vector<int> chunk, tile, prev_tile, last_of(n_dof, -2), seen(T, -1);
    order.clear();
    order.reserve(T);
    int next_seed = 0;
    while ((int)order.size() < T) {
        const int pos = (int)order.size(), ci = pos / chunk_len, ti = pos / tile_len;
        if (pos % tile_len == 0) { prev_tile.swap(tile); tile.clear(); }
        if (pos % chunk_len == 0) chunk.clear();
        int best = -1;
        long long best_key = 0;
        const std::vector<int> *pools[3] = {&chunk, &tile, &prev_tile};
        for (int lvl = 0; lvl < 3 && best < 0; ++lvl)
            for (int v : *pools[lvl])
                for (int e = start[v]; e < end[v] && e - start[v] < scan;) {
                    const int u = inc[e];
                    if (used[u]) {
                        inc[e] = inc[--end[v]];
                        continue;
                    }
                    ++e;
                    if (seen[u] == pos) continue;
                    seen[u] = pos;
                    int new_c = 0, new_t = 0, with_last = 0, left = 0;
                    for (int l = 0; l < 3; ++l) {
                        const int d = l2g[3 * u + l];
                        new_c += chunk_of[d] != ci;
                        new_t += tile_of[d] != ti;
                        with_last += last_of[d] == pos - 1;
                        left += open[d];
                    }
                    // lexicographic: smallest first
                    const int k0 = lvl == 0 ? new_c * 4 + new_t : (lvl == 1 ? new_t : 0);
                    const int k1 = lvl == 0 ? 3 - with_last : left, k2 = lvl == 0 ? left : 3 - with_last;
                    const long long key = (((long long)k0 << 10 | std::min(k1, 1023)) << 10 | std::min(k2, 1023)) << 32 |
                                          (unsigned)rank[u];
                    if (best < 0 || key < best_key) {
                        best = u;
                        best_key = key;
                    }
                }
        if (best < 0) {
            while (used[seed[next_seed]]) ++next_seed;
            best = seed[next_seed];
        }
        used[best] = 1;
        order.push_back(best);
        for (int l = 0; l < 3; ++l) {
            const int d = l2g[3 * best + l];
            --open[d];
            last_of[d] = pos;
            if (chunk_of[d] != ci) { chunk_of[d] = ci; chunk.push_back(d); }
            if (tile_of[d] != ti) { tile_of[d] = ti; tile.push_back(d); }
        }
    }
}

}  // namespace hbem
