// CPU walk over the rows form's tile list for m-tile groups wider than one: every (m tile, output set, n tile) appears
// exactly once, groups are consecutive and the last one may be narrower.  Built and run by
// tests/test_rows_group.py (nvcc, host code only).
#include <cstdio>
#include <set>

#include "../mixture-of-kittens_b200/csrc/gemm_tiles.cuh"

using namespace mok::tiles;

int main() {
    for (int group : {0, 1, 2, 8})
        for (int m_tiles : {1, 7, 8, 9, 16, 23})
            for (int n_blocks : {1, 3, 16})
                for (int n_sets : {1, 2}) {
                    const int cum[2] = {0, (m_tiles + 2) * BM};
                    KernelParams p{};
                    p.num_experts = 1;
                    p.n_blocks = n_blocks;
                    p.n_sets = n_sets;
                    p.k_blocks = p.k_sets = 1;
                    p.m_group = group;
                    const int lo = BM, hi = lo + m_tiles * BM, per_group = (group > 1 ? group : 1) * n_blocks * n_sets;
                    std::set<long long> seen;
                    const int n = total_tiles<MODE_ROWS>(p, lo, hi);
                    for (int t = 0; t < n; ++t) {
                        Tile tile;
                        const bool work = decode_tile<MODE_ROWS, 64>(p, cum, lo, hi, t, tile);
                        const int m = (tile.row0 - lo) / BM;
                        if (!work || tile.row0 < lo || tile.row0 >= hi || tile.set >= n_sets || tile.n0 / BN >= n_blocks ||
                            m / (group > 1 ? group : 1) != t / per_group ||
                            !seen.insert((static_cast<long long>(m) * 8 + tile.set) * 1024 + tile.n0 / BN).second) {
                            std::printf("FAILED group %d m %d n %d sets %d tile %d\n", group, m_tiles, n_blocks, n_sets, t);
                            return 1;
                        }
                    }
                    if (static_cast<int>(seen.size()) != m_tiles * n_blocks * n_sets) return 1;
                }
    std::printf("ok\n");
    return 0;
}
