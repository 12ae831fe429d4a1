// Host check of the CTA-pair GEMM's work units: for many problem shapes and grids, every K tile of every output tile is
// in exactly one unit, units of one tile agree on their number of parts, scratch slots and shared-memory pieces stay in
// bounds, and the 32-column chunks of a split tile have exactly one owner.
#include <cstdio>
#include <cstring>
#include <vector>

#include "../../catccos_b200/csrc/mx_gemm_pair.cuh"

using namespace catccos;

static int check(uint32_t m, uint32_t n, uint32_t k, uint32_t max_pairs, uint32_t parts, bool gated)
{
    GemmParams p;
    memset(&p, 0, sizeof(p));
    uint32_t word = 0;
    p.flags = gated ? &word : nullptr;
    p.world = 1;
    p.Mg = m;
    p.N = n;
    p.K = k;
    const uint32_t tiles = ((m + 255) / 256) * ((n + 255) / 256);
    const PairGrid grid = pair_grid(tiles, max_pairs, parts);
    const uint32_t pairs = grid.pairs;
    p.ksplit = grid.ksplit;
    if (p.ksplit > k / 128) return 0;  // no part without a K tile is asked for
    if (pairs == 0 || pairs > max_pairs || p.ksplit < 1 || p.ksplit > (parts > 1 ? parts : 1)) return 6;
    std::vector<std::vector<int>> seen(tiles, std::vector<int>(k / 128, 0));
    std::vector<int> slots(max_pairs, 0);
    uint32_t readers = 0, split_units = 0;
    for (uint32_t pair = 0; pair < pairs; ++pair) {
        const PairWork w(p, pair, pairs);
        readers += pair < w.split_units() ? 1 : 0;
        split_units = w.split_units();
        for (uint32_t i = 0; i < w.units; ++i) {
            const PairUnit u = w.unit(i, p);
            const uint32_t tile = u.m0 / 256 * w.n_tiles + u.n_tile;
            if (tile >= tiles || u.kt0 >= u.kt1 || u.kt1 > k / 128 || u.n0 != u.n_tile * 256) return 1;
            if (u.width % 32 != 0 || u.width > 256 || u.n0 + u.width < (n < u.n0 + 256 ? n : u.n0 + 256)) return 5;
            if (u.last != (i + 1 == w.units) || (u.split && (gated ? !u.last : i != 0))) return 2;  // a split unit comes first, in a gated launch last
            if (u.split) {
                const uint32_t slot = u.rem_ix * w.ksplit + u.part;
                if (slot >= max_pairs || slots[slot]++ != 0) return 3;
            }
            for (uint32_t kt = u.kt0; kt < u.kt1; ++kt) seen[tile][kt]++;
        }
    }
    for (auto& t : seen) for (int c : t) if (c != 1) return 4;
    if (readers != split_units) return 7;  // the pairs that read the launch's epoch are as many as it is counted for
    for (uint32_t i = 0; i < max_pairs; ++i) if ((i < split_units) != (slots[i] == 1)) return 8;
    return 0;
}

int main()
{
    for (uint32_t pairs : {1u, 2u, 66u, 74u})
        for (uint32_t m : {1u, 255u, 257u, 1024u, 3001u, 32768u})
            for (uint32_t n : {16u, 256u, 272u, 2304u, 7168u})
                for (uint32_t k : {128u, 384u, 2304u, 7168u})
                    for (uint32_t parts = 1; parts <= kSplitKMax; ++parts)
                        if (int rc = check(m, n, k, pairs, parts, false) + 10 * check(m, n, k, pairs, parts, true)) {
                            printf("m %u n %u k %u pairs %u parts %u: %d\n", m, n, k, pairs, parts, rc);
                            return 1;
                        }
    for (uint32_t chunks : {4u, 8u})
        for (uint32_t parts = 2; parts <= (chunks < kSplitKMax ? chunks : kSplitKMax); ++parts) {
            uint32_t next = 0;
            for (uint32_t part = 0; part < parts; ++part) {
                const uint32_t own0 = (part * chunks + parts - 1) / parts, own1 = ((part + 1) * chunks + parts - 1) / parts;
                if (own0 != next || own1 <= own0 || (own1 - own0) * (parts - 1) * kSplitPieceBytes > kSplitRedBytes) return 1;
                next = own1;
            }
            if (next != chunks) return 1;
        }
    puts("pair work ok");
    return 0;
}
