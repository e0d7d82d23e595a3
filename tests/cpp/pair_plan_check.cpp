// The prefill kernel's plan and work list (csrc/pair_plan.h) for a test on the CPU.
#include <vector>

#include "pair_plan.h"

using namespace nvfp4::pair;

extern "C" {

// out: T, R, m_tiles, row_tiles, items, dp_items, sk_tiles, w_stages, x_stages, units, accs, a_col0, smem, pairs used, units of the ring
void pair_plan(int M, int N, int K, int pairs, int stream_k, int dense, int* out) {
    Plan p{};
    p.M = M; p.N = N; p.K = K;
    int smem = 0;
    const int used = make_plan(p, pairs, stream_k != 0, dense != 0, &smem);
    const int v[] = {p.T, p.R, p.m_tiles, p.row_tiles, p.items, p.dp_items, p.sk_tiles, p.w_stages, p.x_stages, p.units, p.accs, p.a_col0, smem, used,
                     ring_units(p, dense != 0)};
    for (int i = 0; i < (int)(sizeof v / sizeof v[0]); ++i) out[i] = v[i];
}

// Whether the plan's units are 64 k.
int pair_fine(int M, int N, int K, int pairs, int dense) {
    Plan p{};
    p.M = M; p.N = N; p.K = K;
    int smem = 0;
    make_plan(p, pairs, true, dense != 0, &smem);
    return fine_units(p, dense != 0);
}

// Walks all pairs' lists.  0: every (row tile, token tile, k stage) that holds outputs is worked on exactly once, no pair writes a
// partial slot twice, every holder of a split tile's part names the same holders, whose slots hold it, and a plan that is split
// all over has no part that is a whole tile.  `prices`: the kernel's own (0), or splitting costs nothing (1: whole parts would be cheapest).
int pair_walk(int M, int N, int K, int pairs, int stream_k, int dense, int prices) {
    Plan p{};
    p.M = M; p.N = N; p.K = K;
    int smem = 0;
    Prices split_free = dense ? kPricesBf16 : kPricesFp4;
    split_free.split = split_free.split_token = split_free.part = split_free.straddle = split_free.tail = split_free.tail_token = split_free.pair = 0.0;
    const int used = make_plan(p, pairs, stream_k != 0, dense != 0, &smem, prices ? &split_free : nullptr), kst = K / WK;
    if (used < 1 || used > pairs) return 1;
    std::vector<unsigned char> seen((size_t)p.row_tiles * p.m_tiles * kst, 0);
    std::vector<std::vector<int>> slot(used, std::vector<int>{-1, -1});      // split tile in the pair's slots (tail or middle, head)
    for (int id = 0; id < used; ++id) {
        Work w(p, kst, used, id);
        Item t;
        while (w.next(p, t)) {
            if (t.rows < 1 || t.rows > 2 || t.mt < 0 || t.mt >= p.m_tiles || t.ks0 < 0 || t.ks1 > kst || t.ks0 >= t.ks1) return 2;
            for (int r = 0; r < t.rows; ++r) {
                if (t.rt + r >= p.row_tiles) {
                    if (t.sk < 0 || p.R != 2) return 3;
                    continue;
                }
                for (int k = t.ks0; k < t.ks1; ++k)
                    if (seen[((size_t)(t.rt + r) * p.m_tiles + t.mt) * kst + k]++) return 4;
            }
            if (p.dp_items == 0 && t.sk >= 0 && t.ks0 == 0 && t.ks1 == kst) return 9;
            if (t.sk >= 0 && (t.ks0 || t.ks1 < kst)) {
                int& s = slot[id][t.ks0 == 0];
                if (s >= 0) return 5;
                s = t.sk;
            }
        }
    }
    for (unsigned char c : seen) if (!c) return 6;
    for (int id = 0; id < used; ++id)
        for (int which = 0; which < 2; ++which)
            if (slot[id][which] >= 0) {
                int first, last;
                participants(p, kst, used, id, slot[id][which], first, last);
                if (first == last || id < first || id > last) return 7;
                for (int c = first; c <= last; ++c)
                    if (slot[c][c == first] != slot[id][which]) return 8;
            }
    return 0;
}

}  // extern "C"
