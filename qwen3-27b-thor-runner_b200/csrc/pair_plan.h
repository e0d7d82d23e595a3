// Tile plan and work list of the prefill kernel on pairs of SMs (prefill_pair.cu): plain arithmetic, no CUDA types, so that a
// test can walk every plan on the CPU.
#pragma once
#include <cmath>

#ifdef __CUDACC__
#define NVFP4_HD __host__ __device__ __forceinline__
#else
#define NVFP4_HD inline
#endif

namespace nvfp4 {
namespace pair {

constexpr int TR = 128;                        // weight rows per CTA and row tile (TMEM lanes); 256 per pair
constexpr int BK = 64;                         // k per operand block (128 bytes of 16-bit elements: one swizzle row)
constexpr int WK = 256;                        // k per raw weight stage and per scheduling unit
constexpr int kBlocks = WK / BK;
constexpr int kWPackedBytes = TR * WK / 2;     // 16 KB
constexpr int kWScaleBytes = TR * WK / 16;     // 2 KB
constexpr int kWStageBytes = kWPackedBytes + kWScaleBytes;
constexpr int XK = 128;                        // k per token stage and planned A unit (two operand blocks)
constexpr int kDenseBlockBytes = TR * BK * 2;  // 16 KB
constexpr int kDenseUnitBytes = 2 * kDenseBlockBytes;
constexpr int kUnitCols = XK / 2;              // 64 TMEM columns of FP16 pairs per A unit (128 rows x 128 k)
constexpr int kMaxUnits = 8, kMaxX = 8, kMaxW = 8, kMaxAccs = 4;
constexpr int kBarBytes = 2048;                // barriers, token factors, a few words
constexpr int kSmemMax = 225 * 1024;
constexpr int kRaster = 8;                     // token tiles that consecutive items share a row group over

struct Plan {
    int M, N, K;
    int T;                     // tokens per tile
    int m_tiles, row_tiles;    // row tiles of 256
    int R;                     // row tiles per item
    int items, dp_items;       // items [0, dp_items) run whole, the rest is split by k, one row tile at a time
    int sk_tiles;              // (items - dp_items) * R
    int w_stages, x_stages, units, accs, a_col0;
};

// ---------------------------------------------------------------- work list
struct Item {
    int rt, rows;      // first row tile, number of row tiles (1 or 2)
    int mt;            // token tile
    int ks0, ks1;      // 256-k stages
    int sk;            // split tile index, -1 = whole
};
struct Work {          // of pair `id` of `pairs`
    long long u, u_end;
    int dp, kst, pairs;
    NVFP4_HD Work(const Plan& p, int kstages, int pairs_, int id) {
        pairs = pairs_;
        const long long units = (long long)p.sk_tiles * kstages;
        u = (long long)id * units / pairs;
        u_end = (long long)(id + 1) * units / pairs;
        dp = id;
        kst = kstages;
    }
    // item index -> first row tile and token tile: blocks of kRaster token tiles, row groups outside them
    NVFP4_HD static void place(const Plan& p, int item, int& rg, int& mt) {
        const int groups = (p.row_tiles + p.R - 1) / p.R;
        const int blk = item / (kRaster * groups), rem = item - blk * (kRaster * groups);
        const int left = p.m_tiles - blk * kRaster, width = left < kRaster ? left : kRaster;
        rg = rem / width;
        mt = blk * kRaster + rem - rg * width;
    }
    NVFP4_HD bool next(const Plan& p, Item& t) {
        int rg;
        if (u < u_end) {
            t.sk = (int)(u / kst);
            t.ks0 = (int)(u % kst);
            const long long room = u_end - u;
            t.ks1 = (kst - t.ks0) < room ? kst : t.ks0 + (int)room;
            u += t.ks1 - t.ks0;
            place(p, p.dp_items + t.sk / p.R, rg, t.mt);
            t.rt = rg * p.R + t.sk % p.R;      // may lie beyond the last row tile (odd number, two an item): rows of zeros, not stored
            t.rows = 1;
            return true;
        }
        if (dp < p.dp_items) {
            place(p, dp, rg, t.mt);
            t.rt = rg * p.R;
            const int left = p.row_tiles - t.rt;
            t.rows = left < p.R ? left : p.R;
            t.ks0 = 0;
            t.ks1 = kst;
            t.sk = -1;
            dp += pairs;
            return true;
        }
        return false;
    }
};

// The kernel's ring of A units: the planned ones of 128 k, or two of 64 k for each ("fine") and in tensor memory (NVFP4) two more in an odd
// 64 columns (`spare_units` of them).  Two groups of warps take every other unit: an even number.
// NVFP4 takes 64 k where tensor memory has room for two units of 128 k only, above 128 tokens a tile.  BF16, whose blocks lie in shared
// memory, takes it up to 128 tokens a tile; beyond, a unit of 64 k is twice the waits and commits, but one row tile a turn takes two
// token stages of few when its unit is 128 k.  So an item of two row tiles has 128 k (4096 x 5120 x 17408 at T = 192 530 us with 64 k,
// 510 with 128, 4096 x 34816 x 5120 at T = 160 1145 and 1077), one of one row tile 64 k (480 x 5120 x 17408 67.9 and 78.2), which
// goes for plans with a tenth of their tiles in parts too (20 of 168 104.0 and 105.5, 96 of 392 244 and 260, but 8 of 896 520 and 502).
// At T = 160 and one or two token tiles the weights' stream is the bound and 64 k is 1 % ahead (320 x 34816 x 5120 87.5 and 88.3).
constexpr int kCoarseT = 128;
constexpr int kRingMax = 2 * kMaxUnits;
NVFP4_HD bool fine_units(const Plan& p, bool dense) {
    if (!dense) return p.T > kCoarseT;
    const bool parts = 10LL * p.sk_tiles >= (long long)p.items * p.R;
    return p.T <= kCoarseT || p.R == 1 || parts || (p.T <= 160 && p.m_tiles <= 2);
}
NVFP4_HD int spare_units(const Plan& p, bool dense) { return !dense && fine_units(p, dense) ? (p.a_col0 - p.accs * p.T) / kUnitCols * 2 : 0; }
NVFP4_HD int ring_units(const Plan& p, bool dense) { return fine_units(p, dense) ? 2 * p.units + spare_units(p, dense) : p.units; }

// Pairs first..last hold the parts of split tile `tile`, of which pair `id` holds one; the first one holds its head (slot 1),
// the others a middle or tail (slot 0).
NVFP4_HD void participants(const Plan& p, int kstages, int pairs, int id, int tile, int& first, int& last) {
    const long long units = (long long)p.sk_tiles * kstages;
    const long long b = (long long)tile * kstages, e = b + kstages;
    first = last = id;
    while (first > 0 && (long long)first * units / pairs > b) --first;
    while (last + 1 < pairs && (long long)(last + 1) * units / pairs < e) ++last;
}

// Clocks, fitted to the times of all plans for each weight form alone, with the kernel as it was when its groups of dequantising warps took
// a half of every unit: an MMA took 100 to 120 clocks then and takes 75 (T = 128), 81 (160) or 110 (192) now, and drains and parts
// cost less.  They were not fitted again since; how far the plans they choose are from the best ones today has not been measured.
struct Prices {
    double mma;            // one MMA at least (alone 65: the issuing warps share their schedulers with the dequantising ones)
    double rate;           // bytes a clock of both operand streams of an SM
    double block_bytes;    // of 64 k of a row tile's weights
    double last_token;     // drain of the last item, per token and row tile
    double item_token, item;   // of an item, what the next one's MMAs do not hide
    double split, split_token, part;   // everything split: parts stored, flags, sums; `part`: one more holder of a tile (a round trip of the readers)
    double straddle;       // parts that straddle tiles: a pair then holds two
    double tail, tail_token;   // splitting what whole waves leave, which hide the reduction
    double pair;           // each pair that takes part: launch, the same weights and tokens read once more
};
constexpr Prices kPricesFp4 = {95.0, 37.0, 4608.0, 3.2, 5.4, 650.0, 7100.0, 27.0, 750.0, 7800.0, 3600.0, 76.0, 9.0};
constexpr Prices kPricesBf16 = {73.5, 68.0, 16384.0, 6.2, 18.8, 1060.0, 7900.0, 35.5, 600.0, 11400.0, 670.0, 188.0, 46.0};

// Fills the tile plan of a launch (p.M, p.N and p.K are set) for at most `pairs` CTA pairs; returns the pairs it runs on, and the
// dynamic shared memory of a CTA in *smem.  `prices` choose among plans that are all valid.
inline int make_plan(Plan& p, int pairs, bool stream_k, bool dense, int* smem, const Prices* prices = nullptr) {
    const int kst = p.K / WK;
    p.row_tiles = (p.N + 2 * TR - 1) / (2 * TR);
    // T up to 192: two accumulators and two 64-column A units (four of 64 k in the kernel) fill tensor memory.  BF16 weights: up to 224,
    // four 32 KB A units and three token stages; from 192 on only with two row tiles an item (one row tile takes two token stages a
    // turn: 512 x 5120 x 8192 at T = 192 64 us, at T = 128 40) and never split all over.
    const int t_max = dense ? 224 : 192;
    // Every plan -- T, row tiles per item (R), items left over after whole waves run whole or split by k -- is priced in clocks,
    // with constants fitted to all plans of some 300 shapes of each weight form (17 to 2048 tokens, N 512 to 34816, K 1024 to
    // 17408, weights from memory): the plan chosen was 0.2 (BF16 1.0) % slower than the best one on average, 1.4 (5.6) at the 95th
    // percentile, for the kernel they were fitted to.  The list before it was fitted to large weights only, charged 23,500 clocks for
    // any split and had none for fewer stages than pairs: 65 x 512 x 5120 ran whole in 25 us, 14 split.
    const Prices& c = prices ? *prices : dense ? kPricesBf16 : kPricesFp4;
    double best = 1e30;
    int used = 1;
    for (int T = 32; T <= t_max; T += 32) {
        if (T > 32 && T - 32 >= p.M) break;                        // a smaller tile already holds all tokens
        const int mt = (p.M + T - 1) / T, tokens = p.M < T ? p.M : T;
        for (int R = dense && T > 160 ? 2 : 1; R <= (p.row_tiles > 1 ? 2 : 1); ++R) {
            const long long items = (long long)((p.row_tiles + R - 1) / R) * mt;
            // clocks of one 64-k block of an item, of one row tile: the MMAs, or the bytes of both streams
            const double mma = 4.0 * (T / 2 > c.mma ? T / 2 : c.mma);
            const double blk = std::fmax(R * mma, (T * 64.0 + R * c.block_bytes) / c.rate);
            const double blk1 = std::fmax(mma, (T * 64.0 + c.block_bytes) / c.rate);
            const long long full = items / pairs, left = items % pairs, sk = left * R;
            const double item = kst * kBlocks * blk + c.item_token * tokens * R + c.item;
            auto take = [&](double cost, bool split, long long on) {
                if (cost >= best) return;
                best = cost;
                p.T = T; p.R = R; p.m_tiles = mt;
                p.items = (int)items;
                p.dp_items = split ? (int)(full * pairs) : (int)items;
                p.sk_tiles = split ? (int)sk : 0;
                used = (int)on;
            };
            take((full + (left ? 1 : 0)) * item + c.last_token * tokens * R + c.pair * (full ? pairs : left), false, full ? pairs : left);
            if (!left || !stream_k) continue;
            if (full) {
                if (sk * kst >= pairs)                             // every pair has a part: a holder's neighbours are holders
                    take(full * item + (double)((sk * kst + pairs - 1) / pairs) * kBlocks * blk1 + c.tail + c.tail_token * tokens + c.pair * pairs,
                         true, pairs);
                continue;
            }
            if (R == 2) continue;                                  // parts are of one row tile each: two an item change nothing
            const long long most = pairs / sk < kst ? pairs / sk : kst;
            if (most >= 2) {
                // S parts a tile on S * sk pairs, no pair on two tiles.  More parts are shorter, each costs c.part: the price is
                // least near sqrt(kst * kBlocks * blk1 / c.part) parts; the whole numbers of stages around that, and `most`.
                const int stages = (int)(kst / std::sqrt(kst * kBlocks * blk1 / c.part));
                for (int i = 0; i < 3; ++i) {
                    const int want = stages + i < 1 ? 1 : stages + i;
                    long long S = i == 2 ? most : (kst + want - 1) / want;
                    if (S > most) S = most;
                    if (S < 2) S = 2;
                    const long long each = (kst + S - 1) / S;
                    S = (kst + each - 1) / each;                   // no more parts than that many stages each need
                    take((double)each * kBlocks * blk1 + c.split + c.split_token * tokens + c.part * S + c.pair * S * sk, true, S * sk);
                }
            }
            const long long on = sk * kst < pairs ? sk * kst : pairs;
            if ((sk * kst + on - 1) / on < kst)                    // no part is a whole tile: the kernel for plans split all over has none
                take((double)((sk * kst + on - 1) / on) * kBlocks * blk1 + c.split + 2.0 * c.split_token * tokens + c.part * on / sk +
                         c.straddle + c.pair * on,
                     true, on);
        }
    }
    const int xbytes = p.T / 2 * (XK * 2);
    if (dense) {
        p.accs = p.T <= 128 ? 4 : 2;
        p.units = 4;
        p.w_stages = 0;
    } else {
        p.accs = p.T <= 64 ? 4 : 2;
        p.units = (512 - p.accs * p.T) / kUnitCols / 2 * 2;
        if (p.units > kMaxUnits) p.units = kMaxUnits;
        p.w_stages = p.T <= 64 ? 8 : 6;
        p.a_col0 = 512 - p.units * kUnitCols;
    }
    const int wbytes = dense ? p.units * kDenseUnitBytes : p.w_stages * kWStageBytes;
    p.x_stages = (kSmemMax - 1024 - kBarBytes - wbytes) / xbytes;
    if (p.x_stages > kMaxX) p.x_stages = kMaxX;
    *smem = 1024 + p.x_stages * xbytes + wbytes + kBarBytes;
    return used;
}

}  // namespace pair
}  // namespace nvfp4
