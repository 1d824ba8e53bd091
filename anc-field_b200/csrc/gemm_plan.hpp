// Which of its forms a GEMM is launched in. Host arithmetic only, so that the
// rule can be checked against measured times without a GPU.
#pragma once

#include <cstdint>
#include <utility>
#include <vector>

namespace afd {
namespace mlp {

constexpr int TM = 128, TN = 128, TK = 64;  // tile of k_gemm, and a step over K
constexpr int PTN = 256;                    // columns of a tile of the persistent forms

// How a GEMM is launched: kPair, kPersist, kDual (k_gemm), else the columns of
// k_gemm_tile's tiles, with the CTAs that share a tile's K range.
enum : int { kPair = 0, kPersist = 1, kDual = 2 };
struct GemmPlan {
    int form, split;
};

// The time of a form in us: start, waves of tiles, per wave its epilogue and
// its steps over K. The constants are fitted to every form's time on 600 sizes
// of 128 .. 16384 rows and columns and 64 .. 16384 deep, of which these are a few
// (M x N x K, us on the device):
//                   pair  persist  dual  tile 128   64    32
//    256x256x64     10.4    10.4    6.3      7.3   6.3   6.3
//   1024x512x512    12.5    12.5    8.4      8.4   6.8   6.3
//   1024x512x2048   20.6    18.6   14.5     12.4  10.4  10.4
//   1024x2048x4096  29.2    28.8   20.6     19.5  29.4  51.4
//   1920x2176x1024    -       -    16.5     20.6  26.8  39.0
//   2048x2048x2048  20.7    20.6   20.7     24.7  37.0  55.4
//   3712x1024x320     -     11.1   12.5     14.5    -     -
//   6016x3840x256     -     53.5   58.5     74.0    -     -
//   9216x768x1600   35.1    35.1   39.2     38.0  53.5  84.6
//  13952x512x12608    -    161.8  180.9    180.4    -     -
//   4096x4096x4096   105     120    125      139     -     -
// The 256-column forms pay a start and an epilogue of their own (10 us even
// for one tile) and fill the chip from 74 and 148 tiles on; below that the
// smaller tiles reach more SMs. Two tiles of k_gemm side by side on an SM share
// its loads and stores; a last round with one tile an SM is shorter. Tiles of
// k_gemm_tile in many waves are bound by L2. A split pays a cluster launch of 4
// us: 128x2048x8192 runs 26.8 as 64-column tiles, 14.5 split four ways and 45.2
// as persistent tiles. On those 600 sizes the form chosen takes 0.5 % longer than
// the fastest on average, and longer than the largest tiles that the sizes allow
// at one only, by 8 % (with all rounds of k_gemm counted alike 1.2 %, and at 26 of
// them by 3 to 19 %); on 250 others at one, by 10 %.
inline double gemm_cost(int form, int split, int64_t tiles, int K, int sms) {
    const int kt = K / TK;
    if (form == kPair) return 8.0 + (double)((tiles + sms / 2 - 1) / (sms / 2)) * (3.0 + 0.34 * kt);
    const int64_t waves = (tiles * split + sms - 1) / sms;
    if (form == kPersist) return 7.7 + (double)waves * (3.0 + 0.345 * kt);
    if (form == kDual) {
        const int64_t rounds = tiles / (2 * sms), rest = tiles % (2 * sms);
        const double both = 5.9 + 0.46 * kt;
        double last = 0.0;
        if (rest > sms) last = both;
        else if (rest > 0) last = 3.3 + (rounds ? 0.36 : 0.225) * kt;
        return 4.0 + (double)rounds * both + last;
    }
    const double step = (form == 128 ? 0.38 : form == 64 ? 0.325 : 0.29) * (waves > 2 ? 1.32 : waves > 1 ? 1.25 : 1.0);
    return 3.0 + (double)waves * (3.3 + 0.01 * form + step * ((kt / 2 + split) / split)) + (split > 1 ? 4.0 : 0.0);
}

inline GemmPlan plan_gemm(int M, int N, int K, bool may_split, int sms) {
    const int64_t mt = M / TM;
    GemmPlan best{kDual, 1};
    double cost = gemm_cost(kDual, 1, mt * (N / TN), K, sms);
    auto consider = [&](int form, int split, int64_t tiles) {
        const double c = gemm_cost(form, split, tiles, K, sms);
        if (c < cost) {
            cost = c;
            best = GemmPlan{form, split};
        }
    };
    if (M % (2 * TM) == 0 && N % PTN == 0 && sms >= 2) consider(kPair, 1, mt / 2 * (N / PTN));
    if (N % PTN == 0) consider(kPersist, 1, mt * (N / PTN));
    for (int tn : {128, 64, 32})
        for (int split : {1, 2, 4, 8}) {
            const int64_t tiles = mt * (N / tn);
            // shares of at least two steps; all clusters resident at once (of
            // eight CTAs only two fit a GPC, and not every one: 16 of them
            // took two rounds)
            if (split > 1 && (!may_split || K / TK < 4 * split || tiles * split > (split == 8 ? sms * 2 / 3 : sms - 16)))
                continue;
            consider(tn, split, tiles);
        }
    return best;
}

// Tile columns with which GEMMs of M x N = `sizes` and one K run in one
// launch, or -1 where one by one is faster.
inline int plan_group(const std::vector<std::pair<int, int>>& sizes, int K, int sms) {
    double alone = 0.0;
    int best = -1;
    for (const auto& z : sizes) {
        const GemmPlan p = plan_gemm(z.first, z.second, K, false, sms);
        const int th = p.form == kPair ? 2 * TM : TM, tw = p.form >= 32 ? p.form : p.form == kDual ? TN : PTN;
        alone += gemm_cost(p.form, 1, (int64_t)(z.first / th) * (z.second / tw), K, sms);
    }
    for (int tn : {128, 64, 32}) {
        int64_t tiles = 0;
        for (const auto& z : sizes) tiles += (int64_t)(z.first / TM) * (z.second / tn);
        const double c = gemm_cost(tn, 1, tiles, K, sms);
        if (c < alone) {
            alone = c;
            best = tn;
        }
    }
    return best;
}

}  // namespace mlp
}  // namespace afd
