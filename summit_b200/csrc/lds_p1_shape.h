// Phase 1's launch shape from the member lists' lengths (host code without CUDA,
// so that the CPU tests compile it as it is).
#pragma once
#include <algorithm>
#include <cstdint>
#include <map>

namespace lds {
namespace umma {

// Member SNPs per phase-1 K-step: member lists are padded to a multiple of it.
constexpr int kP1Step = 64;

constexpr int64_t kMaxGridY = 65535;   // CTAs along a grid's y, where the super-bins lie
constexpr int kPlainWindowed = 8;

// Super-bins per CTA for the member lists off[0..K] over `tiles` sample tiles;
// `period` super-bins make a window.  `plain` is the number without a choice:
// kPlainWindowed, or 1 for a genome-wide plan.
//
// The number with the earliest estimated end of the launch.  A CTA pays about
// 10,000 cycles before its pipeline runs, then per super-bin the epilogue's
// share and its K-steps (fits of measured launches); tiles CTAs
// of each group go to the SMs in launch order.  Beyond 12 waves the sum and half
// the longest CTA stand for that walk.  More per CTA than needed leave a long last
// wave and mix long lists with short ones; hence whole windows or even parts of
// one, up to 64, and the plain number: a K with few divisors (97: only 1) has no
// other near the best (N = 20,000, M = 12,000, K = 97, B = 20: 1 per CTA 4.04 ms, 8
// 1.79; N = 5,000, M = 9,000, K = 67: 696 and 303 us).  Another has to be estimated
// a twentieth earlier than the plain number: below that there was no gain
// (N = 5,000, M = 3,000, K = 47, B = 20: 47 per CTA, 0.4 % earlier, 104 us, 8 92;
// one window of 2,000 SNPs, N = 10,000, K = 13, B = 10: 13, 0.4 % earlier, 34.8, 8
// 30.7).  A genome-wide plan's plain number is 1 because its few long lists lose by
// 8 where the estimate gains (N = 10,000, M = 20,000, K = 11, B = 20: 98 and 109 us).
// Windowed, 8 per CTA -> this choice: N = 50,000, M = 60,000, K = 24, B = 50:
// 8.1 -> 7.2 ms; N = 10,007, K = 6, B = 10: 113 -> 104 us; genome-wide, 1 per CTA ->
// this choice: N = 50,000, M = 40,000, K = 24, B = 50: 1.95 -> 1.75 ms.
inline int choose_sb_per_cta(const int64_t* off, int K, int ncolp, int64_t tiles, int period,
                             int plain) {
    constexpr double kSms = 148.0, kStart = 10000.0;
    const double per_job = 2000.0 * ((ncolp + 255) / 256);
    const double per_member = (200.0 + 1.5 * ncolp) / kP1Step;
    // the fewest per CTA whose CTAs fit the grid
    const int fit = (int)((K + kMaxGridY - 1) / kMaxGridY);
    int best = std::max(fit, 1);
    double least = -1.0, plain_end = -1.0;
    for (int s = best; s <= std::min(K, std::max(64, fit)); ++s) {
        if (s % period != 0 && period % s != 0 && s != plain && s != fit) continue;
        const int groups = (K + s - 1) / s;
        const bool walk = (double)tiles * groups <= 12.0 * kSms;
        std::map<double, int64_t> free_at;   // when how many SMs are free
        free_at[0.0] = (int64_t)kSms;
        double sum = 0.0, longest = 0.0, end = 0.0;
        for (int g = 0; g < groups; ++g) {
            const int q0 = g * s, q1 = std::min(K, q0 + s);
            const double c = kStart + (q1 - q0) * per_job + (double)(off[q1] - off[q0]) * per_member;
            sum += c;
            longest = std::max(longest, c);
            for (int64_t left = walk ? tiles : 0; left > 0;) {
                const auto first = free_at.begin();
                const int64_t n = std::min(left, first->second);
                const double done = first->first + c;
                if ((first->second -= n) == 0) free_at.erase(first);
                free_at[done] += n;
                end = std::max(end, done);
                left -= n;
            }
        }
        if (!walk) end = sum * (double)tiles / kSms + 0.5 * longest;
        if (least < 0.0 || end < least) {
            least = end;
            best = s;
        }
        if (s == plain) plain_end = end;
    }
    return plain_end >= 0.0 && least > 0.95 * plain_end ? plain : best;
}

}  // namespace umma
}  // namespace lds
