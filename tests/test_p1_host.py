"""Phase-1 host logic, compiled from the library's own headers with the host
compiler (no CUDA): the launch shape, the
digits' rounding, the drain after an abort."""
from __future__ import annotations

import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def run_cpp(tmp_path, body: str, *flags: str) -> str:
    """Compile `body` against summit_b200/csrc and run it."""
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(body)
    subprocess.run(["g++", "-std=c++17", "-O1", *flags, "-I", str(ROOT / "summit_b200" / "csrc"),
                    str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout


SHAPE = """
#include <cstdio>
#include <vector>
#include "lds_p1_shape.h"
int main() {
    const int K = %d, W = %d, members = %d;
    std::vector<int64_t> off{0};
    for (int q = 0; q < K * W; ++q) off.push_back(off.back() + members);
    std::printf("%%d", lds::umma::choose_sb_per_cta(off.data(), K * W, %d, %d, K, %d));
}
"""


# Windowed plans took 8 super-bins per CTA before the choice: a number of bins
# with no divisor near 8 is not left with 1, whose CTAs are mostly start-up.
@pytest.mark.parametrize("K", [67, 97, 134])
@pytest.mark.parametrize("W,tiles", [(20, 40), (700, 391)])
def test_bins_with_few_divisors_share_a_cta(tmp_path, K, W, tiles):
    assert int(run_cpp(tmp_path, SHAPE % (K, W, 128, 208, tiles, 8))) >= 8


# The super-bins' CTAs lie along grid.y, which holds 65,535: 97 bins x 700 windows
# at one per CTA would not fit, nor 24 x 3,000 (or x 200,000) at few per CTA.
@pytest.mark.parametrize("K,W", [(97, 700), (24, 3000), (1, 70000), (24, 200000)])
def test_the_grid_holds_the_ctas(tmp_path, K, W):
    s = int(run_cpp(tmp_path, SHAPE % (K, W, 64, 48, 2, 8)))
    assert 1 <= s <= 256 and -(-K * W // s) <= 65535


# 8 windows x 23 bins over 40 sample tiles, and one window of 13 over 79: whole windows
# are estimated up to 2.6 % earlier than 8 per CTA, within the estimate's own error.
@pytest.mark.parametrize("K,W,members,ncolp,tiles", [(23, 8, 128, 80, 40), (13, 1, 192, 48, 79)])
def test_a_near_tie_keeps_the_plain_number(tmp_path, K, W, members, ncolp, tiles):
    assert int(run_cpp(tmp_path, SHAPE % (K, W, members, ncolp, tiles, 8))) == 8


# A genome-wide plan (plain number 1) gains no candidate by that.
def test_genome_wide_numbers_are_divisors(tmp_path):
    assert int(run_cpp(tmp_path, SHAPE % (11, 1, 2048, 80, 79, 1))) in (1, 11)
    assert int(run_cpp(tmp_path, SHAPE % (24, 1, 4096, 208, 391, 1))) == 8


def test_even_parts_of_a_window(tmp_path):
    assert int(run_cpp(tmp_path, SHAPE % (24, 60, 128, 208, 391, 8))) in (8, 12, 24, 48)


DIGITS = """
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include "lds_digits.h"
using namespace lds::umma;
typedef long long ll;
static uint64_t state = 7;
static uint64_t rnd() {
    state ^= state << 13, state ^= state >> 7, state ^= state << 17;
    return state * 2685821657736338717ull;
}
static void check(int32_t t0, int32_t t1, int32_t t2, int32_t t3, int r) {
    const ll T = (((ll)t0 * 128 + t1) * 128 + t2) * 128 + t3;
    ll want = T >> r;                                    // to the nearest, ties to even
    const ll rest = T - want * (1ll << r), half = r ? 1ll << (r - 1) : 1;
    if (r && (rest > half || (rest == half && (want & 1)))) ++want;
    if (std::llabs(want) > 127ll << 21) return;          // (the columns' scale: top digit at most 127)
    const int32_t got = narrow_round(t0, t1, t2, t3, narrow_shift(r));
    if (got != want) { std::printf("%d %d %d %d >> %d: %d, not %lld", t0, t1, t2, t3, r, got, want); std::exit(0); }
    const uint32_t w = digits_word(got);
    const ll back = (((ll)(int8_t)(w >> 24) * 128 + (int8_t)(w >> 16)) * 128 + (int8_t)(w >> 8)) * 128 + (int8_t)w;
    if (back != got) { std::printf("digits of %d: %lld", got, back); std::exit(0); }
}
int main() {
    const int32_t big = 85952 * 3 * 64;                  // digit products of the longest narrow list
    for (int r = 0; r <= 14; ++r)
        for (int n = 0; n < 200000; ++n) {
            // a result R and low digits in range, and the high digits that go with them
            const int32_t t2 = n % 3 ? (int32_t)(rnd() % (2u * big + 1)) - big : (n % 2 ? big : -big);
            const int32_t t3 = n % 5 ? (int32_t)(rnd() % (2u * big + 1)) - big : (n % 2 ? big : -big);
            const ll R = (ll)(rnd() % (1u << 29)) - (1 << 28);
            const ll H = (R * (1ll << r) - ((ll)t2 * 128 + t3)) >> 14;
            const int32_t t1 = (int32_t)(rnd() % 257) - 128;
            check((int32_t)((H - t1) >> 7), (int32_t)(H - ((H - t1) >> 7) * 128), t2, t3, r);
        }
    digits_word(INT32_MAX), digits_word(INT32_MIN);      // (columns that are not finite)
    std::printf("ok");
}
"""


# The 32-bit rounding of the digit sums against 64-bit arithmetic, over low parts
# up to the longest list's, where its terms wrap; no step of it may be undefined.
def test_narrow_rounding(tmp_path):
    assert run_cpp(tmp_path, DIGITS, "-fsanitize=undefined",
                   "-fno-sanitize-recover=all") == "ok"


DRAIN = """
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "lds_p1_drain.h"
int main() {
    srand(5);
    const int sets = 4, warps = 2;
    for (int n = 0; n < 20000; ++n) {
        // Steps [0, used) consumed, [0, issued) issued by the producer, each decoder
        // warp stopped somewhere in the steps whose stages were free.
        const int nst = 4 + rand() % 5, used = rand() % 40, issued = used + rand() % (nst + 1);
        std::vector<int> next(sets * warps);
        for (int w = 0; w < sets * warps; ++w) next[w] = used + rand() % (nst + 1);
        // arrivals per step: the producer's and the warps'; steps share nst barriers
        std::vector<int> got(issued + 2 * nst, 0);
        for (int j = 0; j < issued + nst; ++j) {
            if (j < issued) ++got[j];
            for (int u = 0; u < warps; ++u)
                if (next[(j % sets) * warps + u] > j) ++got[j];
        }
        lds::umma::p1_settle(issued, nst, sets, warps, [&](int w) { return next[w]; }, [&](int s) {
            int j = issued - 1;              // the stage's step that is under way
            while (j % nst != s) --j;
            ++got[j];
        });
        for (int j = issued > nst ? issued - nst : 0; j < issued; ++j) {
            if (got[j] != warps + 1) { std::printf("step %d of %d: %d arrivals", j, issued, got[j]); return 0; }
        }
    }
    std::printf("ok");
}
"""


# After an abort every stage that holds a copy in flight gets the arrivals its
# barrier still needs, and no more, wherever the decoders stopped.
def test_drain_completes_every_stage(tmp_path):
    assert run_cpp(tmp_path, DRAIN) == "ok"
