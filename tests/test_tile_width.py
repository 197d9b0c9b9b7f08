"""The rule for the FP8 GEMM's columns per tile, compiled on its own: it needs no GPU."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "dlblas_b200", "csrc")


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    """rule(lists of (most, likely or None, rows, experts, n, sms, may_be_64)): the widths; None = the likely number of tiles"""
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text("""
#include <cstdio>
#include "tile_width.h"
int main() {
  long long most, likely, rows, experts, n;
  int sms, may;
  while (std::scanf("%lld %lld %lld %lld %lld %d %d", &most, &likely, &rows, &experts, &n, &sms, &may) == 7) {
    if (likely < 0) likely = dlb::likely_tiles(rows, experts, most);
    std::printf("%d\\n", dlb::fp8_tile_width(most, likely, n, sms, may != 0));
  }
}
""")
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I", CSRC, str(d / "rule.cpp"), "-o", str(d / "rule")],
                   check=True)

    def ask(calls):
        text = "\n".join(" ".join(str(-1 if v is None else int(v)) for v in c) for c in calls)
        return [int(v) for v in subprocess.run([str(d / "rule")], input=text, capture_output=True, text=True, check=True)
                .stdout.split()]

    return ask


def test_dense(rule):
    """One wave of 64, else of 128, else 256."""
    calls, want = [], []
    for tiles in (1, 2, 7, 37, 74, 148, 149):
        for n in (8, 64, 72, 4736, 4744, 9472, 9480, 18944, 18952, 24576):
            for may in (0, 1):
                calls.append((tiles, tiles, 0, 0, n, 148, may))
                want.append(64 if may and tiles * -(-n // 64) <= 148 else 128 if tiles * -(-n // 128) <= 148 else 256)
    assert rule(calls) == want


def test_grouped_launches_by_the_likely_number_of_tiles(rule):
    """Rows, experts and columns, and the width that was the faster one when both were timed."""
    timed = [(400, 8, 2048, 128), (5142, 64, 256, 128), (4666, 39, 256, 128), (2575, 32, 512, 128),
             (956, 8, 2048, 256), (3828, 32, 512, 256), (9965, 39, 256, 256), (8199, 32, 256, 256), (144, 39, 768, 256),
             (24, 16, 2048, 256), (801, 16, 1536, 256), (2052, 8, 1024, 256),
             (2, 8, 4096, 128), (4, 8, 4096, 256), (4, 16, 1536, 128), (9, 16, 1536, 256), (9, 39, 640, 128)]
    assert rule([(rows // 128 + e, None, rows, e, n, 148, 1) for rows, e, n, _ in timed]) == [w for *_, w in timed]


def test_grouped_launches_are_within_the_bound(rule):
    """Where even the most tiles make a wave of 64 or 128 columns the likely number changes nothing, and a launch that could
    exceed a wave of 256 takes 256."""
    calls = [(rows // 128 + e, None, rows, e, n, sms, may) for rows in (1, 8, 100, 127, 128, 129, 1000, 5000, 40000)
             for e in (1, 8, 39, 256) for n in (128, 256, 384, 2048, 7168) for sms in (148, 100) for may in (0, 1)]
    for (most, _, _, _, n, sms, may), width in zip(calls, rule(calls)):
        one = [w for w in (64, 128) if (may or w > 64) and most * -(-n // w) <= sms]
        if one:
            assert width == one[0]
        else:
            assert width == 256 or (width == 128 and most * -(-n // 256) < sms)
