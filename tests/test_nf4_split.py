"""The rule that shares an NF4 matrix out over CTAs, compiled for the host."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "rew_b200", "csrc")

MAIN = """
#include <stdio.h>
#include "nf4_split.cuh"
int main() {
  long sms, K, N, most;
  while (scanf("%ld %ld %ld %ld", &sms, &K, &N, &most) == 4) {
    const rewb::Nf4Split s = rewb::nf4_split((int)sms, K, N, most);
    printf("%d %d %d\\n", s.slabs, s.span, rewb::nf4_tile_split((int)sms, K, N));
  }
}
"""


@pytest.fixture(scope="module")
def split(tmp_path_factory):
    d = tmp_path_factory.mktemp("split")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "main")], check=True)

    def run(cases):
        out = subprocess.run([str(d / "main")], input="".join("%d %d %d %d\n" % c for c in cases), capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]
    return run


def test_shares_that_do_not_fit_give_way_to_whole_tiles(split):
    """2048 x 9728 on 148 SMs is shared out in five slabs; with room for four of them it is cut as if there were no shares (three CTAs a
    tile, one wave), not into four (304 CTAs for 296 slots)."""
    assert split([(148, 2048, 9728, m) for m in (16, 5, 4, 3, 2, 1)]) == [(5, 9, 3), (5, 9, 3), (3, 0, 3), (3, 0, 3), (2, 0, 3), (1, 0, 3)]
    assert split([(148, 4096, 28672, 16)]) == [(3, 49, 1)]


@pytest.mark.parametrize("sms", [148, 132])
def test_every_tile_gets_as_many_slabs_as_there_are_at_most(split, sms):
    """Whatever the sizes: no more slabs than there is room for, the same answer when asked again with just that room (what the launch
    does), no tile shared by more CTAs than there are slabs, and no CTA in more than two tiles."""
    cases = [(sms, 64 * kb, 64 * g, m) for kb in (1, 3, 8, 24, 32, 64, 76, 224) for g in (1, 2, 3, 24, 75, 150, 151, 155, 300, 448, 1000) for m in (16, 5, 4, 2, 1)]
    got = split(cases)
    assert split([(s, k, n, max(1, slabs)) for (s, k, n, _), (slabs, _, _) in zip(cases, got)]) == got
    shared = 0
    for (s, k, n, most), (slabs, span, whole) in zip(cases, got):
        KB, tiles = k // 64, (n + 127) // 128
        assert 1 <= slabs <= max(1, min(most, 16))
        if not span:
            assert slabs == max(1, min(whole, most))
            continue
        shared += 1
        assert span <= KB
        for t in range(tiles):
            assert ((t + 1) * KB - 1) // span - t * KB // span + 1 <= slabs
    assert shared > 3
