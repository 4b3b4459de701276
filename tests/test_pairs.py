"""The numbering of a warp's (rectangle, tile) pairs at its largest sizes,
compiled for the host from the kernels' own header."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "jaxrenderer_gb300" / "csrc"
MAIN = """
#include <cstdio>
#include "rast_pairs.cuh"
int main() {
  unsigned n[32], before[32], rounds, base;
  for (unsigned s = 0, k = 0; k < 32; ++k) {
    if (std::scanf("%u", n + k) != 1) return 1;
    before[k] = s;
    s += n[k];
  }
  if (std::scanf("%u", &rounds) != 1) return 1;
  while (rounds--) {
    if (std::scanf("%u", &base) != 1) return 1;
    unsigned begun = 0;
    for (int k = 0; k < 32; ++k) begun |= rast::pair_begin_bit(before[k], n[k], base);
    std::printf("%u\\n", begun);
  }
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("pairs")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-I", str(CSRC), str(d / "main.cpp"), "-o", str(d / "pairs")], check=True)
    return d / "pairs"


@pytest.mark.parametrize("counts", [
    [1] * 32, [0] * 31 + [5], [33] + [0] * 30 + [1], [1 << 26] * 32,          # 2^31 pairs
    [0, 1 << 26] * 16, [1 << 26] * 25 + [0] * 7, [(1 << 26) - 1, 0, 7, 32] * 8])  # lanes without pairs past 2^30
def test_every_round_has_the_pairs_that_begin_in_it(program, counts):
    before = np.concatenate([[0], np.cumsum(counts, dtype=np.int64)])
    total = int(before[-1])
    near = {int(b) // 32 * 32 + d for b in [*before, 1 << 30, (1 << 30) + (1 << 29)] for d in (-32, 0, 32)}
    bases = sorted(b for b in near if 0 <= b < total)
    out = subprocess.run([str(program)], input=" ".join(map(str, [*counts, len(bases), *bases])), text=True, capture_output=True, check=True)
    for base, got in zip(bases, map(int, out.stdout.split()), strict=True):
        want = 0
        for b, n in zip(before, counts):
            if n and base <= b < base + 32:
                want |= 1 << int(b - base)
        assert got == want, base
