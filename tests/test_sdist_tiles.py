"""The tiles of the distance sums (tfm_gb300/csrc/sdist.h) on the host: every
pair of a chain in one tile, and positions inside the chain at lengths whose
tile numbers do not fit 32 bits."""
import os
import random
import shutil
import subprocess

import pytest

HEADER = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tfm_gb300",
                      "csrc", "sdist.h")
PROGRAM = """
#include <cstdio>
#include "%s"
int main() {
  int len;
  long long k;
  while (std::scanf("%%d %%lld", &len, &k) == 2) {
    int s0, p0;
    ccpgpu::sdist_tile(k, len / 2, s0, p0);
    std::printf("%%lld %%d %%d\\n", ccpgpu::sdist_tiles(len, len / 2), s0, p0);
  }
}
"""


@pytest.fixture(scope="module")
def tiles(tmp_path_factory):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    d = tmp_path_factory.mktemp("sdist")
    src, exe = str(d / "tiles.cpp"), str(d / "tiles")
    with open(src, "w") as f:
        f.write(PROGRAM % HEADER)
    subprocess.check_call([cxx, "-O1", "-Wall", "-Werror", "-o", exe, src])

    def ask(rows):
        out = subprocess.run([exe], input="".join("%d %d\n" % r for r in rows), text=True,
                             capture_output=True, check=True).stdout
        return [tuple(int(v) for v in ln.split()) for ln in out.splitlines()]

    return ask


@pytest.mark.parametrize("n", [2, 255, 256, 257, 511, 1026, 2051])
def test_every_pair_has_one_tile(tiles, n):
    total = -(-(n // 2) // 128) * -(-n // 256)
    got = tiles([(n, k) for k in range(total)])
    assert {g[0] for g in got} == {total}
    assert sorted(g[1:] for g in got) == sorted(
        (s + 1, p) for s in range(0, n // 2, 128) for p in range(0, n, 256))


# 11.8 million beads fill 31 bits of tile numbers, 11.9 million pass them; the
# longest chain that the limits allow has 2^28 - 1 beads
@pytest.mark.parametrize("n", [11_800_000, 11_900_000, 16_777_217, 200_000_000, (1 << 28) - 1])
def test_long_chains(tiles, n):
    nsep, nrow = -(-(n // 2) // 128), -(-n // 256)
    total = nsep * nrow
    rng = random.Random(n)
    ks = [0, nsep - 1, nsep, total - 1] + [k for k in (2 ** 31 - 1, 2 ** 31, 2 ** 32 + 5) if k < total]
    ks += [rng.randrange(total) for _ in range(200)]
    for k, (tot, s0, p0) in zip(ks, tiles([(n, k) for k in ks])):
        assert tot == total
        assert (s0, p0) == (k % nsep * 128 + 1, k // nsep * 256)
        assert 1 <= s0 <= n // 2 and 0 <= p0 < n
