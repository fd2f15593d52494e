"""The marched operator's reads of kappa stay inside its array without the padding: march_task's index
arithmetic (rg_march.cuh: a lane's first node, the stand-in past a run's end, NR + 1 lines, the layer above every
plane) is enumerated on the host for grids with ragged groups and long lines."""
import itertools
import shutil
import subprocess

import pytest

from conftest import PKG_DIR


def reads(dim, nn, NR):
    """Highest index that march_task loads from khat over all strips, lanes and planes."""
    NN0 = nn[0]
    NL = nn[1] if dim == 3 else 1
    M, NP = NN0 * NL, nn[2] if dim == 3 else nn[1]
    J = (NL + NR - 1) // NR * NN0
    lines = NR + 1 if dim == 3 else 1
    top = 0
    for j in {0, J - 1, J, J + 30} | {k for k in range(J + 31) if k % NN0 in (0, NN0 - 1)}:
        jj = min(max(j, 0), J - 1)
        group = jj // NN0
        c = group * NR * NN0 + (jj - group * NN0)
        ck = c if j < J else group * NR * NN0
        top = max(top, NP * M + ck + (lines - 1) * NN0)  # planes 0 .. NP (the layer above the last)
    return top


@pytest.mark.skipif(shutil.which("g++") is None, reason="no C++ compiler")
def test_reads_of_kappa_stay_inside_the_array(tmp_path):
    (tmp_path / "k.cpp").write_text('#include <cstdio>\n#include "rg_khat.cuh"\nint main() { long long n, a, b; while (scanf('
                                    '"%lld %lld %lld", &n, &a, &b) == 3) printf("%lld\\n", (long long)rg::khat_reach(n, a, b)); }')
    exe = tmp_path / "k"
    subprocess.run(["g++", "-std=c++17", "-I", PKG_DIR + "/csrc", "-o", str(exe), str(tmp_path / "k.cpp")], check=True)
    grids = [(3, g) for g in itertools.product((2, 3, 31, 300, 1500), (2, 3, 8), (2, 5))]
    grids += [(2, g + (1,)) for g in itertools.product((2, 30, 1500), (2, 7))]
    text = "".join("%d %d %d\n" % (g[0] * g[1] * g[2], g[0], g[1]) for _, g in grids)
    got = subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True).stdout.split()
    for (dim, g), size in zip(grids, got):
        for NR in (1, 2) if dim == 3 else (1,):
            assert reads(dim, g, NR) < int(size), (dim, g, NR)
