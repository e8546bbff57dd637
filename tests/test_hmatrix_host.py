"""Host-side restatement of the recompression's order of singular values
(csrc/hmatrix.cuh), compiled on its own: no GPU."""
import math
import os
import subprocess

import pytest

from cc_abstemious_gb300 import build


@pytest.fixture(scope="module")
def places(tmp_path_factory):
    folder = str(tmp_path_factory.mktemp("order"))
    src, out = os.path.join(folder, "t.cu"), os.path.join(folder, "t")
    with open(src, "w") as f:
        f.write("""#include <cstdlib>
#include "hmatrix.cuh"
int main(int argc, char** argv) {
    std::vector<double> S;
    for (int i = 1; i < argc; ++i) S.push_back(strtod(argv[i], nullptr));
    for (int j = 0; j < (int)S.size(); ++j) printf("%d ", bem::descending_rank(S.data(), (int)S.size(), j));
    return 0;
}
""")
    r = subprocess.run([build.NVCC] + build.ARCH + ["-O2", "-std=c++17", "-I", build.CSRC, src, "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lambda S: [int(v) for v in subprocess.run([out] + [repr(v) for v in S], capture_output=True, text=True,
                                                     check=True).stdout.split()]


@pytest.mark.parametrize("S", [[1.0], [3.0, 2.0, 2.0, 1.0], [0.0, 0.0, 5e-324, 1e300, 2.0], [1e-17, 1.0, 1e-9, 1.0]])
def test_descending_and_stable(places, S):
    order = sorted(range(len(S)), key=lambda i: (-S[i], i))
    assert places(S) == [order.index(j) for j in range(len(S))]


@pytest.mark.parametrize("S", [[math.nan] * 5, [3.0, math.nan, 2.0, 0.0], [-math.nan, 1.0, math.nan],
                               [math.inf, math.nan, math.inf, 1.0], [0.0, -0.0, 0.0]])
def test_a_permutation_for_any_values(places, S):
    """Its places index the factors: with NaNs among them, counting comparisons gave the
    same place to several and none to others."""
    assert sorted(places(S)) == list(range(len(S)))
