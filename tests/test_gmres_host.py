"""Host-side parts of GMRES (csrc/gmres.cuh), compiled on their own: no GPU."""
import os
import subprocess

import pytest

from cc_abstemious_gb300 import build


def compiled(folder, body):
    """A program whose main() is `body`, after gmres.cuh."""
    src, out = os.path.join(str(folder), "t.cu"), os.path.join(str(folder), "t")
    with open(src, "w") as f:
        f.write('#include <chrono>\n#include <cstdlib>\n#include "gmres.cuh"\nusing namespace bem;\n'
                "int main(int argc, char** argv) {\n%s\nreturn 0;\n}\n" % body)
    r = subprocess.run([build.NVCC] + build.ARCH + ["-O2", "-std=c++17", "-I", build.CSRC, src, "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return lambda *args: subprocess.run([out] + [str(a) for a in args], capture_output=True, text=True,
                                        check=True).stdout.split()


@pytest.fixture(scope="module")
def reported(tmp_path_factory):
    return compiled(tmp_path_factory.mktemp("states"), """
    std::vector<GmState> st((size_t)argc - 1);
    for (int s = 1; s < argc; ++s) {
        GmState& t = st[(size_t)s - 1];
        t = GmState{};
        t.done = 1;
        if (argv[s][0] == 'c') t.converged = 1;
        if (argv[s][0] == 'w') t.gave_up = 1;
    }
    try {
        gm_require_waits(st.data(), st.size());
        printf("0");
    } catch (const Error& e) {
        printf("%d", (int)e.status);
    }""")


@pytest.mark.parametrize("states,status", [("c", 0), ("n", 0), ("w", 7), ("ccn", 0), ("ccw", 7), ("wcc", 7)])
def test_a_wait_that_ran_out_is_not_reported_as_non_convergence(reported, states, status):
    """c: converged, n: out of iterations, w: a kernel's wait gave up (BEM_ERR_TIMEOUT = 7)."""
    assert reported(*states) == [str(status)]
