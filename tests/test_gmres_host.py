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


@pytest.fixture(scope="module")
def pairs(tmp_path_factory):
    """argv: the systems' operators as 'offset,n,lda'; or 'time', their number and how
    many of them share one operator: prints milliseconds."""
    return compiled(tmp_path_factory.mktemp("pairs"), """
    const bool time = argc > 1 && argv[1][0] == 't';
    std::vector<GmSys> sys((size_t)(time ? atoi(argv[2]) : argc - 1));
    for (size_t s = 0; s < sys.size(); ++s) {
        long long off = 0, n = 100, ld = 128;
        if (time) off = (long long)(s / (size_t)atoi(argv[3])) * 12800;
        else sscanf(argv[s + 1], "%lld,%lld,%lld", &off, &n, &ld);
        sys[s].a_off = (size_t)off;
        sys[s].n = n;
        sys[s].lda = ld;
    }
    const auto t0 = std::chrono::steady_clock::now();
    const int any = gm_pair_systems(sys);
    const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    if (time) return 0 * printf("%f", ms);
    printf("%d", any);
    for (const GmSys& d : sys) printf(" %d", d.mate);""")


def reference_pairs(systems):
    """The first later system with the same operator that has no mate yet."""
    mate = [-1] * len(systems)
    for s in range(len(systems)):
        for o in range(s + 1, len(systems)):
            if mate[s] < 0 and mate[o] < 0 and systems[s] == systems[o]:
                mate[s], mate[o] = o, s
    return mate


@pytest.mark.parametrize("seed", range(12))
def test_pairs_of_systems_that_share_an_operator(pairs, seed):
    import random
    rng = random.Random(seed)
    systems = [(rng.randrange(1 + seed) * 640, 100 + rng.randrange(2), 128) for _ in range(rng.randrange(1, 40))]
    mate = reference_pairs(systems)
    assert pairs(*["%d,%d,%d" % s for s in systems]) == [str(v) for v in [int(max(mate) >= 0)] + mate]


@pytest.mark.parametrize("share", [1, 3, 20000])
def test_pairing_of_many_systems_is_not_quadratic(pairs, share):
    """20000 systems: every one against every other takes 200 million comparisons, a
    third of a second."""
    assert min(float(pairs("time", 20000, share)[0]) for _ in range(3)) < 60
