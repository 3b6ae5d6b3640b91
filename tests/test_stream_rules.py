"""Which blocks run which rows of a streaming launch, from the library's own host code (compiled against its internal header;
no GPU): every row group has one block, small independent jobs of a plan share the grid, the others have all of it."""
import subprocess
from pathlib import Path

import pytest

import magnitude_b200 as mb
from magnitude_b200 import _binding as B

ROOT = Path(__file__).resolve().parent.parent
WAITS, SUM_RANKS, SWIGLU = 1, 2, 4
GRID, SMEM = 148, 232448

# reads "M grid smem", then per job "type K flags segments rows..."; prints per job "cta0 ctas share rest section groups"
SOURCE = r"""
#include <cstdio>
#include <vector>
#include "kernels.h"
int main() {
    using namespace b200q;
    int M, grid, njobs;
    unsigned long smem;
    if (scanf("%d %d %lu %d", &M, &grid, &smem, &njobs) != 4) return 1;
    std::vector<StreamJob> jobs(njobs);
    for (StreamJob &J : jobs) {
        J = StreamJob{};
        if (scanf("%d %d %d %d", &J.qt, &J.K, &J.flags, &J.nseg) != 4) return 1;
        J.Kpad = (J.K + 255) / 256 * 256;
        for (int s = 0; s < J.nseg; ++s)
            if (scanf("%d", &J.seg[s].n) != 1) return 1;
        stream_job_finish(J, grid);
    }
    stream_fit_jobs(jobs.data(), njobs, M, grid, smem);
    for (const StreamJob &J : jobs) printf("%d %d %d %d %d %d\n", J.cta0, J.ctas, J.share, J.share_rest, J.section, J.total_groups);
}
"""


@pytest.fixture(scope="module")
def fit(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SOURCE)
    lib = Path(B.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", f"-I{ROOT}/magnitude_b200/csrc", "-I/usr/local/cuda/include", str(d / "rules.cpp"),
                    "-o", str(d / "rules"), str(lib), f"-Wl,-rpath,{lib.parent}", "-Wl,--allow-shlib-undefined"], check=True)

    def run(jobs, m=1, grid=GRID, smem=SMEM):
        text = f"{m} {grid} {smem} {len(jobs)}\n" + "\n".join(f"{qt} {k} {flags} {len(ns)} {' '.join(map(str, ns))}" for qt, k, flags, *ns in jobs)
        out = subprocess.run([str(d / "rules")], input=text, capture_output=True, text=True, check=True).stdout
        return [tuple(map(int, line.split())) for line in out.splitlines()]

    return run


def _covered(job, flags):
    """A job's row groups are shared out whole: gate/up pairs for SWIGLU, sections of at least one row quad."""
    cta0, ctas, share, rest, section, groups = job
    assert (2 if flags & SWIGLU else 1) * (ctas * share + rest) == groups
    assert 0 <= rest < ctas and cta0 >= 0 and cta0 + ctas <= GRID and section >= 1


@pytest.mark.parametrize("m", [1, 2, 4])
@pytest.mark.parametrize("n,k", [(1, 256), (4, 84992), (593, 5120), (2369, 4096), (152064, 5120)])
def test_a_call_has_the_whole_grid(fit, m, n, k):
    job, = fit([(mb.TYPE_Q4_K, k, 0, n)], m)
    assert job[:2] == (0, GRID)
    _covered(job, 0)


@pytest.mark.parametrize("m", [1, 2])
def test_small_independent_jobs_share_the_grid(fit, m):
    small, large = (mb.TYPE_Q4_K, 4096, 0, 1024), (mb.TYPE_Q4_K, 4096, 0, 14336)
    fits = fit([small] * 20, m)
    assert {j[:2] for j in fits} == {(37 * i, 37) for i in range(4)}          # quarters, five jobs each
    assert all(sum(j[0] == 37 * i for j in fits) == 5 for i in range(4))
    # the plan of test_gpu_stream.py, with and without its SWIGLU job
    shapes = ([(mb.TYPE_Q4_K, 1024, 0, 512), (mb.TYPE_Q4_K, 4096, 0, 1000), (mb.TYPE_Q6_K, 512, 0, 37), (mb.TYPE_Q8_0, 4096, 0, 4096),
               (mb.TYPE_Q4_K, 4096, 0, 14336)] * 5)[:23]
    for extra in ([], [(mb.TYPE_Q4_K, 1024, SWIGLU, 512, 512)]):
        mixed = fit(shapes + extra, m)
        assert all(j[1] == GRID for j in mixed[4::5] + mixed[23:])            # long shares, and pairs, stay whole
        assert sum(j[1] < GRID for j in mixed) >= 10
        for job, flags in zip(fits + mixed, [0] * 43 + [SWIGLU]):
            _covered(job, flags)


@pytest.mark.parametrize("flag", [WAITS, SUM_RANKS])
def test_jobs_that_meet_have_the_whole_grid(fit, flag):
    fits = fit([(mb.TYPE_Q4_K, 4096, 0, 1024)] * 10 + [(mb.TYPE_Q4_K, 4096, flag, 1024)] * 10)
    assert {j[:2] for j in fits} == {(0, GRID)}


def test_long_plans_are_dealt_launch_by_launch(fit):
    """64 jobs a launch: one that waits in the second launch does not concern the first."""
    fits = fit([(mb.TYPE_Q4_K, 4096, 0, 1024)] * 70 + [(mb.TYPE_Q4_K, 4096, WAITS, 1024)])
    assert all(j[1] < GRID for j in fits[:64]) and all(j[1] == GRID for j in fits[64:])
