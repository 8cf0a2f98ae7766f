"""How many CTAs share a trajectory of a ring-polymer batch (team_log2), from the batch's bead and atom
counts: compiled for the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "md_tian2_gb300" / "csrc"

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <vector>
#include "mdt_emt.cuh"
using namespace mdt;
int main(int argc, char **argv) {  // slots, then natoms nbeads count ...
    TeamWork w{};
    long n = 0;
    int most = 1;
    for (int k = 2; k + 2 < argc; k += 3)
        for (int c = 0; c < atoi(argv[k + 2]); ++c, ++n) {
            w.add(atoi(argv[k]), atoi(argv[k + 1]));
            most = atoi(argv[k + 1]) > most ? atoi(argv[k + 1]) : most;
        }
    std::printf("%d\n", 1 << team_log2(w, n, most, atol(argv[1])));
    return 0;
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("team")
    (d / "team.cu").write_text(SOURCE)
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O1", "-std=c++17", "-I", str(CSRC),
                    str(d / "team.cu"), "-o", str(d / "team")], check=True, capture_output=True)

    def run(slots, *groups):
        args = [str(slots)] + [str(x) for g in groups for x in g]
        return int(subprocess.run([str(d / "team"), *args], check=True, capture_output=True, text=True).stdout)
    return run


@pytest.mark.parametrize("groups,parts", [
    ([(37, 2, 1)], 2),                                  # no more CTAs than beads
    ([(37, 32, 1)], 8),
    ([(37, 4, 24), (65, 6, 24), (65, 10, 24), (101, 16, 24)], 8),  # few: all SMs by teams
    ([(65, 4, 256), (65, 8, 256), (65, 16, 256), (65, 32, 256)], 2),  # many: four waves at most
    ([(37, 1, 1199), (37, 2, 1)], 1),                   # single beads would leave half the CTAs waiting
    ([(37, 1, 2000), (37, 8, 4)], 1),
    ([(37, 1, 300), (37, 32, 1)], 8),                   # one long ring polymer decides
    ([(37, 1, 4000), (37, 2, 4000)], 1),
])
def test_ctas_per_trajectory(rule, groups, parts):
    assert rule(608, *groups) == parts
