"""Two atoms on one site under the generic HDNNP kernels: the pair counts in the descriptors with
r = 0 (their limit for r -> 0), the forces between the two are no finite numbers (they divide by r), and the
fused steps retire that trajectory while the others go on."""
import numpy as np
import pytest

from md_tian2_gb300 import nene
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import PES_NENE, Engine, SimParams

pytestmark = pytest.mark.gpu

ERR_NONFINITE = -11


def _engine(us, descriptor):
    m = nene.random_model(["H", "C"], hidden=(9, 7), act="t", seed=4, descriptor=descriptor,
                          neighbours=["C"] if descriptor == "acsf" else ["H", "C"])
    eng = Engine(0)
    eng.define(us)
    eng.read_nene(m, ["H", "C"], max_neighbors=96)
    eng.set_pes(PES_NENE, 0.0)
    eng.nn_fast_path(False)
    eng.upload()
    return eng


def _pair(apart):
    rng = np.random.default_rng(3)
    us = [W.h_on_graphene(rng, 1.0, z0=2.0, k=3) for _ in range(2)]
    us[0].r[0] = us[0].r[6] + [0.0, 0.0, apart]
    return us


@pytest.mark.parametrize("descriptor", ["radial", "acsf"])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_two_atoms_on_one_site(built_lib, descriptor, precision):
    got = []
    for apart in (0.0, 1e-7):
        eng = _engine(_pair(apart), descriptor)
        eng.calc_force(SimParams(), precision=precision)
        out = eng.download()
        got.append((out["epot"].copy(), eng.split(out["f"], 0)[:, 0], eng.split(out["f"], 1)[:, 0]))
        if apart == 0.0:
            eng.md_steps(3, SimParams(), precision=precision)
            q = eng.query(SimParams())
            assert q["status"][0] == ERR_NONFINITE and q["steps_done"][0] == 1
            assert q["status"][1] == 0 and q["steps_done"][1] == 3
        eng.close()
    f = got[0][1]
    assert not np.isfinite(f[0]).all() and not np.isfinite(f[6]).all()
    assert np.isfinite(got[0][2]).all()
    if descriptor == "radial":
        # smooth in r: 1e-7 A apart changes the energy by the slope times 1e-7, far below 1e-5 eV
        assert np.isfinite(got[0][0]).all()
        assert np.abs(got[0][0] - got[1][0]).max() < (1e-5 if precision == "fp64" else 1e-3)
