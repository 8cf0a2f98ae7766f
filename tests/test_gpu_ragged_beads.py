"""Ring polymers of very different atom counts in one batch: the shared memory is laid out for the
largest, the beads evaluated together are counted by each trajectory.  Every trajectory gives what
it gives alone, and the oracle's results.

Tolerances: FP64, a trajectory alone and in the batch differ in the order of sums (1e-11 of the
largest force) and the oracle's parity bar is 1e-10; FP32 pair terms of a few eV/A rounded to 24 bits and
summed over up to 80 partners, 2e-4 of the largest force."""
import numpy as np
import pytest

from md_tian2_gb300 import constants as C
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import SimParams

from .helpers import make_engine, oracle_list

pytestmark = pytest.mark.gpu

KEYS = ("r", "v", "f", "dens", "epot")


def _run(us, emt, sp, precision):
    eng = make_engine(us, emt)
    got = []
    eng.calc_force(sp, precision=precision)
    for steps in (0, 2):
        if steps:
            eng.md_steps(steps, sp, precision=precision)
        out = eng.download()
        per = [{k: eng.split(out[k], t, 1 if k == "dens" else 3).copy() for k in ("r", "v", "f", "dens")}
               for t in range(len(us))]
        for t, p in enumerate(per):
            p["epot"] = out["epot"][eng.bead_off[t]:eng.bead_off[t + 1]].copy()
        got.append(per)
    eng.close()
    return got


def _close(a, b, tol, what):
    assert np.isfinite(b).all(), what
    assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max()), (what, np.abs(a - b).max())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("k,nb,small", [(9, 16, (16, 7, 16)), (12, 2, (2, 4, 6, 1)), (8, 4, (4, 1, 3)), (9, 1, (8, 2))])
def test_ragged_ring_polymers(built_lib, oracle_lib, k, nb, small, precision):
    rng = np.random.default_rng(100 * k + nb)
    us = []
    for kk, b in [(k, nb)] + [(3, b) for b in small]:
        u = W.h_on_metal(rng, "Pt", kk, 0.5, 0.0, 0.0, 300.0, C.PROP_ID_VERLET, C.PROP_ID_VERLET, z0=1.5, nbeads=b)
        u.r += rng.normal(scale=0.03, size=u.r.shape) * ~u.is_fixed
        us.append(u)
    emt = W.emt_params("H", "Pt")
    sp = SimParams(step=0.1)
    got = _run(us, emt, sp, precision)
    tol = 1e-11 if precision == "fp64" else 2e-4
    for t, u in enumerate(us):
        alone = _run([u], emt, sp, precision)
        for s in (0, 1):
            for key in KEYS:
                _close(got[s][t][key], alone[s][0][key], tol, (s, t, key))
    if precision == "fp64":
        for t, o in enumerate(oracle_list(us, emt)):
            o.calc_force(sp)
            for s in (0, 1):
                for _ in range(2 * s):
                    o.propagate_1(sp)
                    o.calc_force(sp)
                    o.propagate_2(sp)
                for key in KEYS:
                    ref = np.asarray(getattr(o, key)).reshape(got[s][t][key].shape)
                    _close(got[s][t][key], ref, 1e-10, (s, t, key))
