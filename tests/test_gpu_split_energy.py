"""HDNNP force calls of small batches, whose trajectories are spread over several CTAs: an energy has
the same bits in every call (the CTAs' shares are added in order), every kernel is counted, and forces
differ by the order of FP32 sums at most (2^-24, about 100 terms up to 10 times the result: 1e-4)."""
import numpy as np
import pytest

from md_tian2_gb300 import nene
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import PES_NENE, Engine, SimParams

pytestmark = pytest.mark.gpu


# kernels of one call: forces, and around a split call two more; the tensor-core form runs
# descriptors, network and forces
@pytest.mark.parametrize("precision,kernels", [("fp64", 1), ("fp32", 1), ("bf16x3", 3)])
def test_energy_bits_and_launches(built_lib, precision, kernels):
    rng = np.random.default_rng(8)
    us = [W.h_on_graphene(rng, 1.0, z0=z, k=6) for z in (1.4, 2.6, 1.8)]
    m = nene.random_model(["H", "C"], hidden=(25, 25), act="t", seed=4, neighbours=["C"])
    eng = Engine(0)
    eng.define(us)
    eng.read_nene(m, ["H", "C"], max_neighbors=96)
    eng.set_pes(PES_NENE, 0.0)
    eng.nn_fast_path(False)
    eng.upload()
    eng.calc_force(SimParams(), precision=precision)  # lists and scratch
    first = None
    for _ in range(30):
        n = eng.launch_count()
        eng.calc_force(SimParams(), precision=precision)
        assert eng.launch_count() - n == kernels + 2
        out = eng.download()
        if first is None:
            first = out
        assert np.array_equal(out["epot"], first["epot"])
        assert np.abs(out["f"] - first["f"]).max() <= 1e-4 * np.abs(first["f"]).max()
        assert np.allclose(out["a"].reshape(-1, 3), out["f"].reshape(-1, 3) / np.concatenate([u.m for u in us])[:, None],
                           rtol=1e-14, atol=0.0)
    eng.close()
