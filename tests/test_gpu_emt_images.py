"""Minimum images of the EMT pair loops against the oracle: with the table of image shifts (512 atoms
and less) and without it, atoms moved to images up to two cells away, and frozen layers exactly on
their lattice sites (pairs half a cell apart, whose image the oracle's rounding decides).

Tolerances: 1e-10 of the largest force in FP64; FP32 pair terms of a few eV/A rounded to 24 bits and summed
over up to 80 partners, 2e-4."""
import numpy as np
import pytest

from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import SimParams
from md_tian2_gb300.universe import Universe

from .helpers import make_engine, oracle_list

pytestmark = pytest.mark.gpu


def _check(u, precision):
    emt = W.emt_params()
    eng = make_engine([u], emt)
    eng.calc_force(SimParams(), precision=precision)
    out = eng.download()
    eng.close()
    o = oracle_list([u], emt)[0]
    o.calc_force(SimParams())
    tol = 1e-10 if precision == "fp64" else 2e-4
    for got, ref in ((out["f"], o.f.reshape(-1)), (out["epot"], o.epot), (out["dens"], o.dens.reshape(-1))):
        assert np.isfinite(got).all()
        assert np.abs(got - ref).max() <= tol * max(1.0, np.abs(ref).max())


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("natoms", [511, 512, 513, 577])
def test_images_around_the_table_limit(built_lib, oracle_lib, natoms, precision):
    rng = np.random.default_rng(natoms)
    u = W.h_on_metal(rng, "Au", 12, 1.0, 0.0, 0.0, 300.0, z0=1.5)
    u = Universe(u.r[:natoms].copy(), u.v[:natoms].copy(), u.m[:natoms], u.idx[:natoms], u.is_fixed[:natoms], u.simbox, u.names,
                 u.is_proj, u.algo)
    u.r += rng.normal(scale=0.05, size=u.r.shape)
    u.r += rng.integers(-2, 3, size=(natoms, 1, 3)) @ u.simbox.T
    _check(u, precision)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("k", [2, 4, 5, 6])
def test_pairs_half_a_cell_apart(built_lib, oracle_lib, k, precision):
    rng = np.random.default_rng(k)
    u = W.h_on_metal(rng, "Au", k, 1.0, 0.0, 0.0, 300.0, z0=1.4)
    u.r += rng.normal(scale=0.05, size=u.r.shape) * ~u.is_fixed
    _check(u, precision)
