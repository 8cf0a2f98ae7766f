"""Paths a call takes by its sizes give the same results: EMT atoms in any order (staged by
species) and from one atom up, wide CTAs of small batches, ring polymers shared by the CTAs of a
cluster, HDNNP force calls spread over several CTAs, and the fixed-cell G3 walk.

Tolerances: the paths differ in the order of FP64 sums only, so forces of one path stay within
1e-11 of the other's largest force; against the oracle the parity bars hold (1e-10 eV/A, scaled by
the largest force where it exceeds 1 eV/A)."""
import numpy as np
import pytest

from md_tian2_gb300 import constants as C
from md_tian2_gb300 import nene
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import PES_NENE, Engine, SimParams
from md_tian2_gb300.universe import Universe

from .helpers import make_engine, oracle_list

pytestmark = pytest.mark.gpu


def _close(a, b, tol=1e-11):
    a, b = np.asarray(a), np.asarray(b)
    assert np.isfinite(b).all()
    assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max()), np.abs(a - b).max()


def _permuted(u, order):
    pick = lambda a: np.ascontiguousarray(a[order])  # noqa: E731
    return Universe(pick(u.r), pick(u.v), pick(u.m), pick(u.idx), pick(u.is_fixed), u.simbox, u.names, u.is_proj, u.algo)


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("natoms", [1, 2, 3, 5, 33, 36, 37])
def test_emt_atom_order_and_size(built_lib, oracle_lib, natoms, precision):
    rng = np.random.default_rng(natoms)
    full = W.h_on_metal(rng, "Au", 3, 1.0, 20.0, 30.0, 300.0, z0=1.3)
    full.r[1:] += rng.normal(scale=0.05, size=full.r[1:].shape)
    u = _permuted(full, np.arange(natoms))
    order = rng.permutation(natoms)
    shifted = _permuted(u, order)
    shifted.r = shifted.r + (rng.integers(-2, 3, size=(natoms, 1, 3)) @ u.simbox.T)  # other images of the atoms
    emt = W.emt_params()
    eng = make_engine([u, shifted], emt)
    eng.calc_force(SimParams(), precision=precision)
    out = eng.download()
    f = [eng.split(out["f"], t)[:, 0] for t in (0, 1)]
    d = [eng.split(out["dens"], t, 1)[:, 0] for t in (0, 1)]
    eng.close()
    # FP32 forces: pair terms up to a few eV/A rounded to 24 bits and summed over 36 partners
    tol = 1e-10 if precision == "fp64" else 2e-4
    _close(f[1], f[0][order], tol)
    _close(d[1], d[0][order], tol)
    _close(out["epot"][1], out["epot"][0], tol)
    if precision == "fp64":
        o = oracle_list([u], emt)[0]
        o.calc_force(SimParams())
        _close(f[0], o.f[:, 0], 1e-10)
        _close(out["epot"][0], o.epot[0], 1e-10)


@pytest.mark.parametrize("nbeads,many", [(1, 400), (4, 1500), (6, 300), (32, 40)])
def test_emt_batch_size(built_lib, nbeads, many):
    """One trajectory alone and among copies of itself: 256 against 128 threads (single beads), a
    cluster of CTAs against one or two CTAs (ring polymers)."""
    rng = np.random.default_rng(nbeads)
    pile = C.PROP_ID_PILE if nbeads > 1 else C.PROP_ID_VERLET
    u = W.h_on_metal(rng, "Pt", 3, 0.5, 0.0, 0.0, 300.0, pile, pile, z0=1.4, nbeads=nbeads)
    u.r += rng.normal(scale=0.02, size=u.r.shape)
    emt = W.emt_params("H", "Pt")
    sp = SimParams(step=0.1, seed=9)
    got = []
    for n in (1, many):
        eng = make_engine([u] * n, emt)
        eng.calc_force(sp)
        eng.md_steps(2, sp)
        out = eng.download()
        got.append({k: eng.split(out[k], 0) for k in ("r", "v", "f")})  # (deviates depend on the trajectory: 0 is alike)
        eng.close()
    for k in ("r", "v", "f"):
        _close(got[1][k], got[0][k], 1e-10)


def _graphene_model(zetas):
    m = nene.random_model(["H", "C"], hidden=(9, 7), act="t", seed=4, neighbours=["C"])
    for e in range(2):
        for sf in m.sfs[e]:
            if sf.type == 3:
                sf.zeta = zetas[(1.0, 4.0, 16.0).index(sf.zeta)]
        m.sfs[e] = nene.sort_symfunctions(m.sfs[e])
    return m


@pytest.mark.parametrize("k", [3, 5])
@pytest.mark.parametrize("zetas", [(1.0, 4.0, 16.0), (1.0, 2.0, 4.0), (1.0, 3.0, 5.0)])
def test_hdnnp_split_and_cells(built_lib, oracle_lib, k, zetas):
    """FP64 force call of two trajectories (their atoms spread over CTAs) against the oracle and
    against the same two in a batch that is not split; zeta 1, 4, 16 takes the fixed-cell walk,
    the other sets the general one."""
    from oracle.oracle import NNOracle
    rng = np.random.default_rng(k)
    us = [W.h_on_graphene(rng, 1.0, z0=z, k=k) for z in (1.4, 2.6)]
    m = _graphene_model(zetas)
    got = []
    for n in (1, 350):
        eng = Engine(0)
        eng.define(us * n)
        eng.read_nene(m, ["H", "C"], max_neighbors=96)
        eng.set_pes(PES_NENE, 0.0)
        eng.upload()
        eng.calc_force(SimParams())
        out = eng.download()
        got.append([(eng.split(out["f"], t)[:, 0], out["epot"][t], eng.split(out["a"], t)[:, 0]) for t in (0, 1)])
        eng.close()
    orc = NNOracle(m)
    for t, u in enumerate(us):
        E, F = orc.energy_force(np.array([0] + [1] * (u.natoms - 1)), u.r[:, 0], u.simbox)
        _close(got[0][t][0], F, 1e-10)
        _close(got[0][t][1], E, 1e-10)
        _close(got[0][t][2], F / u.m[:, None], 1e-10)
        for a, b in zip(got[0][t], got[1][t]):
            _close(a, b)
