"""The three forms of the G3 walks by the structure of a function set: products of two lambdas and three or
four zetas, up to four etas, with functions missing and with one lambda; sets that are no such product, and one of three
lambdas, which takes the walk over a list.
FP64 energies and forces against the oracle (parity bar 1e-10, scaled by the largest force above
1 eV/A), and the training gradient, which takes the tangent walk, against central differences of the
oracle's loss (its second-order error and rounding: 1e-5)."""
import numpy as np
import pytest

from md_tian2_gb300 import constants as C
from md_tian2_gb300 import nene
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import PES_NENE, Engine, SimParams
from md_tian2_gb300.surrogate import Trainer

from .test_gpu_train import _oracle_loss, _tiny_dataset

pytestmark = pytest.mark.gpu

BOTH = (-1.0, 1.0)
# name: (etas in 1/A^2, (zeta, lambdas) ...)
SETS = {
    "3x3": ((0.001, 0.01, 0.1), ((1.0, BOTH), (2.0, BOTH), (4.0, BOTH))),
    "3x4": ((0.001, 0.01, 0.1), ((1.0, BOTH), (2.0, BOTH), (4.0, BOTH), (16.0, BOTH))),
    "4x3": ((0.001, 0.01, 0.05, 0.1), ((1.0, BOTH), (4.0, BOTH), (16.0, BOTH))),
    "2x4": ((0.01, 0.1), ((1.0, BOTH), (3.0, BOTH), (9.0, BOTH), (32.0, BOTH))),
    "4x1": ((0.001, 0.01, 0.05, 0.1), ((5.0, BOTH),)),
    "missing": ((0.001, 0.01, 0.1), ((1.0, (1.0,)), (4.0, BOTH), (16.0, (-1.0,)))),
    "one lambda": ((0.01, 0.1), ((1.0, (1.0,)), (2.0, (1.0,)), (8.0, (1.0,)))),
    "other lambda": ((0.01, 0.1), ((1.0, (0.5, 1.0)), (4.0, (0.5, 1.0)))),
    "3 lambdas": ((0.01, 0.1), ((1.0, (-1.0, 0.5, 1.0)), (4.0, (-1.0, 0.5, 1.0)))),
    "5 zetas": ((0.01, 0.1), ((1.0, (1.0,)), (2.0, BOTH), (3.0, (-1.0,)), (4.0, BOTH), (6.0, (1.0,)))),
    "7 zetas": ((0.001, 0.01, 0.1), tuple((float(z), (1.0,)) for z in (1, 2, 3, 5, 8, 16, 31))),
}


def _model(name, elements, neighbour, act="t", hidden=(7, 6)):
    etas, cells = SETS[name]
    rc = 6.5 * C.ANG2BOHR
    z = nene.Z_OF[neighbour]
    sfs = [nene.SymFunc(2, eta=float(e) / C.ANG2BOHR ** 2, rc=rc, e1=z) for e in (0.01, 0.1, 0.4)]
    sfs += [nene.SymFunc(3, eta=e / C.ANG2BOHR ** 2, lam=lam, zeta=zeta, rc=rc, e1=z, e2=z)
            for e in etas for zeta, lams in cells for lam in lams]
    m = nene.random_model(elements, hidden=hidden, act=act, seed=4, neighbours=[neighbour])
    m.sfs = [nene.sort_symfunctions(list(sfs)) for _ in m.elements]
    rng = np.random.default_rng(6)
    n = [len(sfs)] + list(hidden) + [1]
    m.nodes = [list(n) for _ in m.elements]
    m.weights = [np.concatenate([np.concatenate([rng.uniform(-0.6, 0.6, a * b), np.zeros(b)]) for a, b in zip(n, n[1:])])
                 for _ in m.elements]
    m.weights = [np.asarray(w, np.float32).astype(np.float64) for w in m.weights]
    m.smin, m.smax, m.savg = ([np.full(n[0], x) for _ in m.elements] for x in (0.0, 1.0, 0.0))
    return m


@pytest.mark.parametrize("name", SETS)
def test_forces_of_each_form(built_lib, oracle_lib, name):
    from oracle.oracle import NNOracle
    rng = np.random.default_rng(5)
    us = [W.h_on_graphene(rng, 1.0, z0=z, k=3) for z in (1.4, 2.6)]
    m = _model(name, ["H", "C"], "C")
    eng = Engine(0)
    eng.define(us)
    eng.read_nene(m, ["H", "C"], max_neighbors=96)
    eng.set_pes(PES_NENE, 0.0)
    eng.nn_fast_path(False)
    eng.upload()
    eng.calc_force(SimParams())
    out = eng.download()
    eng.calc_force(SimParams(), precision="fp32")
    out32 = eng.download()
    orc = NNOracle(m)
    for t, u in enumerate(us):
        E, F = orc.energy_force(np.array([0] + [1] * (u.natoms - 1)), u.r[:, 0], u.simbox)
        scale = max(1.0, np.abs(F).max())
        assert np.abs(eng.split(out["f"], t)[:, 0] - F).max() <= 1e-10 * scale
        assert abs(out["epot"][t] - E) <= 1e-10 * max(1.0, abs(E))
        # FP32: descriptors and forces to 24 bits through sums of a few thousand triplets
        assert np.abs(eng.split(out32["f"], t)[:, 0] - F).max() <= 2e-3 * scale
    eng.close()


@pytest.mark.parametrize("name", ["3x3", "3x4", "4x3", "missing", "5 zetas"])
def test_training_gradient_of_each_form(built_lib, oracle_lib, name):
    data = _tiny_dataset()
    m = _model(name, ["H", "Au"], "Au", act="p", hidden=(6, 5))
    tr = Trainer(data, m)  # sets scaling from the GPU descriptors
    g = tr.gradient([0, 1, 2], 3.0, 1.0, "fp64")
    tr.close()
    mw = max(m.n_weights(e) for e in range(m.nelem))
    rng = np.random.default_rng(5)
    for e in range(m.nelem):
        for k in rng.choice(m.n_weights(e), 5, replace=False):
            w0, h = m.weights[e][k], 1e-4 * max(1.0, abs(m.weights[e][k]))
            loss = []
            for s in (1, -1):
                m.weights[e][k] = w0 + s * h
                loss.append(_oracle_loss(m, data, 3.0, 1.0))
            m.weights[e][k] = w0
            fd = (loss[0] - loss[1]) / (2 * h)
            assert abs(g[e * mw + k] - fd) <= 1e-5 * max(abs(fd), 1e-6) + 1e-9, (e, k, g[e * mw + k], fd)
