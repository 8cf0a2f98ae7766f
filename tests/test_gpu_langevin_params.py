"""Constant-friction Langevin propagation takes its friction, step and temperatures from each call,
whatever ran before: other parameters in turn, calls captured in a CUDA graph and replayed between
others, another stream.  Against the oracle with the same deviates (parity bar 1e-10)."""
import ctypes as ct

import numpy as np
import pytest

from md_tian2_gb300 import constants as C
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import SimParams

from .helpers import flat, injected, make_engine, max_abs, oracle_list

pytestmark = pytest.mark.gpu

A = SimParams(step=0.1, gamma_const=1e-3)
B = SimParams(step=0.1, gamma_const=0.5, Tsurf=900.0)  # gamma dt above the series' limit: other formulas
D = SimParams(step=0.07, gamma_const=1e-3, Tproj=50.0)


def _both(nbeads):
    rng = np.random.default_rng(nbeads)
    us = [W.h_on_metal(rng, "Au", 3, 1.0, 20.0, 30.0, 300.0, C.PROP_ID_LANGEVIN_CONST, C.PROP_ID_LANGEVIN_CONST, z0=1.6,
                       nbeads=nbeads) for _ in range(2)]
    emt = W.emt_params()
    eng = make_engine(us, emt)
    orcs = oracle_list(us, emt)
    dev = injected(us, rng)
    eng.set_random_arrays(*[flat(d) for d in dev])
    return us, eng, orcs, dev


def _inj(sp):
    return SimParams(**{**sp.__dict__, "rng_mode": 1})


def _oracle_step(orcs, dev, sp):
    randy, zeta, av, au = dev
    for t, o in enumerate(orcs):
        sh = o.r.shape
        o.propagate_1(sp, randy[t].reshape(sh), zeta[t].reshape(sh), av[t].reshape(sh), au[t].reshape(sh[:2]))
        o.calc_force(sp)
        o.propagate_2(sp, randy[t].reshape(sh))


def _same(eng, orcs):
    out = eng.download()
    for k in ("r", "v"):
        assert max_abs(out[k], np.concatenate([getattr(o, k).reshape(-1) for o in orcs])) < 1e-10, k


@pytest.mark.parametrize("nbeads", [1, 4])
@pytest.mark.parametrize("fused", [True, False])
def test_parameters_of_each_call(built_lib, oracle_lib, nbeads, fused):
    us, eng, orcs, dev = _both(nbeads)
    eng.calc_force(A)
    for o in orcs:
        o.calc_force(A)
    for sp in (A, B, A, D, D, B):
        if fused:
            eng.md_steps(1, _inj(sp))
        else:
            eng.propagate_1(_inj(sp))
            eng.calc_force(_inj(sp))
            eng.propagate_2(_inj(sp))
        _oracle_step(orcs, dev, sp)
        _same(eng, orcs)
    eng.close()


def test_graph_replay_between_calls(built_lib, oracle_lib):
    torch = pytest.importorskip("torch")
    us, eng, orcs, dev = _both(1)
    s, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    eng.synchronize()
    eng._check(eng.lib.mdt_set_stream(eng.h, ct.c_void_p(s.cuda_stream)), "mdt_set_stream")
    eng.calc_force(A)
    for o in orcs:
        o.calc_force(A)
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=s, capture_error_mode="thread_local"):
        eng.md_steps(1, _inj(A))  # recorded, not run

    def replay():
        with torch.cuda.stream(s):
            graph.replay()

    for sp in (A, B, None, B, None, A, None):
        if sp is None:
            replay()
        else:
            eng.md_steps(1, _inj(sp))
        _oracle_step(orcs, dev, sp or A)
        _same(eng, orcs)
    eng.synchronize()
    eng._check(eng.lib.mdt_set_stream(eng.h, ct.c_void_p(s2.cuda_stream)), "mdt_set_stream")
    for sp in (A, D):
        eng.md_steps(1, _inj(sp))
        _oracle_step(orcs, dev, sp)
        _same(eng, orcs)
    eng.synchronize()
    del graph
    eng.close()
