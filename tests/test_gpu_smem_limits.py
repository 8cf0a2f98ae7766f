"""Sizes up to the shared-memory limit of a CTA run: a training network with as many neighbours as its
buffers leave room for (positions, weights, one gradient per warp, neighbour caches, network buffers)."""
import numpy as np
import pytest

from md_tian2_gb300 import nene
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.surrogate import Dataset, Trainer

pytestmark = pytest.mark.gpu

SLACK = 64  # the kernel's own static variables


def _train_bytes(natoms, maxnb, nelem, weights, ngeta):
    r16 = lambda b: (b + 15) // 16 * 16  # noqa: E731
    rs, warps = 4, 4
    s = 3 * r16(8 * natoms) + r16(8 * 18) + r16(8 * 64) + r16(natoms) + 6 * r16(rs * natoms)
    s += r16(rs * nelem * weights) * (1 + warps)
    s += r16(rs * warps * maxnb * (6 + ngeta)) + r16(rs * warps * maxnb * 3) + r16(4 * warps * maxnb) + r16(warps * maxnb)
    return s + r16(rs * warps * (2 * 64 + 6 * 5 * 64)) + r16(8 * 4)


def test_training_at_the_limit(built_lib):
    torch = pytest.importorskip("torch")
    limit = torch.cuda.get_device_properties(0).shared_memory_per_block_optin - SLACK
    rng = np.random.default_rng(2)
    us = [W.h_on_metal(rng, "Au", 3, 1.0, 0.0, 0.0, 300.0, z0=1.5 + 0.3 * t) for t in range(3)]
    for u in us:
        u.r[1:] += rng.normal(scale=0.06, size=u.r[1:].shape)
    data = Dataset(us, np.zeros(3), [np.zeros((u.natoms, 3)) for u in us])
    model = nene.random_model(["H", "Au"], hidden=(55, 55), act="p", seed=2, neighbours=["H", "Au"], descriptor="radial")
    w = max(model.n_weights(e) for e in range(model.nelem))
    maxnb = max(m for m in range(1, 400) if _train_bytes(us[0].natoms, m, model.nelem, w, 0) <= limit)
    assert 90 <= maxnb <= 255  # (the test's own sizes: room for the neighbours of the slab)
    tr = Trainer(data, model, max_neighbors=maxnb)
    g = tr.gradient([0, 1, 2], 1.0, 1.0, "fp32")
    tr.close()
    assert np.isfinite(g).all() and np.abs(g).max() > 0
