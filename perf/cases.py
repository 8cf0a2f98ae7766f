"""Performance cases of the engine: what a user's program has it do, through its public calls.

Every pass of a trajectory case is the call sequence of a host program that owns the state:
upload r and v from pinned host memory, evaluate the forces, run MD steps, download the state
(``Engine.upload_ptr``, ``calc_force``, ``md_steps``, ``mdt_state_download``).  The workloads
are the engine's own benchmark configurations (``workloads.config1`` ... ``config4`` and the
learned surrogate) from one trajectory to the full batch: FP64, FP32 and split-BF16
arithmetic, one force call up to many fused steps, and one training gradient.  Slabs are
displaced by thermal amounts (the reference starts from thermalised slab files) and the
projectile starts anywhere between the surface and its start height, as in a running batch.

Outputs: positions in FP64 always; velocities, forces, energies and embedded densities in
FP64 when the forces are computed in FP64, and in FP32 when the force arithmetic is FP32 or
split BF16 and holds no more than that.

``exact`` restates the same passes in 64-bit torch: energies from the formulas, forces by
autograd, the propagators step by step, the deviates from the same counter-based generator.
"""
import math
from functools import lru_cache

import numpy as np
import torch

from md_tian2_gb300 import constants as C
from md_tian2_gb300 import nene
from md_tian2_gb300 import workloads as W
from md_tian2_gb300.engine import PES_NENE, PES_SURROGATE, Engine, SimParams
from md_tian2_gb300.surrogate import Dataset, Trainer, shipped_surrogate, surrogate_model
from md_tian2_gb300.universe import Universe

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
F64 = torch.float64
SKIN = 0.5       # A, the skin the autotuner picks for the shipped surrogate
MARGIN = 0.1     # descriptor range margin before the surrogate's EMT fallback
MAXNB = {"surrogate": 80, "hdnnp": 96}
STEP, TEMP, GAMMA, PILE_TAU, RNG_SEED = 0.1, 300.0, 1e-3, 200.0, 2024
W_ENERGY, W_FORCE = 10.0, 1.0


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the reference's own use: one trajectory, one force call per host step (latency)
        dict(name="emt_force_one", kind="emt", prec="fp64", ntraj=1, kmin=3, kmax=3, algo="verlet", steps=0),
        # the plain 100-trajectory run on 3x3 slabs, velocity Verlet, fused steps
        dict(name="emt_fp64_100x3x3", kind="emt", prec="fp64", ntraj=100, kmin=3, kmax=3, algo="verlet", steps=100),
        # the uneven batch (37-145 atoms), Langevin metal: plain EMT in both force precisions
        dict(name="emt_fp64_4096", kind="emt", prec="fp64", ntraj=4096, kmin=3, kmax=6, algo="langevin", steps=20),
        dict(name="emt_fp32_4096", kind="emt", prec="fp32", ntraj=4096, kmin=3, kmax=6, algo="langevin", steps=20),
        # ring polymers with bead counts mixed per trajectory, PILE: the full batch with FP32
        # bead forces, a small one in FP64
        dict(name="rpmd_fp32_1024", kind="rpmd", prec="fp32", ntraj=1024, kmin=4, kmax=4, beads="4,8,16,32", steps=10),
        dict(name="rpmd_fp64_96", kind="rpmd", prec="fp64", ntraj=96, kmin=3, kmax=5, beads="4,6,10,16", steps=10),
        # the RuNNer-style network with angular functions on H/graphene: fused FP32 steps, the
        # tensor-core network's force call, and the FP64 parity force call of a small batch
        dict(name="hdnnp_fp32_2048", kind="hdnnp", prec="fp32", ntraj=2048, kmin=6, kmax=6, steps=5),
        dict(name="hdnnp_bf16x3_2048", kind="hdnnp", prec="bf16x3", ntraj=2048, kmin=6, kmax=6, steps=0),
        dict(name="hdnnp_fp64_64", kind="hdnnp", prec="fp64", ntraj=64, kmin=6, kmax=6, steps=0),
        # the learned surrogate: the full scattering batch on the tensor-core network, and a
        # small batch on the FP32 network
        dict(name="surrogate_bf16x3_4096", kind="surrogate", prec="bf16x3", ntraj=4096, kmin=3, kmax=6,
             algo="langevin", steps=100),
        dict(name="surrogate_fp32_100", kind="surrogate", prec="fp32", ntraj=100, kmin=3, kmax=6, algo="verlet",
             steps=50),
        # one gradient of the surrogate's training (energy and force loss, 256 configurations)
        dict(name="train_fp32_256", kind="train", prec="fp32", ntraj=512, batch=256, kmin=3, kmax=6,
             descriptor="radial"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["emt", "emt", "rpmd", "hdnnp", "surrogate", "surrogate", "train"])
    kmin = rng.randint(3, 6)
    kmax = rng.randint(kmin, 6)
    if kind == "emt":
        c = dict(kind=kind, prec=rng.choice(["fp64", "fp64", "fp32"]), ntraj=_log_int(rng, 1, 4000), kmin=kmin,
                 kmax=kmax, algo=rng.choice(["verlet", "langevin"]), steps=rng.choice([0, 1, 7, 20]))
        if c["ntraj"] > 2000:
            c.update(kmin=3, steps=min(c["steps"], 7))
        return c
    if kind == "rpmd":
        return dict(kind=kind, prec=rng.choice(["fp32", "fp64"]), ntraj=_log_int(rng, 1, 200), kmin=3,
                    kmax=rng.randint(3, 5), beads=rng.choice(["4,8,16,32", "2,4,8", "6,10,14", "8", "12,24", "16"]),
                    steps=rng.choice([1, 3, 10]))
    if kind == "hdnnp":
        prec = rng.choice(["fp32", "bf16x3", "fp64"])
        n = _log_int(rng, 1, {"fp32": 1000, "bf16x3": 1000, "fp64": 100}[prec])
        return dict(kind=kind, prec=prec, ntraj=n, kmin=rng.randint(4, 6), kmax=6,
                    steps=rng.choice([0, 1, 4]) if prec == "fp32" else 0)
    if kind == "surrogate":
        return dict(kind=kind, prec=rng.choice(["fp32", "bf16x3"]), ntraj=_log_int(rng, 1, 4000), kmin=3, kmax=kmax,
                    algo=rng.choice(["verlet", "langevin"]), steps=rng.choice([1, 10, 30]))
    n = _log_int(rng, 8, 600)
    return dict(kind=kind, prec=rng.choice(["fp32", "bf16x3"]), ntraj=n, batch=rng.randint(max(1, n // 3), n),
                kmin=kmin, kmax=kmax, descriptor=rng.choice(["radial", "acsf"]) if n < 100 else "radial")


# ---------------------------------------------------------------------------
# inputs from a seed
# ---------------------------------------------------------------------------
@lru_cache(maxsize=None)
def _slab(metal, k):
    """One trajectory's fixed data of a 4-layer k x k slab with its projectile (or of graphene)."""
    if metal == "C":
        pos, cell = W.graphene(k, ripple=0.0)
        fixed = np.zeros(len(pos), bool)
    else:
        pos, cell, fixed = W.fcc111_slab(W.LATTICE_A[metal], k)
    n = len(pos) + 1
    m = np.full(n, C.MASS_AMU[metal] * C.AMU2MASS)
    m[0] = C.MASS_AMU["H"] * C.AMU2MASS
    return pos, cell, np.concatenate([[False], fixed]), m, np.array([1] + [2] * (n - 1), np.int32)


def _metal(case):
    return {"rpmd": "Pt", "hdnnp": "C"}.get(case["kind"], "Au")


ALGO = {"verlet": C.PROP_ID_VERLET, "langevin": C.PROP_ID_LANGEVIN_CONST}


def _algos(case):
    if case["kind"] == "rpmd":
        return [C.PROP_ID_PILE, C.PROP_ID_PILE]
    return [C.PROP_ID_VERLET, ALGO[case.get("algo", "verlet")]]


@lru_cache(maxsize=4)
def _shapes(kmin, kmax, beads, ntraj):
    """Slab size and bead count per trajectory: the case's own, whatever the seed."""
    rng = np.random.default_rng(ntraj)
    ks = rng.integers(kmin, kmax + 1, ntraj)
    nbs = rng.choice([int(b) for b in beads.split(",")], ntraj)
    return ks, nbs


def _groups(case, seed):
    """Trajectories of one shape together: [(k, nb, indices, r (M, N, nb, 3), v)]."""
    ks, nbs = _shapes(case["kmin"], case["kmax"], case.get("beads", "1"), case["ntraj"])
    rng = np.random.default_rng(seed + 1000003)
    metal = _metal(case)
    out = []
    for k in np.unique(ks):
        for nb in np.unique(nbs[ks == k]):
            ids = np.where((ks == k) & (nbs == nb))[0]
            pos, cell, fixed, m, _ = _slab(metal, int(k))
            M, N = len(ids), len(m)
            r = np.empty((M, N, nb, 3))
            v = np.zeros((M, N, nb, 3))
            if metal == "C":
                r[:, 1:] = pos[None, :, None, :] + rng.normal(size=(M, N - 1, 1, 3)) * [0.02, 0.02, 0.05]
            else:
                amp = np.where(fixed[1:], 0.01, 0.06)[None, :, None, None]
                r[:, 1:] = pos[None, :, None, :] + amp * rng.normal(size=(M, N - 1, 1, 3))
            uv = rng.random((M, 2))
            r[:, 0, :, :2] = (uv @ cell[:2, :2].T)[:, None, :]
            r[:, 0, :, 2] = rng.uniform(1.6, 4.0 if metal == "C" else 6.0, (M, 1))
            sd = np.sqrt(C.KB * TEMP * nb / m[1:])[None, :, None, None]
            v[:, 1:] = sd * rng.normal(size=(M, N - 1, nb, 3)) * ~fixed[1:][None, :, None, None]
            einc = rng.uniform(0.5, 5.0 if metal == "Au" else 2.0, M)
            pol = np.radians(rng.uniform(0.0, 60.0 if metal == "Au" else 0.0, M))
            azi = np.radians(rng.uniform(0.0, 360.0, M))
            vi = np.sqrt(2.0 * einc / m[0])
            v[:, 0] += np.stack([vi * np.sin(pol) * np.cos(azi), vi * np.sin(pol) * np.sin(azi), -vi * np.cos(pol)],
                                1)[:, None, :]
            if nb > 1:  # beads of an equilibrated ring polymer lie apart
                r += np.where(fixed, 0.0, np.where(np.arange(N) == 0, 0.1, 0.01))[None, :, None, None] * \
                    rng.normal(size=r.shape)
                v[:, 0] += math.sqrt(C.KB * TEMP * nb / m[0]) * rng.normal(size=v[:, 0].shape)
            out.append((int(k), int(nb), ids, r, v))
    return out


def _universes(case, groups):
    metal = _metal(case)
    us = [None] * case["ntraj"]
    for k, nb, ids, r, v in groups:
        _, cell, fixed, m, idx = _slab(metal, k)
        fx = np.broadcast_to(fixed[:, None, None], (len(m), nb, 3)).copy()
        for a, t in enumerate(ids):
            us[t] = Universe(r=r[a], v=v[a], m=m, idx=idx, is_fixed=fx, simbox=cell, names=["H", metal],
                             is_proj=np.array([True, False]), algo=np.array(_algos(case), np.int32))
    return us


@lru_cache(maxsize=None)
def _hdnnp_model():
    """The H/graphene network (8 G2 + 16 G3, 24-25-25-1 tanh, seeded weights), scaling from the
    descriptors of eight configurations."""
    m = nene.random_model(["H", "C"], hidden=(25, 25), act="t", seed=5, neighbours=["C"])
    g = _groups(dict(kind="hdnnp", kmin=6, kmax=6, ntraj=8), 77)[0]
    G = _descriptors(m, torch.tensor(g[3][:, :, 0]), *_nn_static(m, "C", 6, "cpu"))
    for e in range(2):
        x = (G[:, :1] if e == 0 else G[:, 1:]).reshape(-1, G.shape[-1])
        lo, hi = x.min(0).values.numpy(), x.max(0).values.numpy()
        pad = np.where(hi - lo < 1e-9, 1e-3, 0.0)
        m.smin[e], m.smax[e], m.savg[e] = lo - pad, hi + pad, x.mean(0).numpy()
    m.scalesym = True
    return m


def _train_model(case):
    m = surrogate_model(seed=11, descriptor=case["descriptor"])
    m.weights = [np.asarray(w, np.float32).astype(np.float64) for w in m.weights]
    return m


def _model(case):
    return {"hdnnp": _hdnnp_model, "surrogate": shipped_surrogate}[case["kind"]]()


def _sim():
    return SimParams(step=STEP, Tsurf=TEMP, Tproj=TEMP, gamma_const=GAMMA, pile_tau=PILE_TAU, seed=RNG_SEED)


class _State:
    def __init__(self, case):
        self.case = case
        self.wide = case["prec"] == "fp64"
        self.sp = _sim()


def _pinned(n):
    t = torch.empty(int(n), dtype=F64)
    return t.pin_memory() if torch.cuda.is_available() else t


def prepare(case, seed):
    s = _State(case)
    groups = _groups(case, seed)
    us = _universes(case, groups)
    if case["kind"] == "train":
        lab = Engine(0)
        lab.read_emt(W.emt_params())
        lab.define(us)
        lab.upload()
        lab.calc_force(s.sp)
        o = lab.download()
        forces = [lab.split(o["f"], t)[:, 0, :].copy() for t in range(len(us))]
        s.trainer = Trainer(Dataset(us, o["epot"].copy(), forces), _train_model(case))
        lab.close()
        s.ids = _train_ids(case, seed)
        return s
    eng = s.eng = Engine(0)
    if case["kind"] != "hdnnp":
        eng.read_emt(W.emt_params("H", _metal(case)))
    eng.define(us)
    if case["kind"] in MAXNB:
        eng.read_nene(_model(case), ["H", _metal(case)], max_neighbors=MAXNB[case["kind"]])
        if case["kind"] == "hdnnp":
            eng.set_pes(PES_NENE, 0.0)
        else:
            eng.set_pes(PES_SURROGATE, MARGIN)
            eng.nn_set_skin(SKIN)
    n3 = 3 * eng.nslots
    s.r0, s.v0 = _pinned(n3), _pinned(n3)
    torch.cat([torch.from_numpy(u.r).reshape(-1) for u in us], out=s.r0)
    torch.cat([torch.from_numpy(u.v).reshape(-1) for u in us], out=s.v0)
    s.out = {"f": _pinned(n3), "epot": _pinned(eng.bead_off[-1])}
    if case["steps"]:
        s.out.update(r=_pinned(n3), v=_pinned(n3))
    if case["kind"] in ("emt", "rpmd"):
        s.out["dens"] = _pinned(eng.nslots)
    return s


def _train_ids(case, seed):
    return np.random.default_rng(seed + 5).permutation(case["ntraj"])[: case["batch"]]


def run(s):
    case = s.case
    if case["kind"] == "train":
        g = s.trainer.gradient(s.ids, W_ENERGY, W_FORCE, case["prec"])
        return {"grad": torch.from_numpy(g).float()}
    eng, prec = s.eng, case["prec"]
    eng.upload_ptr(s.r0.data_ptr(), s.v0.data_ptr())
    eng.calc_force(s.sp, precision=prec)
    if case["steps"]:
        eng.md_steps(case["steps"], s.sp, precision=prec)
    ptr = {k: t.data_ptr() for k, t in s.out.items()}
    eng._check(eng.lib.mdt_state_download(eng.h, ptr.get("r"), ptr.get("v"), ptr["f"], None, ptr["epot"],
                                          ptr.get("dens")), "mdt_state_download")
    return {k: t if s.wide or k == "r" else t.float() for k, t in s.out.items()}


# ---------------------------------------------------------------------------
# work that a pass cannot do without
# ---------------------------------------------------------------------------
@lru_cache(maxsize=None)
def _counts(metal, k, rc, images):
    """Directed neighbour pairs within rc of the undisplaced slab (nearest images, or all)."""
    pos, cell, *_ = _slab(metal, k)
    d = pos[:, None] - pos[None]
    if not images:
        f = d @ np.linalg.inv(cell).T
        d = (f - np.round(f)) @ cell.T
        r = np.linalg.norm(d, axis=-1)
        return int(((r > 0) & (r <= rc)).sum())
    n = 0
    for a in range(-4, 5):
        for b in range(-4, 5):
            r = np.linalg.norm(d + a * cell[:, 0] + b * cell[:, 1], axis=-1)
            n += int(((r > 1e-9) & (r <= rc)).sum())
    return n


def work(case):
    metal = _metal(case)
    ks = range(case["kmin"], case["kmax"] + 1)
    beads = [int(b) for b in case.get("beads", "1").split(",")]
    nb = sum(beads) / len(beads)
    slots = float(np.mean([_slab(metal, k)[3].size for k in ks])) * case["ntraj"] * nb
    if case["kind"] == "train":
        pairs = float(np.mean([_counts(metal, k, 6.5, True) for k in ks])) * case["batch"]
        rows = slots * case["batch"] / case["ntraj"]
        return {"bytes": 48.0 * rows, "flops": 5 * 492.0 / 2 * pairs + 30000.0 * rows}
    nf = 1 + case["steps"]
    # r and v in; r, v, f (and the energies) out
    moved = slots * 8 * (6 + (9 if case["steps"] else 3) + 1)
    if case["kind"] in ("emt", "rpmd"):
        cut = 1.5 * W.EMT_TABLE[("H", metal)][metal][6] * (16 * math.pi / 3) ** (1 / 3) / math.sqrt(2) * math.sqrt(3)
        pairs = float(np.mean([_counts(metal, k, cut, False) for k in ks])) / 2 * case["ntraj"] * nb
        flops = nf * (200.0 * pairs + 100.0 * slots)
        if case["kind"] == "rpmd":
            flops += case["steps"] * slots * 3 * 6 * 2 * sum(b * b for b in beads) / sum(beads)
        return {"bytes": moved, "flops": flops}
    pairs = float(np.mean([_counts(metal, k, 6.5, True) for k in ks])) * case["ntraj"]
    if case["kind"] == "surrogate":
        return {"bytes": moved, "flops": nf * (492.0 * pairs + 11000.0 * slots)}
    # about 12 valid triplets (j < k, all three distances inside the cutoff) per neighbour
    return {"bytes": moved, "flops": nf * ((120.0 + 12 * 220.0) * pairs + 9000.0 * slots)}


# ---------------------------------------------------------------------------
# the same passes in 64 bits
# ---------------------------------------------------------------------------
def _emt_const(metal):
    t = W.EMT_TABLE[("H", metal)]
    beta = (16.0 * math.pi / 3.0) ** (1.0 / 3.0) / math.sqrt(2.0)
    prm = [dict(zip(("eta2", "n0", "e0", "lam", "v0", "kappa", "s0"), t[x])) for x in ("H", metal)]
    bs0 = [beta * p["s0"] for p in prm]
    rcut = max(bs0) * math.sqrt(3.0)
    acut = 9.21034037197618 / (4.0 * rcut / (math.sqrt(3.0) + 2) - rcut)
    for p, b in zip(prm, bs0):
        shell = [(n / 12.0 / (1 + math.exp(acut * (b * q - rcut))), b * q) for n, q in
                 ((12, 1.0), (6, math.sqrt(2.0)), (24, math.sqrt(3.0)))]
        p["g1"] = sum(x * math.exp(-p["eta2"] * (r - b)) for x, r in shell)
        p["g2"] = sum(x * math.exp(-p["kappa"] / beta * (r - b)) for x, r in shell)
        p["b"], p["kb"], p["be"] = b, p["kappa"] / beta, beta * p["eta2"]
    c21 = prm[0]["n0"] / prm[1]["n0"] * math.exp(0.5 / C.BOHR2ANG * (prm[1]["s0"] - prm[0]["s0"]))
    return prm, rcut, acut, torch.tensor([[1.0, 1.0 / c21], [c21, 1.0]], dtype=F64, device=DEVICE)


def _emt(r, metal, k):
    """EMT of configurations r (M, N, 3): energy, forces, embedded density."""
    _, cell, _, _, idx = _slab(metal, k)
    prm, rcut, acut, chi = _emt_const(metal)
    per = lambda key: torch.tensor([p[key] for p in prm], dtype=F64, device=DEVICE)  # noqa: E731
    ty = torch.tensor(idx.astype(np.int64) - 1, device=DEVICE)
    box = torch.tensor(cell, device=DEVICE)
    ib = torch.linalg.inv(box)
    N = r.shape[1]
    es, fs, ds = [], [], []
    for x in torch.split(r, max(1, int(2e7 // (N * N)))):
        x = x.detach().clone().requires_grad_(True)
        d = x[:, :, None] - x[:, None]
        d = d - (torch.round(d.detach() @ ib.T) @ box.T)
        r2 = (d * d).sum(-1)
        eye = torch.eye(N, dtype=torch.bool, device=DEVICE)
        on = (r2.detach() <= (1.5 * rcut) ** 2) & ~eye
        q = torch.sqrt(torch.where(eye, torch.ones_like(r2), r2))
        th = torch.where(on, 1.0 / (1.0 + torch.exp(acut * (q - rcut))), torch.zeros_like(q))
        c = chi[ty][:, ty]
        sig = (th * torch.exp(-per("eta2")[ty] * (q - per("b")[ty])) * c).sum(-1) / per("g1")[ty]
        pair = -0.5 * (th * torch.exp(-per("kb")[ty] * (q - per("b")[ty])) * c).sum(-1) * (per("v0") / per("g2"))[ty]
        # the density is floored in the energy at 1e-9 but its derivative is that of log(sigma)
        ln = torch.log(torch.clamp(sig, min=1e-30))
        sa = -(ln + (torch.log(torch.clamp(sig, min=1e-9)) - ln).detach() - math.log(12.0)) / per("be")[ty]
        lam = per("lam")[ty]
        e = (pair + per("e0")[ty] * ((1 + lam * sa) * torch.exp(-lam * sa) - 1) +
             6 * per("v0")[ty] * torch.exp(-per("kappa")[ty] * sa)).sum(-1)
        fs.append(-torch.autograd.grad(e.sum(), x)[0])
        es.append(e.detach())
        ds.append((per("n0")[ty] * torch.exp((0.5 / C.BOHR2ANG - per("be")[ty]) * sa)).detach())
    return torch.cat(es), torch.cat(fs), torch.cat(ds)


def _nn_static(model, metal, k, dev):
    """Cell (bohr, columns), element per atom and the cell images that can hold neighbours."""
    cell = _slab(metal, k)[1] * C.ANG2BOHR
    names = ["H", metal]
    elem = torch.tensor([model.elements.index(names[i - 1]) for i in _slab(metal, k)[4]], device=dev)
    inv = np.linalg.inv(cell)
    reach = [int(math.ceil(model.maxcut * np.linalg.norm(inv[d]))) for d in range(3)]
    sh = [(a, b, c) for a in range(-reach[0], reach[0] + 1) for b in range(-reach[1], reach[1] + 1)
          for c in range(-reach[2], reach[2] + 1)]
    return torch.tensor(cell, device=dev), elem, torch.tensor(sh, dtype=F64, device=dev)


def _descriptors(model, r, box, elem, shifts):
    """Symmetry functions (M, N, nsf) of r (M, N, 3) in A (differentiable)."""
    dev = r.device
    M, N, _ = r.shape
    x = r * C.ANG2BOHR
    x = x - torch.floor(x.detach() @ torch.linalg.inv(box).T) @ box.T
    rc = model.maxcut
    # neighbours (directed), padded to the longest list
    xd = x.detach()
    found = []
    for s in shifts:
        d = xd[:, None] + (box @ s) - xd[:, :, None]  # (M, i, j, 3)
        r2 = (d * d).sum(-1)
        ok = r2 <= rc * rc
        if bool((s == 0).all()):
            ok &= ~torch.eye(N, dtype=torch.bool, device=dev)
        w = ok.nonzero()
        found.append(torch.cat([w, (box @ s).expand(len(w), 3)], 1) if len(w) else torch.zeros(0, 6, device=dev, dtype=F64))
    found = torch.cat(found)
    ci = (found[:, 0] * N + found[:, 1]).long()
    ci, perm = torch.sort(ci, stable=True)
    found = found[perm]
    cnt = torch.bincount(ci, minlength=M * N)
    start = torch.cumsum(cnt, 0) - cnt
    P = max(1, int(cnt.max()))
    slot = torch.arange(len(ci), device=dev) - start[ci]
    j = torch.zeros(M * N, P, dtype=torch.long, device=dev)
    off = torch.full((M * N, P, 3), 0.0, dtype=F64, device=dev)
    on = torch.zeros(M * N, P, dtype=torch.bool, device=dev)
    j[ci, slot] = (found[:, 0] * N + found[:, 2]).long()
    off[ci, slot] = found[:, 3:]
    on[ci, slot] = True
    xf = x.reshape(-1, 3)
    d = xf[j] + off - xf[:, None]
    d = torch.where(on[..., None], d, torch.full_like(d, 1.0))
    q = torch.sqrt((d * d).sum(-1))
    zn = torch.tensor(model.z, device=dev)[elem][j % N]
    zn = torch.where(on, zn, torch.zeros_like(zn))
    fc = torch.where(on, 0.5 * (torch.cos(math.pi * q / rc) + 1.0), torch.zeros_like(q))
    G2, G3 = {}, {}
    tri = None
    for sf in (s for e in model.sfs for s in e):
        if sf.type == 2 and (sf.eta, sf.rshift, sf.e1) not in G2:
            g = torch.exp(-sf.eta * (q - sf.rshift) ** 2) * fc
            G2[(sf.eta, sf.rshift, sf.e1)] = torch.where(zn == sf.e1, g, torch.zeros_like(g)).sum(-1)
        elif sf.type == 3 and (sf.eta, sf.lam, sf.zeta, sf.e1, sf.e2) not in G3:
            if tri is None:
                a, b = torch.triu_indices(P, P, 1, device=dev)
                # keep the triplets whose third distance is inside the cutoff
                dd = d.detach()
                keep = (((dd[:, a] - dd[:, b]) ** 2).sum(-1) <= rc * rc) & on[:, a] & on[:, b]
                w = keep.nonzero()
                cen, a, b = w[:, 0], a[w[:, 1]], b[w[:, 1]]
                da, db = d[cen, a], d[cen, b]
                dj = da - db
                q2 = (dj * dj).sum(-1)
                qjk = torch.sqrt(q2)
                cs = (da * db).sum(-1) / (q[cen, a] * q[cen, b])
                base = fc[cen, a] * fc[cen, b] * 0.5 * (torch.cos(math.pi * qjk / rc) + 1.0)
                tri = (cen, zn[cen, a], zn[cen, b], cs, base, q[cen, a] ** 2 + q[cen, b] ** 2 + q2, {})
            cen, za, zb, cs, base, ssum, memo = tri
            if ("x", sf.eta) not in memo:
                memo[("x", sf.eta)] = torch.exp(-sf.eta * ssum) * base
            if (sf.lam, sf.zeta) not in memo:
                memo[(sf.lam, sf.zeta)] = 2.0 ** (1.0 - sf.zeta) * torch.clamp(1.0 + sf.lam * cs, min=0.0) ** sf.zeta
            g = memo[("x", sf.eta)] * memo[(sf.lam, sf.zeta)]
            m = ((za == sf.e1) & (zb == sf.e2)) | ((za == sf.e2) & (zb == sf.e1))
            G3[(sf.eta, sf.lam, sf.zeta, sf.e1, sf.e2)] = torch.zeros(M * N, dtype=F64, device=dev).index_add(
                0, cen, torch.where(m, g, torch.zeros_like(g)))
    rows = []
    for e in range(model.nelem):
        rows.append(torch.stack([(G2[(s.eta, s.rshift, s.e1)] if s.type == 2 else
                                  G3[(s.eta, s.lam, s.zeta, s.e1, s.e2)]) for s in model.sfs[e]], -1))
    ef = elem.repeat(M)
    G = rows[0]
    for e in range(1, model.nelem):
        G = torch.where((ef == e)[:, None], rows[e], G)
    return G.reshape(M, N, -1)


ACT = {"t": torch.tanh, "l": lambda v: v, "p": torch.nn.functional.softplus, "s": torch.sigmoid}


def _network(model, G, elem, theta):
    """Energies (M,) in eV of raw descriptors G; theta: flat weights per element."""
    e_atom = torch.zeros(G.shape[:2], dtype=F64, device=G.device)
    for e in range(model.nelem):
        lo = torch.tensor(np.asarray(model.smin[e], float), device=G.device)
        hi = torch.tensor(np.asarray(model.smax[e], float), device=G.device)
        sel = (elem == e).nonzero()[:, 0]
        v = (G[:, sel] - lo) / (hi - lo) * (model.scmax - model.scmin) + model.scmin if model.scalesym else G[:, sel]
        nodes, ic = model.nodes[e], 0
        for l in range(1, len(nodes)):
            w = theta[e][ic: ic + nodes[l - 1] * nodes[l]].reshape(nodes[l - 1], nodes[l])
            ic += nodes[l - 1] * nodes[l]
            v = v @ w + theta[e][ic: ic + nodes[l]]
            ic += nodes[l]
            a = model.acts[e][l - 1][0]
            v = torch.where(v > 30, v, torch.log1p(torch.exp(torch.clamp(v, max=30.0)))) if a == "p" else ACT[a](v)
        e_atom = e_atom.index_add(1, sel, v[..., 0])
    return e_atom.sum(-1) * C.HA2EV


def _theta(model):
    return [torch.tensor(np.asarray(w, float), device=DEVICE) for w in model.weights]


def _nn(r, model, metal, k, fallback):
    """Network energies and forces of r (M, N, 3); fallback: EMT where a descriptor leaves its range."""
    box, elem, sh = _nn_static(model, metal, k, DEVICE)
    th = _theta(model)
    es, fs = [], []
    per = max(1, int((6000 if any(s.type == 3 for e in model.sfs for s in e) else 30000) // r.shape[1]))
    for x in torch.split(r, per):
        x = x.detach().clone().requires_grad_(True)
        G = _descriptors(model, x, box, elem, sh)
        e = _network(model, G, elem, th)
        f = -torch.autograd.grad(e.sum(), x)[0]
        e = e.detach()
        if fallback:
            lo = torch.stack([torch.tensor(np.asarray(model.smin[i], float), device=DEVICE) for i in elem.tolist()])
            hi = torch.stack([torch.tensor(np.asarray(model.smax[i], float), device=DEVICE) for i in elem.tolist()])
            w = MARGIN * (hi - lo)
            out = ((G.detach() < lo - w) | (G.detach() > hi + w)).any(-1).any(-1)
            if bool(out.any()):
                ee, ff, _ = _emt(x[out], metal, k)
                e[out], f[out] = ee, ff
        es.append(e)
        fs.append(f)
    return torch.cat(es), torch.cat(fs), None


def _normals(ids, step, nb, N, stream):
    """Counter-based N(0, 1) deviates (M, N, nb, 3): Philox4x32-10, Box-Muller on 24-bit uniforms."""
    mask = 0xFFFFFFFF
    slot = torch.arange(nb * N * 3, device=DEVICE, dtype=torch.int64)[None]
    traj = torch.tensor(np.asarray(ids, np.int64), device=DEVICE)[:, None]
    x, y, z, w = (torch.zeros(len(ids), nb * N * 3, dtype=torch.int64, device=DEVICE) + c for c in (step, slot, stream, traj))
    k0, k1 = RNG_SEED & mask, RNG_SEED >> 32
    for _ in range(10):
        a, b = x * 0xD2511F53, z * 0xCD9E8D57
        x, y, z, w = ((b >> 32) & mask) ^ y ^ k0, b & mask, ((a >> 32) & mask) ^ w ^ k1, a & mask
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    u1 = ((x >> 8) + 1).to(F64) / 16777216.0
    u2 = (z >> 8).to(F64) / 16777216.0
    g = torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * u2)
    return g.reshape(len(ids), nb, N, 3).transpose(1, 2)


def _cjk(nb):
    c = np.zeros((nb, nb))
    for j in range(1, nb + 1):
        for k in range(nb):
            if k == 0:
                c[j - 1, k] = math.sqrt(1.0 / nb)
            elif k <= nb // 2 - 1:
                c[j - 1, k] = math.sqrt(2.0 / nb) * math.cos(2 * math.pi * j * k / nb)
            elif k == nb // 2:
                c[j - 1, k] = math.sqrt(1.0 / nb) * (-1.0 if j % 2 else 1.0)
            else:
                c[j - 1, k] = math.sqrt(2.0 / nb) * math.sin(2 * math.pi * j * k / nb)
    return torch.tensor(c, device=DEVICE)


def _exact_group(case, k, nb, ids, r, v):
    metal = _metal(case)
    _, _, fixed, m, _ = _slab(metal, k)
    N = len(m)
    r, v = torch.tensor(r, device=DEVICE), torch.tensor(v, device=DEVICE)
    mass = torch.tensor(m, device=DEVICE)[:, None, None]
    mob = torch.tensor(~fixed, device=DEVICE).to(F64)[:, None, None]
    hbar, kb = 0.6582119514467406, 8.61733238496e-5
    kt = kb * TEMP
    cj = _cjk(nb)
    mode = torch.arange(nb, device=DEVICE, dtype=F64)
    model = _model(case) if case["kind"] in MAXNB else None

    def force(r, v):
        if nb > 1:  # free ring-polymer step in normal modes, mobile atoms
            p = torch.einsum("mibd,bk->mikd", mass * v, cj)
            q = torch.einsum("mibd,bk->mikd", r, cj)
            wk = (2.0 * kt * nb / hbar) * torch.sin(torch.minimum(mode, nb - mode) * math.pi / nb)
            cw, sw = torch.cos(wk * STEP)[:, None], torch.sin(wk * STEP)[:, None]
            wm = torch.where(mode == 0, torch.ones_like(mode), wk)[:, None] * mass
            first = (mode == 0)[:, None]
            pn = torch.where(first, p, p * cw - q * wm * sw)
            qn = torch.where(first, q + p * STEP / mass, p * sw / wm + q * cw)
            moved = torch.einsum("mikd,bk->mibd", qn, cj)
            r = torch.where(mob > 0, moved, r)
            v = torch.where(mob > 0, torch.einsum("mikd,bk->mibd", pn, cj) / mass, v)
        x = r.transpose(1, 2).reshape(-1, N, 3)
        if model is None:
            e, f, dens = _emt(x, metal, k)
        else:
            e, f, dens = _nn(x, model, metal, k, case["kind"] == "surrogate")
        f = f.reshape(len(ids), nb, N, 3).transpose(1, 2)
        dens = None if dens is None else dens.reshape(len(ids), nb, N).transpose(1, 2)
        return r, v, f, e.reshape(len(ids), nb), dens

    algo = [case.get("algo", "verlet") if case["kind"] != "rpmd" else "pile"]
    lang = torch.zeros(N, 1, 1, dtype=F64, device=DEVICE)
    if algo[0] == "langevin":
        lang[1:] = 1.0
    xi = GAMMA * STEP
    T = kt / mass
    c0, c1 = 1 - xi + 0.5 * xi * xi, (1 - 0.5 * xi + xi * xi / 6) * STEP
    c2 = (0.5 - xi / 6 + xi * xi / 24) * STEP
    s_r = STEP * torch.sqrt(T * (8 / 12 * xi - 0.5 * xi * xi))
    s_v = torch.sqrt(2 * T * xi * (1 - xi))
    c_rv = 0.5 * math.sqrt(3.0) * (1 - 0.125 * xi)
    r, v, f, e, dens = force(r, v)
    for step in range(1, case["steps"] + 1):
        a = f / mass * mob
        if algo[0] == "pile":
            gam = torch.where(mode == 0, torch.full_like(mode, 1.0 / PILE_TAU),
                              4 * kt * nb / hbar * torch.sin(mode * math.pi / nb))
            d1 = torch.exp(-0.5 * STEP * gam)[:, None]
            d2 = torch.sqrt(1 - d1 * d1)
            p = torch.einsum("mibd,bk->mikd", mass * v, cj)
            p = d1 * p + torch.sqrt(mass * kt * nb) * d2 * _normals(ids, step, nb, N, 2)
            v = torch.einsum("mikd,bk->mibd", p, cj) / mass * mob
        if algo[0] == "langevin":
            g = _normals(ids, step, nb, N, 1)
            vn = v + 0.5 * STEP * a
            rl = r + (c1 * v + c2 * STEP * a + s_r * g) * mob
            vl = (c0 * v + (c1 - c2) * a + s_v * c_rv * g) * mob
            r = torch.where(lang > 0, rl, r + STEP * vn * mob)
            v = torch.where(lang > 0, vl, vn * mob)
        else:
            v = (v + 0.5 * STEP * a) * mob
            if nb == 1:
                r = r + STEP * v * mob
        if algo[0] == "pile":
            com = (mass * v).sum(2).sum(1) / mass.sum() / nb
            v = v - com[:, None, None] * (1 - (1 - 1.0 / N) ** 1000)
        r, v, f, e, dens = force(r, v)
        a = f / mass * mob
        if algo[0] == "langevin":
            v = torch.where(lang > 0, (v + c2 * a + s_v * math.sqrt(1 - c_rv * c_rv) * g) * mob,
                            (v + 0.5 * STEP * a) * mob)
        else:
            v = (v + 0.5 * STEP * a) * mob
    return {"r": r, "v": v, "f": f, "epot": e, "dens": dens}


def _exact_train(case, seed, groups):
    model = _train_model(case)
    ids = _train_ids(case, seed)
    # labels and scaling from every configuration of the set
    lab, low, high = {}, {}, {}
    for k, _, idx, r, _ in groups:
        x = torch.tensor(r[:, :, 0], device=DEVICE)
        e, f, _ = _emt(x, "Au", k)
        box, elem, sh = _nn_static(model, "Au", k, DEVICE)
        for part in torch.split(torch.arange(len(idx)), max(1, 6000 // x.shape[1])):
            with torch.no_grad():
                G = _descriptors(model, x[part.to(DEVICE)], box, elem, sh)
            for el in range(2):
                g = G[:, (elem == el).nonzero()[:, 0]].reshape(-1, G.shape[-1])
                low[el] = torch.minimum(low[el], g.min(0).values) if el in low else g.min(0).values
                high[el] = torch.maximum(high[el], g.max(0).values) if el in high else g.max(0).values
        for a, t in enumerate(idx):
            lab[int(t)] = (k, x[a], e[a], f[a])
    for el in range(2):
        lo, hi = low[el].cpu().numpy(), high[el].cpu().numpy()
        pad = np.where(hi - lo < 1e-12, np.maximum(0.05 * np.abs(lo), 5e-4), 0.0)
        model.smin[el], model.smax[el] = lo - pad, hi + pad
    model.scalesym = True
    th = [t.requires_grad_(True) for t in _theta(model)]
    total = [torch.zeros_like(t) for t in th]
    for k in sorted({lab[int(t)][0] for t in ids}):
        here = [int(t) for t in ids if lab[int(t)][0] == k]
        box, elem, sh = _nn_static(model, "Au", k, DEVICE)
        N = len(elem)
        for s in range(0, len(here), max(1, 1500 // N)):
            part = [lab[t] for t in here[s: s + max(1, 1500 // N)]]
            x = torch.stack([p[1] for p in part]).requires_grad_(True)
            E = _network(model, _descriptors(model, x, box, elem, sh), elem, th)
            F = -torch.autograd.grad(E.sum(), x, create_graph=True)[0]
            dE = (E - torch.stack([p[2] for p in part])) / N
            dF = F - torch.stack([p[3] for p in part])
            loss = W_ENERGY * (dE * dE).sum() + W_FORCE * (dF * dF).sum() / (3 * N)
            for t, g in zip(total, torch.autograd.grad(loss, th)):
                t += g
    mw = max(model.n_weights(e) for e in range(2))
    out = torch.zeros(2, mw, dtype=F64)
    for e in range(2):
        out[e, : len(total[e])] = total[e].cpu() / len(ids)
    return {"grad": out.reshape(-1)}


def exact(case, seed):
    groups = _groups(case, seed)
    if case["kind"] == "train":
        return _exact_train(case, seed, groups)
    slots = sum(r.shape[0] * r.shape[1] * r.shape[2] for *_, r, _ in groups)
    cost = {"emt": 1e-7, "rpmd": 1e-7, "surrogate": 2e-6, "hdnnp": 1.4e-5}[case["kind"]]
    if cost * slots * (1 + case["steps"]) > 15.0:  # about 20 s and more
        return None
    parts = {}
    ks, nbs = _shapes(case["kmin"], case["kmax"], case.get("beads", "1"), case["ntraj"])
    for k, nb, ids, r, v in groups:
        got = _exact_group(case, k, nb, ids, r, v)
        for key, t in got.items():
            if t is not None:
                flat = t.reshape(len(ids), -1).cpu()
                for a, i in enumerate(ids):
                    parts.setdefault(key, [None] * case["ntraj"])[i] = flat[a]
    keys = ("f", "epot") + (("r", "v") if case["steps"] else ()) + (("dens",) if "dens" in parts else ())
    wide = case["prec"] == "fp64"
    return {key: torch.cat(parts[key]).to(F64) if wide or key == "r" else torch.cat(parts[key]) for key in keys}
