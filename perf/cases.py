"""Performance cases of the library: the work a program built on it has it do, through its Python front end.

A case is a dict of plain values; "kind" selects the program:

  step      one step of a measurement loop in one call (Engine.sweeps_io), from a replayed graph
  scan      one point of a mode loop: thermalisation sweeps, measured sweeps, the series and the final field
  batch     a batch of replicas in blocks of measured sweeps (Engine.sweeps_io with every replica's temperature)
  polar     the pear mode loop: after every measured sweep its record and the polar and radial order parameters
  collect   training samples for the learned proposal from states a few sweeps apart
  learned   measured sweeps with the learned proposal
  train     optimiser steps of the proposal network on mini-batches of samples
  snapshot  the observables of a given field, its local order and the field itself, as a snapshot writer needs them

Records of measured sweeps are kept in float32: their terms are FP32 site energies and directors, and the programs
print six digits of them (po.dat). What is computed from a given field (snapshot) stays in the type it comes in.

A sweep's result is a Markov chain state: a replay in 64 bits takes another decision wherever a trial lies within
FP32 rounding of its threshold, and is another chain from there on. exact() therefore has values for the network
training and for the snapshot, and None for the chains.
"""
import math

import numpy as np
import torch

import mclics_b200 as M
from mclics_b200 import learned

FRANK = (1.0, 0.5, 1.5)          # K11 : K22 : K33 of the GHRL slab and droplet
CHIRAL = (1.48, 1.0, 2.28, 12.0)  # ... of the cholesteric, pitch 12 sites
SAMPLES = 166667                  # training samples per replica and state


def listed():
    return [
        # the smallest call: a 32^3 Lebwohl-Lasher lattice stepped by a caller that reads every record
        dict(name="ll_32_step", kind="step", model="ll", nx=32, ny=32, nz=32, geometry="bulk", px=1, py=1, pz=1, T=1.1),
        # one temperature of the 32^3 phase-transition scan
        dict(name="ll_32_scan", kind="scan", model="ll", nx=32, ny=32, nz=32, geometry="bulk", px=1, py=1, pz=1, T=1.1,
             therm=100, meas=200),
        # many lattices of uneven sizes over a range of temperatures (finite-size scaling): 64 replicas, 16^3 to 128^3
        dict(name="ll_batch_64", kind="batch", model="ll", replicas=64, lo=16, hi=128, blocks=8, meas=10),
        # the default benchmark lattice: GHRL slab of 256^3 between homeotropic plates
        dict(name="ghrl_slab_256", kind="scan", model="ghrl", nx=256, ny=256, nz=256, geometry="slab", px=1, py=1, pz=0,
             T=0.8, therm=200, meas=400),
        # a cholesteric in a box with free faces and a field: odd sizes, chiral term
        dict(name="chiral_box", kind="scan", model="chiral", nx=101, ny=75, nz=50, geometry="bulk", px=0, py=0, pz=0,
             T=0.4, therm=50, meas=50),
        # a nematic droplet with homeotropic anchoring (point types: sphere geometry)
        dict(name="droplet_64", kind="scan", model="ghrl", nx=64, ny=64, nz=64, geometry="sphere", px=0, py=0, pz=0,
             T=0.6, therm=50, meas=50),
        # the electric-field series of pear-shaped molecules: 32 slabs of 256 x 256 x 64, one field each; the largest
        dict(name="pear_fields_32", kind="batch", model="pear", replicas=32, lo=256, hi=256, blocks=2, meas=10),
        # the polar order of one such slab, followed sweep by sweep
        dict(name="pear_polar", kind="polar", model="pear", nx=128, ny=128, nz=64, geometry="slab", px=1, py=1, pz=0,
             T=0.5, meas=10),
        # samples for the learned proposal from three 128^3 lattices
        dict(name="ll_128_collect", kind="collect", size=128, replicas=3, gap=10, snapshots=2, samples=SAMPLES),
        # the learned proposal on the same lattices
        dict(name="ll_128_learned", kind="learned", size=128, replicas=3, therm=5, meas=15),
        # its training: mini-batches of the default size
        dict(name="train_8192", kind="train", batch=8192, steps=16),
        # a snapshot of a pear slab
        dict(name="pear_snapshot", kind="snapshot", nx=256, ny=256, nz=64, px=1, py=1, pz=0),
    ]


def _size(rng, lo, hi, even=False):
    n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return n + (n & 1) if even else n


def draw(rng):
    kind = rng.choice(["step", "scan", "scan", "scan", "batch", "batch", "polar", "collect", "learned", "train", "snapshot"])
    if kind in ("step", "scan", "polar"):
        geometry = "slab" if kind == "polar" else rng.choice(["bulk", "slab", "sphere"])
        model = "pear" if kind == "polar" else rng.choice(["ll", "ghrl", "chiral", "pear"])
        if geometry == "sphere":
            nx = ny = nz = _size(rng, 16, 160)
            px = py = pz = 0
        else:
            px, py, pz = (int(rng.random() < 0.7) for _ in range(3))
            nx, ny, nz = (_size(rng, 12, 224, p) for p in (px, py, pz))
            pz = 0 if geometry == "slab" else pz
        c = dict(kind=kind, model=model, nx=nx, ny=ny, nz=nz, geometry=geometry, px=px, py=py, pz=pz,
                 T=round(rng.uniform(0.3, 1.2), 3))
        if kind == "scan":
            c.update(therm=_size(rng, 10, 100), meas=_size(rng, 10, 100))
        elif kind == "polar":
            c.update(meas=_size(rng, 4, 16))
        return c
    if kind == "batch":
        pear = rng.random() < 0.3
        lo = _size(rng, 16, 64, True)
        return dict(kind=kind, model="pear" if pear else "ll", replicas=_size(rng, 2, 64), lo=lo,
                    hi=lo if pear else _size(rng, lo, 128, True), blocks=_size(rng, 1, 4), meas=_size(rng, 1, 16))
    if kind == "collect":
        return dict(kind=kind, size=_size(rng, 16, 128, True), replicas=_size(rng, 1, 4), gap=_size(rng, 2, 16),
                    snapshots=_size(rng, 1, 4), samples=_size(rng, 4096, SAMPLES))
    if kind == "learned":
        return dict(kind=kind, size=_size(rng, 16, 144, True), replicas=_size(rng, 1, 4), therm=_size(rng, 1, 8),
                    meas=_size(rng, 4, 16))
    if kind == "train":
        return dict(kind=kind, batch=_size(rng, 256, 32768), steps=_size(rng, 4, 24))
    px, py, pz = (int(rng.random() < 0.7) for _ in range(3))
    return dict(kind=kind, nx=_size(rng, 12, 256, px), ny=_size(rng, 12, 256, py), nz=_size(rng, 12, 128, pz), px=px,
                py=py, pz=0)


# ---- models and lattices -----------------------------------------------------------------------------------------
def _model(name, geometry):
    """The physics of a case; a slab has two plates, a sphere one surface."""
    n_surf = {"bulk": 0, "slab": 2, "sphere": 1}[geometry]
    if name == "ll":
        return M.Model("ll", surfaces=[("homeotropic", 1.0, 0, 0)] * n_surf)
    if name == "ghrl":
        return M.Model("ghrl", k=FRANK, surfaces=[("homeotropic", 1.5, 0, 0)] * n_surf)
    if name == "chiral":
        return M.Model("ghrl", k=CHIRAL, field_dir=(0.0, 0.0, 1.0), elecA=0.1,
                       surfaces=[("rp_ghrl", 1.0, 90, 30)] * n_surf)
    return M.Model("pear", field_dir=(0.0, 0.0, 1.0), elecP=1.0, surfaces=[("fg", 1.0, 0, 0)] * n_surf)


def _batch_sizes(c):
    """Replica shapes of a batch: cubes over [lo, hi] evenly in the logarithm, or the pear slabs lo x lo x lo / 4."""
    if c["model"] == "pear":
        return [(c["lo"], c["lo"], max(2, c["lo"] // 4))] * c["replicas"]
    n, out = c["replicas"], []
    for i in range(n):
        f = i / max(1, n - 1)
        L = 2 * round(math.exp(math.log(c["lo"]) + f * (math.log(c["hi"]) - math.log(c["lo"]))) / 2)
        out.append((L, L, L))
    return out


def _temperatures(c):
    """LL: evenly across the transition; pear: one temperature."""
    n = c["replicas"]
    if c["model"] == "pear":
        return np.full(n, 0.5, np.float32)
    return np.linspace(1.0, 1.2, n).astype(np.float32) if n > 1 else np.array([1.1], np.float32)


def _ll_cubes(c, seed):
    L, Ts = c["size"], (0.3, 0.8, 1.12, 1.0)
    e = M.Engine(M.Model("ll"), [M.Replica(L, L, L, T=Ts[r], seed=seed + r) for r in range(c["replicas"])])
    for r in range(c["replicas"]):
        e.random_directors(r, seed + 1000 + r)
    return e


def _records(rec):
    """The columns a program keeps of a series (the director is the eigenvector of q)."""
    return {k: np.asarray(rec[k], np.float32) for k in ("energy", "q", "S", "nsum", "acceptance", "ang_var")}


# ---- training data: sites of ordered neighbourhoods, made without the library --------------------------------------
def _samples(n, seed):
    """Rows as Engine.extract_samples gives them: each site and its six neighbours scatter about a local axis, more at
    the higher of three temperatures. Float32 on the host."""
    rng = np.random.default_rng(seed)
    T = np.array([0.3, 0.8, 1.12])[rng.integers(0, 3, n)]
    axis = rng.normal(size=(n, 1, 3))
    axis /= np.linalg.norm(axis, axis=2, keepdims=True)
    v = axis + (0.45 * np.sqrt(T))[:, None, None] * rng.normal(size=(n, 7, 3))
    v /= np.linalg.norm(v, axis=2, keepdims=True)
    nb = v[:, 1:]
    f = np.zeros((n, 8), np.float32)
    for k, (a, b) in enumerate(((0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2))):
        f[:, k] = (1.5 * (nb[:, :, a] * nb[:, :, b]).sum(1) - (3.0 if a == b else 0.0)) / 6.0
    f[:, 6] = T
    f[:, 7] = 1.0
    return f, v[:, 0].astype(np.float32)


def _weights(seed):
    """Weights of a proposal network trained for a while on such samples (in torch, 64 bits, then on the grid of 1/256,
    so that the same seed gives the same weights everywhere)."""
    f, d = _samples(4096, seed)
    x, n = torch.from_numpy(f[:, :7]).double().cuda(), torch.from_numpy(d).double().cuda()
    p = torch.from_numpy(learned.init_params(seed % 1000)).double().cuda()
    m, v = torch.zeros_like(p), torch.zeros_like(p)
    for i in range(60):
        p.requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = _unpack(p)
        h = torch.nn.functional.silu(x @ w1.T + b1)
        h = torch.nn.functional.silu(h @ w2.T + b2)
        (g,) = torch.autograd.grad(_loss(h @ w3.T + b3, n).mean(), p)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p.detach() - 0.02 * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
    return (torch.round(p * 256) / 256).float().cpu().numpy()


def _unpack(p):
    out, o = [], 0
    for shape in ((64, 7), (64,), (64, 64), (64,), (4, 64), (4,)):
        m = math.prod(shape)
        out.append(p[o:o + m].reshape(shape))
        o += m
    return out


def _loss(o, n, kappa_max=500.0):
    """-log(4 pi q(n)) per sample: antipodal von Mises-Fisher about o[:3] with kappa = softplus(o[3]), 5 % uniform."""
    mu = o[:, :3] / o[:, :3].norm(dim=1, keepdim=True)
    kappa = torch.nn.functional.softplus(o[:, 3]).clamp(1e-3, kappa_max)
    t = (mu * n).sum(1).abs()
    g = kappa * (torch.exp(kappa * (t - 1)) + torch.exp(-kappa * (t + 1))) / (-torch.expm1(-2 * kappa))
    return -torch.log(0.95 * g + 0.05)


# ---- a given field for the snapshot --------------------------------------------------------------------------------
def _field(c, seed):
    """Directors of a splayed texture with thermal noise, float32, 3 per site, x fastest (on the host)."""
    rng = np.random.default_rng(seed)
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    x = np.arange(nx, dtype=np.float32)[None, None, :]
    y = np.arange(ny, dtype=np.float32)[None, :, None]
    z = np.arange(nz, dtype=np.float32)[:, None, None]
    n = rng.standard_normal((nz, ny, nx, 3), dtype=np.float32)
    n *= np.float32(0.35)
    n[..., 0] += np.float32(0.4) * np.sin(2 * np.pi * (x / nx + z / nz)).astype(np.float32)
    n[..., 1] += np.float32(0.3) * np.cos(2 * np.pi * y / ny).astype(np.float32)
    n[..., 2] += 1
    n /= np.sqrt((n * n).sum(-1, keepdims=True))
    return n.reshape(-1)


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind in ("step", "scan", "polar"):
        rep = M.Replica(c["nx"], c["ny"], c["nz"], c["geometry"], (c["px"], c["py"], c["pz"]), T=c["T"], seed=seed)
        e = M.Engine(_model(c["model"], c["geometry"]), [rep])
        e.random_directors(0, seed)
        if kind == "step":
            e.set_graphs(True)
            return dict(c, engine=e, T=np.array([c["T"]], np.float32), out=np.zeros(1, M.OBS_DTYPE))
        e.reserve_series(c["meas"])
        return dict(c, engine=e)
    if kind == "batch":
        sizes, T = _batch_sizes(c), _temperatures(c)
        pear = c["model"] == "pear"
        reps = [M.Replica(*s, "slab" if pear else "bulk", (1, 1, 0) if pear else (1, 1, 1), T=float(T[r]),
                          elecE=2.0 * r / max(1, len(sizes) - 1) if pear else 1.0, seed=seed + r)
                for r, s in enumerate(sizes)]
        e = M.Engine(_model(c["model"], "slab" if pear else "bulk"), reps)
        for r in range(len(sizes)):
            e.random_directors(r, seed + 1000 + r)
        e.reserve_series(c["blocks"] * c["meas"])
        e.set_graphs(True)
        return dict(c, engine=e, T=T, out=np.zeros(c["meas"] * len(sizes), M.OBS_DTYPE))
    if kind == "collect":
        return dict(c, engine=_ll_cubes(c, seed), seed=seed)
    if kind == "learned":
        e = _ll_cubes(c, seed)
        e.sweeps(20)  # the learned arm starts from a state of the plain sweep
        e.set_proposal(_weights(seed))
        e.reserve_series(c["meas"])
        return dict(c, engine=e)
    if kind == "train":
        f, d = _samples(c["batch"] * c["steps"], seed)
        f, d = torch.from_numpy(f).cuda(), torch.from_numpy(d).cuda()
        return dict(c, trainer=M.Trainer(learned.init_params(seed % 1000), c["batch"]), features=f, directors=d)
    rep = M.Replica(c["nx"], c["ny"], c["nz"], "slab", (c["px"], c["py"], 0), T=0.5, elecE=1.0, seed=seed)
    e = M.Engine(_model("pear", "slab"), [rep])
    e.upload(0, _field(c, seed))
    return dict(c, engine=e)


def run(state):
    kind = state["kind"]
    if kind == "train":
        t, b = state["trainer"], state["batch"]
        losses = []
        for i in range(state["steps"]):
            f, d = state["features"][i * b:(i + 1) * b], state["directors"][i * b:(i + 1) * b]
            losses.append(t.step(f.data_ptr(), d.data_ptr(), b, 3e-3))
        return {"losses": np.array(losses, np.float32), "params": t.params()}
    e = state["engine"]
    if kind == "step":
        return _records(e.sweeps_io(1, state["T"], state["out"]))
    if kind == "scan":
        e.set_temperature(state["T"])
        e.sweeps(state["therm"])
        e.clear_series()
        e.sweeps(state["meas"], measure=True)
        return {"series": _records(e.series(0)), "directors": e.download(0)}
    if kind == "batch":
        e.clear_series()
        return [_records(e.sweeps_io(state["meas"], state["T"], state["out"])) for _ in range(state["blocks"])]
    if kind == "polar":
        e.clear_series()
        columns, records = [], []
        for s in range(state["meas"]):
            e.sweeps(1, measure=True)
            rec = e.series(0, s, 1)
            x = e.measure_extras(0, rec[0]["director"])
            records.append(rec)
            columns.append([x[k] for k in sorted(x)])
        return {"series": _records(np.concatenate(records)), "extras": np.array(columns, np.float32),
                "directors": e.download(0)}
    if kind == "collect":
        return list(learned.collect(e, state["snapshots"], state["gap"], state["samples"], seed=state["seed"] % 1000))
    if kind == "learned":
        e.sweeps(state["therm"])
        e.clear_series()
        e.sweeps(state["meas"], measure=True)
        return {"series": [_records(e.series(r)) for r in range(e.n)], "directors": e.download(0)}
    o = e.measure(0)
    x = e.measure_extras(0, o["director"])
    return {"energy": float(o["energy"]), "q": np.array(o["q"]), "S": float(o["S"]), "nsum": np.array(o["nsum"]),
            "extras": np.array([x[k] for k in sorted(x)]), "local_order": e.local_order(0), "directors": e.download(0)}


# ---- work ----------------------------------------------------------------------------------------------------------
# Floating-point operations of one site update: six bonds for the old and the trial director and the trial itself.
UPDATE_FLOPS = {"ll": 160, "ghrl": 370, "chiral": 480, "pear": 560}


def _droplet_share(n):
    """Share of a sphere replica's sites that are not empty."""
    return min(1.0, 4.0 / 3.0 * math.pi * (n // 2 + 1) ** 3 / n ** 3)


def work(case):
    c, kind = case, case["kind"]
    if kind == "train":
        n = c["batch"] * c["steps"]
        return {"bytes": n * 44 + 2 * 4 * M.N_MLP_PARAMS, "flops": 6 * 4800 * n}
    if kind == "snapshot":
        n = c["nx"] * c["ny"] * c["nz"]
        return {"bytes": n * (12 + 12 + 4), "flops": 400 * n}
    if kind in ("collect", "learned"):
        n = c["replicas"] * c["size"] ** 3
        if kind == "collect":
            rows = c["snapshots"] * c["replicas"] * c["samples"]
            s = c["gap"] * c["snapshots"]
            return {"bytes": 24 * n * s + 44 * rows, "flops": (UPDATE_FLOPS["ll"] * n * s) + 90 * rows}
        s = c["therm"] + c["meas"]
        return {"bytes": 24 * n * s, "flops": (UPDATE_FLOPS["ll"] + 2 * 4800 + 200) * n * s}
    if kind == "batch":
        n = sum(x * y * z for x, y, z in _batch_sizes(c))
        s = c["blocks"] * c["meas"]
    else:
        n = c["nx"] * c["ny"] * c["nz"] * (_droplet_share(c["nx"]) if c["geometry"] == "sphere" else 1.0)
        s = c.get("therm", 0) + c.get("meas", 1)
    return {"bytes": 24 * n * s, "flops": UPDATE_FLOPS[c["model"]] * n * s}


# ---- the same in 64 bits -------------------------------------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "snapshot":
        return _exact_snapshot(case, seed)
    return None


def _bf16(x):
    """The nearest BF16 value (the network's weights, inputs and activations are BF16 by definition); gradients pass."""
    return x + (x.detach().to(torch.float32).to(torch.bfloat16).to(torch.float64) - x.detach())


class _Silu(torch.autograd.Function):
    """SiLU rounded to BF16, with the derivative of the unrounded function."""

    @staticmethod
    def forward(ctx, z):
        ctx.save_for_backward(z)
        return (z * torch.sigmoid(z)).to(torch.float32).to(torch.bfloat16).to(torch.float64)

    @staticmethod
    def backward(ctx, g):
        (z,) = ctx.saved_tensors
        s = torch.sigmoid(z)
        return g * s * (1 + z * (1 - s))


def _exact_train(c, seed):
    f, d = _samples(c["batch"] * c["steps"], seed)
    x, n = _bf16(torch.from_numpy(f[:, :7]).double()), torch.from_numpy(d).double()
    p = torch.from_numpy(learned.init_params(seed % 1000)).double()
    m, v, losses = torch.zeros_like(p), torch.zeros_like(p), []
    for i in range(c["steps"]):
        p = p.detach().requires_grad_(True)
        w1, b1, w2, b2, w3, b3 = _unpack(p)
        rows = slice(i * c["batch"], (i + 1) * c["batch"])
        h = _Silu.apply(x[rows] @ _bf16(w1).T + b1)
        h = _Silu.apply(h @ _bf16(w2).T + b2)
        loss = _loss(h @ _bf16(w3).T + b3, n[rows]).mean()
        (g,) = torch.autograd.grad(loss, p)
        m, v = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g
        p = p.detach() - 3e-3 * (m / (1 - 0.9 ** (i + 1))) / ((v / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
        losses.append(loss.item())
    return {"losses": np.array(losses), "params": p.numpy()}


def _shifted(n, axis, step, periodic):
    """Neighbours at +step along an array axis, and which exist."""
    nb = torch.roll(n, -step, dims=axis)
    there = torch.ones(n.shape[:3], dtype=torch.bool, device=n.device)
    if not periodic:
        there.select(axis, n.shape[axis] - 1 if step > 0 else 0).fill_(False)
    return nb, there.double()


def _exact_snapshot(c, seed):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    where = "cuda" if torch.cuda.is_available() else "cpu"
    host = _field(c, seed)
    n = torch.from_numpy(host).to(where).double().reshape(nz, ny, nx, 3)
    N = nx * ny * nz
    A, B1, C = 1.0, float(np.float32(0.04)), float(np.float32(0.3))
    energy = torch.zeros((), dtype=torch.float64, device=where)
    splay = torch.zeros(3, dtype=torch.float64, device=where)
    bonds, div = 0.0, torch.zeros(n.shape[:3], dtype=torch.float64, device=where)
    local = 1.5 * n[..., :, None] * n[..., None, :]
    points = torch.ones(n.shape[:3], dtype=torch.float64, device=where)
    for a, periodic in ((0, c["px"]), (1, c["py"]), (2, 0)):
        step_div, step_count = torch.zeros_like(div), torch.zeros_like(div)
        for s in (1, -1):
            m, w = _shifted(n, 2 - a, s, periodic)
            b = (n * m).sum(-1)
            ra, rb = s * n[..., a], s * m[..., a]
            energy += (w * (-A * b * b - B1 * b - 0.25 * C * (1 + b) ** 2 * (rb - ra))).sum()
            term = m * rb[..., None] - n * ra[..., None] + n * (b * rb)[..., None] - m * (b * ra)[..., None]
            splay += 0.5 * (w[..., None] * term).sum((0, 1, 2))
            bonds += float(w.sum())
            step_div += w * s * (m[..., a] - n[..., a])
            step_count += w
            local += w[..., None, None] * 1.5 * m[..., :, None] * m[..., None, :]
            points += w
        div += torch.where(step_count > 0, step_div / step_count.clamp(min=1), step_div)
    energy += (-1.0 * n[..., 2]).sum() + (n[0, ..., 2] ** 2).sum()
    if nz > 1:
        energy += (n[-1, ..., 2] ** 2).sum()
    q = 1.5 * torch.einsum("zyxa,zyxb->ab", n, n) / N - 0.5 * torch.eye(3, dtype=torch.float64, device=where)
    vals, vecs = torch.linalg.eigh(q)
    axes = [torch.arange(k, device=where).double() - k // 2 for k in (nz, ny, nx)]
    r = torch.stack(torch.meshgrid(*axes, indexing="ij")[::-1], -1)
    radial = {}
    for name, keep in (("cyl", (1.0, 1.0, 0.0)), ("sph", (1.0, 1.0, 1.0))):
        v = r * torch.tensor(keep, dtype=torch.float64, device=where)
        length = v.norm(dim=-1)
        far = length >= 0.5
        cosine = ((n * v).sum(-1) / length.clamp(min=0.5))[far]
        radial["Pr_" + name] = float(cosine.mean()) if cosine.numel() else 0.0
        radial["Sr_" + name] = float((1.5 * cosine * cosine - 0.5).mean()) if cosine.numel() else 0.0
    extras = {"P": float((n.sum((0, 1, 2)) * vecs[:, 2]).sum().abs()) / N, "dtheta": 1.5 * float(splay.norm()) / bonds,
              "divn": float(div.mean()), **radial}
    # largest eigenvalue of the traceless symmetric local tensor: the trigonometric root of its cubic
    local = local / points[..., None, None] - 0.5 * torch.eye(3, dtype=torch.float64, device=where)
    p2 = ((local * local).sum((-1, -2)) / 6).clamp(min=1e-300).sqrt()
    angle = torch.acos((torch.linalg.det(local / p2[..., None, None]) / 2).clamp(-1, 1)) / 3
    return {"energy": float(energy) / N, "q": torch.stack([q[0, 0], q[0, 1], q[0, 2], q[1, 1], q[1, 2], q[2, 2]]).cpu().numpy(),
            "S": float(vals[2]), "nsum": n.sum((0, 1, 2)).cpu().numpy(),
            "extras": np.array([extras[k] for k in sorted(extras)]),
            "local_order": (2 * p2 * torch.cos(angle)).cpu().numpy().reshape(-1), "directors": host.astype(np.float64)}
