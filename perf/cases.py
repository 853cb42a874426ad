"""The work that users of this package have it do, as timed cases.

A case is a dict of plain values.  ``prepare`` makes what a program has in
hand before the call (models on the device, points, plans), ``run`` is one
pass through the public entry points, ``exact`` the same result in 64 bits
with plain torch, ``work`` the bytes and operations a pass cannot do without.

Kinds:

* ``query``    ``SIREN.forward`` under ``no_grad``: the signed distance at a
               list of points (a picking or collision query of a few hundred
               points, a chunk of 64^3 points, a large ragged list);
* ``normals``  ``level_gradient``: value and gradient at a point list (mesh
               normals, hit points);
* ``volume``   one level over a whole N^3 grid (``create_mesh``'s sampling);
* ``recon``    the three nested levels with their bands over an N^3 grid and
               marching cubes (``reconstruct.py --multistage``);
* ``train``    ``ResidualTrainer.step``: the fine trainer's step on a batch of
               surface, offset and dithered rows;
* ``autograd`` the reference trainers' own loop body on a ``SIREN`` level:
               forward, create_graph gradient, loss, backward;
* ``frame``    one sphere-traced frame with normals and shading;
* ``batch``    many levels of many models in one call (serving);
* ``deltas``   ``calc_deltas`` over a mesh's vertices (training preparation).
"""

from __future__ import annotations

import functools
import math
import os
import random

import numpy as np
import torch
import torch.nn.functional as F

from mplicits_gb300 import synthetic
from mplicits_gb300.batch import BatchedLevels, BatchEntry
from mplicits_gb300.grad import level_gradient
from mplicits_gb300.meshing import BandedReconstruction
from mplicits_gb300.model import SIREN
from mplicits_gb300.scene import RaycastingScene, calc_deltas
from mplicits_gb300.trace import SphereTracer, orbit_cameras
from mplicits_gb300.train import ResidualTrainer, create_training_data_on_neighborhood

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OMEGA = 30.0
DEV = "cuda"


def listed():
    return [
        # a handful of points (picking, collision): the call's latency
        {"name": "query_500_fp32", "kind": "query", "points": 500, "width": 256,
         "precision": "fp32"},
        # one chunk of the reference's sampling loops (max_batch = 64^3), default precision
        {"name": "query_chunk_fp32", "kind": "query", "points": 64 ** 3, "width": 256,
         "precision": "fp32"},
        # normals of a mesh's vertices, a ragged count
        {"name": "normals_fp16", "kind": "normals", "points": 1000003, "width": 256,
         "precision": "fp16"},
        # create_mesh's sampling at its default resolution and precision
        {"name": "volume_256_fp32", "kind": "volume", "N": 256, "width": 256,
         "precision": "fp32"},
        # the headline reconstruction
        {"name": "recon_512_fp16", "kind": "recon", "N": 512, "precision": "fp16",
         "delta0": 0.05, "delta1": 0.01},
        # a preview mesh on an odd grid
        {"name": "recon_101_bf16", "kind": "recon", "N": 101, "precision": "bf16",
         "delta0": 0.05, "delta1": 0.01},
        # the fine trainer's step at the benchmark's batch, tensor cores
        {"name": "train_65536_bf16", "kind": "train", "samples": 65536, "precision": "bf16"},
        # the same step at the default precision and a small batch
        {"name": "train_5000_fp32", "kind": "train", "samples": 5000, "precision": "fp32"},
        # the reference trainers' loop body through autograd
        {"name": "autograd_6000_fp32", "kind": "autograd", "points": 6000},
        # one full-HD frame
        {"name": "frame_1080p_bf16", "kind": "frame", "width": 1920, "height": 1080,
         "camera": 0, "precision": "bf16"},
        # 64 three-level models, point lists of 1e4 to 2e6
        {"name": "batch_64_bf16", "kind": "batch", "models": 64, "layout": 11, "most": 2000000,
         "precision": "bf16"},
        # the neighbourhood radii of a 523,266-vertex mesh
        {"name": "deltas_512", "kind": "deltas", "rings": 512},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "normals", "volume", "recon", "train", "train",
                       "autograd", "frame", "batch", "deltas"])
    if kind == "query":
        return {"kind": kind, "points": _log(rng, 1, 2000000),
                "width": rng.choice([64, 128, 256, 256]),
                "precision": rng.choice(["fp32", "fp32", "fp16", "bf16"])}
    if kind == "normals":
        return {"kind": kind, "points": _log(rng, 100, 1500000),
                "width": rng.choice([64, 128, 256, 256]),
                "precision": rng.choice(["fp32", "fp16", "bf16"])}
    if kind == "volume":
        return {"kind": kind, "N": _log(rng, 32, 256), "width": rng.choice([64, 128, 256]),
                "precision": rng.choice(["fp32", "fp16", "bf16"])}
    if kind == "recon":
        return {"kind": kind, "N": _log(rng, 48, 512), "precision": rng.choice(["fp16", "bf16"]),
                "delta0": round(rng.uniform(0.03, 0.08), 4),
                "delta1": round(rng.uniform(0.006, 0.02), 4)}
    if kind == "train":
        return {"kind": kind, "samples": _log(rng, 500, 65536),
                "precision": rng.choice(["bf16", "fp32"])}
    if kind == "autograd":
        return {"kind": kind, "points": _log(rng, 200, 30000)}
    if kind == "frame":
        h = _log(rng, 120, 1080)
        return {"kind": kind, "width": int(h * rng.choice([1.0, 4 / 3, 16 / 9])), "height": h,
                "camera": rng.randrange(8), "precision": rng.choice(["bf16", "fp16"])}
    if kind == "batch":
        return {"kind": kind, "models": rng.randrange(2, 65), "layout": rng.randrange(1000),
                "most": _log(rng, 20000, 2000000), "precision": rng.choice(["bf16", "fp16"])}
    return {"kind": kind, "rings": _log(rng, 16, 512)}


# -- models and inputs ---------------------------------------------------

@functools.lru_cache(maxsize=1)
def _trained():
    """The trained three-level model of the synthetic surface (256 wide)."""
    d = np.load(os.path.join(ROOT, "tests", "golden", "three_level_sphere.npz"))
    return [{k[3:]: d[k] for k in d.files if k.startswith(f"L{i}.")} for i in range(3)]


def _rotation(seed):
    q, r = np.linalg.qr(np.random.RandomState(seed % (1 << 32)).normal(size=(3, 3)))
    q = q * np.sign(np.diag(r))
    if np.linalg.det(q) < 0:
        q[:, 0] = -q[:, 0]
    return q


def _levels(seed, precision, which=(0, 1, 2)):
    """The trained levels seen from a seeded rotation of space: f(R x)."""
    R = _rotation(seed)
    out = []
    for i in which:
        sd = dict(_trained()[i])
        sd["net.0.0.weight"] = (sd["net.0.0.weight"].astype(np.float64) @ R).astype(np.float32)
        m = SIREN(3, 1, [256] * 3, w0=30, delay_init=True, precision=precision)
        m.load_state_dict({k: torch.from_numpy(v) for k, v in sd.items()})
        out.append(m.to(DEV).eval())
    return out


def _rescaled(levels, seed):
    """The same surface from other weights: seeded sign flips of hidden units
    (sin is odd) and a power-of-two scale of the output, so that the values
    change and the mesh keeps its vertex and face counts.  Returns the scale."""
    rng = np.random.RandomState(seed % (1 << 32))
    scale = 2.0 ** (seed % 16 - 8)
    for m in levels:
        lins = m.linears()
        with torch.no_grad():
            for a, b in zip(lins[:-1], lins[1:]):
                s = torch.from_numpy(rng.choice([-1.0, 1.0], a.out_features)).float().to(DEV)
                a.weight.mul_(s[:, None])
                a.bias.mul_(s)
                b.weight.mul_(s)
            lins[-1].weight.mul_(scale)
            lins[-1].bias.mul_(scale)
    return scale


def _random_level(width, seed, precision):
    """A freshly initialised level (the reference's init)."""
    with torch.random.fork_rng(devices=[]):
        torch.manual_seed(seed)
        return SIREN(3, 1, [width] * 3, w0=30, precision=precision).to(DEV).eval()


def _level(case, seed):
    if case["width"] == 256:
        return _levels(seed, case["precision"], (0,))[0]
    return _random_level(case["width"], seed, case["precision"])


def _generator(seed):
    return torch.Generator(DEV).manual_seed(seed)


def _points(n, seed):
    """Half uniform in the cube, half near the surface's mean radius."""
    g = _generator(seed)
    x = torch.rand(n, 3, device=DEV, generator=g) * 2 - 1
    h = n // 2
    r = torch.randn(h, 3, device=DEV, generator=g)
    r = r / r.norm(dim=1, keepdim=True).clamp_min(1e-6)
    x[:h] = r * (synthetic.R0 + 0.05 * torch.randn(h, 1, device=DEV, generator=g))
    return x


def _surface(n, seed):
    """n rows (xyz, normal) of the synthetic surface, rotated as the levels."""
    pts, nrm = synthetic.surface_points(n, np.random.default_rng(seed), noise=0.002)
    R = _rotation(seed)
    rows = np.concatenate([pts.astype(np.float64) @ R, nrm.astype(np.float64) @ R], 1)
    return torch.from_numpy(rows.astype(np.float32)).to(DEV)


def _train_rows(samples, seed):
    rows = _surface(samples, seed)
    return create_training_data_on_neighborhood(rows, samples, device=DEV, delta=0.01,
                                                seed=seed)["on_surf"]


def _batch_layout(case):
    """(width, three nested list sizes) of every model."""
    r = random.Random(case["layout"])
    lo, hi = math.log(1e4), math.log(case["most"])
    return [(r.choice([128, 256]),
             sorted((int(math.exp(r.uniform(lo, hi))) for _ in range(3)), reverse=True))
            for _ in range(case["models"])]


def _mesh(rings, seed):
    """The triangulated surface, rotated, with 2% of an edge of vertex noise."""
    pos, nrm, faces = synthetic.surface_mesh(rings, 2 * rings)
    R = _rotation(seed)
    rng = np.random.default_rng(seed)
    noise = rng.standard_normal(pos.shape, dtype=np.float32) * (0.02 * math.pi * 0.6 / rings)
    pos = (pos.astype(np.float64) @ R).astype(np.float32) + noise
    return pos, (nrm.astype(np.float64) @ R).astype(np.float32), faces


# -- one case --------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("query", "normals"):
        s["model"], s["x"] = _level(case, seed), _points(case["points"], seed)
    elif kind == "volume":
        s["rec"] = BandedReconstruction([_level(case, seed)], [], case["N"], DEV)
    elif kind == "recon":
        levels = _levels(0, case["precision"])
        scale = _rescaled(levels, seed)
        s["deltas"] = [case["delta0"] * scale, case["delta1"] * scale]
        s["rec"] = BandedReconstruction(levels, s["deltas"], case["N"], DEV)
    elif kind == "train":
        frozen = _levels(seed, case["precision"], (0, 1))
        fine = _random_level(256, seed, case["precision"]).train()
        s["trainer"] = ResidualTrainer(fine, frozen, lr=1e-4, precision=case["precision"])
        s["rows"] = _train_rows(case["samples"], seed)
    elif kind == "autograd":
        s["levels"] = _levels(seed, "fp32", (0, 1)) + [_random_level(256, seed, "fp32").train()]
        for m in s["levels"][:2]:
            m.requires_grad_(False)
        x, n, d = _train_rows((case["points"] + 2) // 3, seed)
        s["rows"] = (x[:case["points"]], n[:case["points"]], d[:case["points"], None])
    elif kind == "frame":
        s["tracer"] = SphereTracer(_levels(seed, case["precision"]), [0.05, 0.01], case["width"],
                                   case["height"], max_steps=96, eps=1e-4,
                                   precision=case["precision"], tail_from=32)
        s["camera"] = orbit_cameras(width=case["width"], height=case["height"])[case["camera"]]
    elif kind == "batch":
        layout = _batch_layout(case)
        g = _generator(seed)
        s["S"] = torch.zeros(3 * sum(sizes[0] for _, sizes in layout), device=DEV)
        entries, at = [], 0
        for i, (width, sizes) in enumerate(layout):
            x = torch.rand(sizes[0], 3, device=DEV, generator=g) * 2 - 1
            perm = torch.randperm(sizes[0], device=DEV, generator=g).to(torch.int32)
            for lv in range(3):
                m = _random_level(width, seed * 1000 + 3 * i + lv, case["precision"])
                idx = None if lv == 0 else perm[:sizes[lv]].contiguous()
                entries.append(BatchEntry(m, s["S"][at:at + sizes[0]], x=x, index=idx,
                                          n=sizes[lv]))
                at += sizes[0]
        s["plan"] = BatchedLevels(entries, case["precision"])
        s["plan"].autotune()
        s["plan"].capture()
    else:
        pos, nrm, faces = _mesh(case["rings"], seed)
        pos, nrm = torch.from_numpy(pos).to(DEV), torch.from_numpy(nrm).to(DEV)
        s["scene"] = RaycastingScene(pos, torch.from_numpy(faces).to(DEV), device=DEV)
        s["rows"] = torch.cat([pos, nrm], 1)
    return s


def _gradient(y, x):
    return torch.autograd.grad(y, [x], grad_outputs=torch.ones_like(y), create_graph=True)[0]


def _residual_loss(pred, grad, frozen, normals, sdf):
    """loss_add_detail_fine from the level's output and gradient and the
    frozen levels' (output, gradient) pairs."""
    S, G = pred, grad
    for f, g in frozen:
        S, G = S + f, G + g.detach()
    on = sdf != -1
    sdf_c = torch.where(on, (sdf - S) ** 2, torch.zeros_like(S))
    nrm_c = torch.where(on, 1 - F.cosine_similarity(normals, G, dim=-1)[..., None],
                        torch.zeros_like(S))
    eik = ((G.norm(dim=-1) - 1.0) ** 2).unsqueeze(-1)
    return torch.stack([sdf_c.mean() * 3e3, nrm_c.mean() * 1e2, eik.mean() * 5e1])


def _autograd_step(levels, x, normals, sdf):
    fine = levels[2]
    for p in fine.parameters():
        p.grad = None
    out = fine(x)
    grad = _gradient(out["model_out"], out["model_in"])
    frozen = []
    for m in levels[:2]:
        o = m(out["model_in"])
        frozen.append((o["model_out"], _gradient(o["model_out"], o["model_in"])))
    losses = _residual_loss(out["model_out"], grad, frozen, normals, sdf)
    losses.sum().backward()
    return [losses.detach()] + [p.grad for p in fine.parameters()]


def run(state):
    kind = state["kind"]
    if kind == "query":
        with torch.no_grad():
            return state["model"](state["x"])["model_out"]
    if kind == "normals":
        return level_gradient(state["model"], state["x"])
    if kind == "volume":
        return state["rec"].sample()
    if kind == "recon":
        S = state["rec"].sample()
        return (S,) + tuple(state["rec"].mesh())
    if kind == "train":
        t = state["trainer"]
        losses = t.step(*state["rows"])
        return [losses] + t.params + t.exp_avg + t.exp_avg_sq
    if kind == "autograd":
        return _autograd_step(state["levels"], *state["rows"])
    if kind == "frame":
        return state["tracer"].render(state["camera"])
    if kind == "batch":
        state["plan"].replay()
        return state["S"]
    return calc_deltas(state["rows"], state["scene"], 0.05, 100)


# -- work -------------------------------------------------------------------

def _eval_flops(width):
    return 2 * (3 * width + 2 * width * width + width)


# forward and three tangent rows, and the products of the double backward
_TRAIN_FLOPS = (_eval_flops(256) + 3 * 2 * (2 * 256 * 256 + 256) + 2 * (2 * 4 * 2 * 256 * 256))


def work(case):
    kind = case["kind"]
    if kind == "query":
        return {"bytes": 16 * case["points"], "flops": _eval_flops(case["width"]) * case["points"]}
    if kind == "normals":  # the backward sweep costs what the forward one does
        return {"bytes": 28 * case["points"],
                "flops": 2 * _eval_flops(case["width"]) * case["points"]}
    if kind == "volume":
        return {"bytes": 4 * case["N"] ** 3, "flops": _eval_flops(case["width"]) * case["N"] ** 3}
    if kind == "recon":
        shell = 4 * math.pi * synthetic.R0 ** 2 / 8 * 2  # share of the cube per unit of delta
        evals = case["N"] ** 3 * (1 + shell * (case["delta0"] + case["delta1"]))
        crossings = 1.5 * math.pi * (synthetic.R0 * (case["N"] - 1)) ** 2 / 2
        return {"bytes": 8 * case["N"] ** 3 + 52 * crossings, "flops": _eval_flops(256) * evals}
    if kind in ("train", "autograd"):
        rows = 3 * case["samples"] if kind == "train" else case["points"]
        return {"bytes": 28 * rows + 28 * 133000,
                "flops": rows * (_TRAIN_FLOPS + 2 * 2 * _eval_flops(256))}
    if kind == "frame":  # about 60% of the pixels meet the bounding sphere, six steps each
        px = case["width"] * case["height"]
        return {"bytes": 8 * px, "flops": 0.6 * 6 * px * _eval_flops(256)}
    if kind == "batch":
        lay = _batch_layout(case)
        return {"bytes": sum(16 * s for _, sizes in lay for s in sizes),
                "flops": sum(_eval_flops(w) * s for w, sizes in lay for s in sizes)}
    v = case["rings"] * case["rings"] * 2
    return {"bytes": v * (24 + 28) + 2 * v * 12 + 12 * v, "flops": 0}


# -- the same in 64 bits -----------------------------------------------------

def _params64(model):
    return [(blk[0].weight.detach().double(), blk[0].bias.detach().double()) for blk in model.net]


def _forward64(params, x):
    for W, b in params[:-1]:
        x = torch.sin(OMEGA * F.linear(x, W, b))
    return F.linear(x, *params[-1])


def _eval64(model, x, chunk=1 << 18):
    params = _params64(model)
    with torch.no_grad():
        return torch.cat([_forward64(params, c.double()) for c in x.split(chunk)])


def _grid64(N):
    """The sampling grid (i3d/meshing.py:42-63), in its float32 steps."""
    i = torch.arange(N ** 3, device=DEV)
    n = torch.tensor(float(N), device=DEV)
    q = i.float() / n
    vs = torch.tensor(np.float32(2.0 / (N - 1)), device=DEV)
    return torch.stack([torch.fmod(q / n, n), torch.fmod(q, n), (i % N).float()], 1) * vs - 1.0


def _loss64(params, frozen, x, normals, sdf, n):
    """The loss terms of some rows of a batch of n, and their gradients."""
    x = x.double().requires_grad_(True)
    f = _forward64(params, x)
    g = _gradient(f, x)
    with torch.enable_grad():
        fr = []
        for p in frozen:
            y = x.detach().requires_grad_(True)
            o = _forward64(p, y)
            fr.append((o.detach(), torch.autograd.grad(o.sum(), y)[0]))
    losses = _residual_loss(f, g, fr, normals.double(), sdf.double()) * (x.shape[0] / n)
    return losses.detach(), torch.autograd.grad(losses.sum(), [t for wb in params for t in wb])


def _batch64(levels, x, normals, sdf, chunk=1 << 14):
    params = [(W.requires_grad_(True), b.requires_grad_(True)) for W, b in _params64(levels[2])]
    frozen = [_params64(m) for m in levels[:2]]
    total = None
    for i in range(0, x.shape[0], chunk):
        l, g = _loss64(params, frozen, x[i:i + chunk], normals[i:i + chunk], sdf[i:i + chunk],
                       x.shape[0])
        total = [l] + list(g) if total is None else [a + b for a, b in zip(total, [l] + list(g))]
    return total[0], total[1:]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("frame", "deltas"):  # whole numbers; a bisection's float32 path
        return None
    if work(case)["flops"] > 6e12:
        return None
    s = prepare(case, seed)
    if kind == "query":
        return _eval64(s["model"], s["x"])
    if kind == "normals":
        params, f, g = _params64(s["model"]), [], []
        for c in s["x"].split(1 << 17):
            c = c.double().requires_grad_(True)
            y = _forward64(params, c)
            f.append(y.detach()[:, 0])
            g.append(torch.autograd.grad(y.sum(), c)[0])
        return torch.cat(f), torch.cat(g)
    if kind == "volume":
        return _eval64(s["rec"].levels[0], _grid64(case["N"]))[:, 0]
    if kind == "recon":
        x = _grid64(case["N"])
        S = _eval64(s["rec"].levels[0], x)[:, 0]
        band = torch.arange(S.numel(), device=DEV)
        for m, d in zip(s["rec"].levels[1:], s["deltas"]):
            band = band[S[band].abs() < d]
            S[band] += _eval64(m, x[band])[:, 0]
        return S, None, None, None, None
    if kind == "train":
        t = s["trainer"]
        x, n, d = s["rows"]
        losses, grads = _batch64(t.frozen + [t.model], x, n, d[:, None])
        m = [0.1 * g for g in grads]
        v = [0.001 * g * g for g in grads]
        p = [q.detach().double().reshape(g.shape) - 1e-4 * g / (g.abs() + 1e-8)
             for q, g in zip(t.params, grads)]
        return [losses] + p + m + v
    if kind == "autograd":
        losses, grads = _batch64(s["levels"], *s["rows"])
        return [losses] + list(grads)
    S = torch.zeros_like(s["S"], dtype=torch.float64)
    at = 0
    for e in s["plan"].entries:
        n0 = e.x.shape[0]
        part = S[at:at + n0]
        if e.index is None:
            part[:] = _eval64(e.model, e.x)[:, 0]
        else:
            idx = e.index.long()
            part[idx] = _eval64(e.model, e.x[idx])[:, 0]
        at += n0
    return S
