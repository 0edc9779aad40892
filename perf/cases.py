"""The work that programs using this framework have it do, as measurable cases.

Every case goes through a public entry point of ``cuda_knn_aggregate``:

* ``forward``: ``knn_aggregate_aniso`` without gradients (evaluating a field);
* ``train``: the same with the gradients of q, p, f, sigma and R for a given
  gradient of f_out (what a network above the op sends back);
* ``eikonal``: forward, dq with ``create_graph`` and the gradients of the mean
  of (|dq| - 1)^2 (the training step the second order exists for);
* ``lookup``: ``knn_aggregate_aniso_lookup`` with its gradients;
* ``ragged``: ``ragged_forward`` over resident clouds of different sizes, half
  of the segments asking for dq.

``layout`` names the point cloud: ``uniform`` (unit cube, random rotations),
``rand`` (every tensor uniform in [0, 1), as in the reference's usage snippet,
so R is no rotation) and ``surface`` (near a unit sphere, the Gaussians
aligned with the surface, queries around it).
"""
import math
import os
import random
import sys

import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "cuda-knn-aniso-gaussian-feature-aggregation_b200"))

from cuda_knn_aggregate import knn_aggregate_aniso, knn_aggregate_aniso_lookup  # noqa: E402
from cuda_knn_aggregate.ragged import CloudSet, ragged_forward  # noqa: E402

DEVICE = "cuda"
RAGGED_KS = (8, 16, 32)


def _case(name, op, layout, B, Q, P, F, K, dtype="float32"):
    return {"name": name, "op": op, "layout": layout, "B": B, "Q": Q, "P": P, "F": F, "K": K, "dtype": dtype}


def listed():
    return [
        # one evaluation at the size of the reference's usage snippet: launches and latency
        _case("usage_forward", "forward", "uniform", 2, 1000, 500, 32, 12),
        # the usage snippet itself (every tensor torch.rand) as an Eikonal step
        _case("usage_eikonal", "eikonal", "rand", 2, 1000, 500, 32, 12),
        # an ordinary training step at sizes that fit no tile, warp or vector width
        _case("odd_train", "train", "uniform", 3, 5003, 2777, 37, 9),
        # the shape of the reference's timing table: evaluation, first order, second order
        _case("table_forward", "forward", "uniform", 2, 12288, 4096, 64, 16),
        _case("table_train", "train", "uniform", 2, 12288, 4096, 64, 16),
        _case("table_eikonal", "eikonal", "uniform", 2, 12288, 4096, 64, 16),
        # evaluating a large surface cloud with wide features and the largest register list
        _case("surface_forward", "forward", "surface", 1, 65536, 65536, 256, 32),
        # the large single-cloud training step
        _case("sphere_eikonal", "eikonal", "surface", 1, 524288, 131072, 128, 16),
        # many neighbours (smooth fields): K above the register lists
        _case("many_neighbours_train", "train", "uniform", 1, 4096, 4096, 32, 48),
        # double precision (checking a model's gradients)
        _case("double_eikonal", "eikonal", "uniform", 2, 2048, 2048, 32, 12, "float64"),
        # neighbours through a table of the template's neighbours
        _case("lookup_train", "lookup", "uniform", 2, 12288, 4096, 64, 16),
        # one batch of clouds of different sizes, queries, K
        {"name": "ragged_grad", "op": "ragged", "clouds": 24, "P_min": 1024, "P_max": 32768, "Q_min": 2048,
         "Q_max": 65536, "F": 64, "sizes_seed": 1003, "dtype": "float32"},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "train", "train", "eikonal", "eikonal", "lookup", "ragged", "many",
                       "double"])
    if kind == "ragged":
        p0, q0 = _log_int(rng, 300, 8192), _log_int(rng, 256, 8192)
        return {"op": "ragged", "clouds": _log_int(rng, 2, 32), "P_min": p0, "P_max": p0 * rng.randint(1, 4),
                "Q_min": q0, "Q_max": q0 * rng.randint(1, 8), "F": _log_int(rng, 8, 128),
                "sizes_seed": rng.randrange(1 << 20), "dtype": "float32"}
    if kind in ("many", "double"):
        K = _log_int(rng, 33, 64) if kind == "many" else _log_int(rng, 4, 24)
        P = _log_int(rng, 300, 4096)
        Q = min(_log_int(rng, 300, 8192), 16_000_000 // P)
        return {"op": rng.choice(["forward", "train", "eikonal"]), "layout": rng.choice(["uniform", "rand"]), "B": 1,
                "Q": Q, "P": P, "F": _log_int(rng, 4, 64), "K": K,
                "dtype": "float64" if kind == "double" else "float32"}
    if kind == "lookup":
        return {"op": "lookup", "layout": "uniform", "B": rng.randint(1, 3), "Q": _log_int(rng, 500, 20000),
                "P": _log_int(rng, 300, 8192), "F": _log_int(rng, 4, 128), "K": _log_int(rng, 4, 32),
                "dtype": "float32"}
    layout = rng.choice(["uniform", "uniform", "rand", "surface"])
    B = rng.randint(1, 3)
    if layout == "surface":
        Q, P = _log_int(rng, 2000, 100000), _log_int(rng, 2000, 100000)
    elif layout == "uniform":
        Q, P = _log_int(rng, 500, 40000), _log_int(rng, 300, 20000)
    else:
        Q, P = _log_int(rng, 500, 10000), _log_int(rng, 300, 4096)
    return {"op": kind, "layout": layout, "B": B, "Q": Q, "P": P, "F": _log_int(rng, 4, 200), "K": _log_int(rng, 1, 32),
            "dtype": "float32"}


# ------------------------------------------------------------------ inputs


def _gen(seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed(int(seed))
    return g


def _rotations(n, g):
    """Uniform random rotations from normalised Gaussian quaternions."""
    v = torch.randn(n, 4, generator=g, device=DEVICE, dtype=torch.float64)
    w, x, y, z = (v / v.norm(dim=1, keepdim=True)).unbind(1)
    return torch.stack([
        1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
        2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
        2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).reshape(n, 3, 3)


def _directions(n, g):
    v = torch.randn(n, 3, generator=g, device=DEVICE, dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _cloud(case, g):
    """q, p, f, sigma, R of a batch in the case's type."""
    B, Q, P, F = case["B"], case["Q"], case["P"], case["F"]
    rand = lambda *s: torch.rand(*s, generator=g, device=DEVICE, dtype=torch.float64)  # noqa: E731
    f = rand(B, P, F)
    if case["layout"] == "surface":
        n = _directions(B * P, g)
        radius = 1.0 + 0.01 * torch.randn(B * P, 1, generator=g, device=DEVICE, dtype=torch.float64)
        p = (n * radius).reshape(B, P, 3)
        near = torch.randn(B * Q, 3, generator=g, device=DEVICE, dtype=torch.float64)
        q = (_directions(B * Q, g) + 0.05 * near).reshape(B, Q, 3)
        axis = torch.where((n[:, :1].abs() < 0.9), torch.tensor([1.0, 0, 0], device=DEVICE, dtype=torch.float64),
                           torch.tensor([0, 1.0, 0], device=DEVICE, dtype=torch.float64))
        t1 = torch.linalg.cross(axis, n)
        t1 = t1 / t1.norm(dim=1, keepdim=True)
        R = torch.stack([t1, torch.linalg.cross(n, t1), n], dim=-1).reshape(B, P, 3, 3)
        sigma = torch.tensor([0.02, 0.02, 0.005], device=DEVICE, dtype=torch.float64).expand(B, P, 3)
    else:
        q, p = rand(B, Q, 3), rand(B, P, 3)
        if case["layout"] == "rand":
            sigma, R = rand(B, P, 3), rand(B, P, 3, 3)
        else:
            sigma, R = 0.05 + 0.15 * rand(B, P, 3), _rotations(B * P, g).reshape(B, P, 3, 3)
    dtype = getattr(torch, case["dtype"])
    return [t.to(dtype).contiguous() for t in (q, p, f, sigma, R)]


def _ragged_sizes(case):
    rng = random.Random(case["sizes_seed"])
    n = case["clouds"]
    Ps = [_log_int(rng, case["P_min"], case["P_max"]) for _ in range(n)]
    Qs = [_log_int(rng, case["Q_min"], case["Q_max"]) for _ in range(n)]
    Ks = [rng.choice(RAGGED_KS) for _ in range(n)]
    return Ps, Qs, Ks


def _inputs(case, seed):
    g = _gen(seed)
    if case["op"] == "ragged":
        Ps, Qs, _ = _ragged_sizes(case)
        ps, qs = [], []
        for P, Q in zip(Ps, Qs):  # a mixture of 8 Gaussians per cloud
            centres = torch.rand(8, 3, generator=g, device=DEVICE, dtype=torch.float64)
            for n, out in ((P, ps), (Q, qs)):
                pick = torch.randint(0, 8, (n,), generator=g, device=DEVICE)
                out.append(centres[pick] + 0.05 * torch.randn(n, 3, generator=g, device=DEVICE, dtype=torch.float64))
        n = sum(Ps)
        sigma = 0.01 + 0.09 * torch.rand(n, 3, generator=g, device=DEVICE, dtype=torch.float64)
        f = torch.rand(n, case["F"], generator=g, device=DEVICE, dtype=torch.float64)
        return {k: t.float().contiguous() for k, t in
                (("q", torch.cat(qs)), ("p", torch.cat(ps)), ("f", f), ("sigma", sigma), ("R", _rotations(n, g)))}
    q, p, f, sigma, R = _cloud(case, g)
    got = {"q": q, "p": p, "f": f, "sigma": sigma, "R": R}
    if case["op"] == "lookup":
        # the batch's clouds are small deformations of one template, whose neighbour table they share
        jitter = 0.002 * torch.randn(p.shape, generator=g, device=DEVICE, dtype=torch.float64)
        got["p"] = (p[:1].double() + jitter).to(p.dtype).contiguous()
        got["table"] = torch.cdist(p[0].double(), p[0].double()).topk(case["K"], largest=False).indices.contiguous()
    if case["op"] in ("train", "lookup"):
        got["grad"] = torch.randn(q.shape[0], q.shape[1], case["F"], generator=g, device=DEVICE,
                                  dtype=torch.float64).to(q.dtype)
    return got


def prepare(case, seed):
    state = dict(_inputs(case, seed), op=case["op"], K=case.get("K"))
    if case["op"] == "ragged":
        Ps, Qs, Ks = _ragged_sizes(case)
        state["clouds"] = CloudSet(state["p"], state["sigma"], state["R"], state["f"], Ps)
        state["Qs"], state["Ks"] = Qs, Ks
        state["order"] = list(range(len(Ps)))
        state["want"] = [i < (len(Ps) + 1) // 2 for i in range(len(Ps))]
    elif case["op"] != "forward":
        for k in ("q", "p", "f", "sigma", "R"):
            state[k].requires_grad_(True)
    return state


# --------------------------------------------------------------------- run


def run(state):
    op, K = state["op"], state["K"]
    if op == "ragged":
        r = ragged_forward(state["clouds"], state["q"], state["order"], state["Qs"], state["Ks"],
                           grad_q=state["want"])
        return {"f_out": r.f_out, "w_out": r.w_out, "dists": r.dists, "idxs": r.idxs, "dq": r.dq}
    ins = [state[k] for k in ("q", "p", "f", "sigma", "R")]
    if op == "forward":
        with torch.no_grad():
            f_out, w_out, dists, idxs = knn_aggregate_aniso(*ins, K)
        return {"f_out": f_out, "w_out": w_out, "dists": dists, "idxs": idxs}
    if op == "lookup":
        f_out, w_out, dists, idxs = knn_aggregate_aniso_lookup(*ins, state["table"], K)
    else:
        f_out, w_out, dists, idxs = knn_aggregate_aniso(*ins, K)
    out = {"f_out": f_out, "w_out": w_out, "dists": dists, "idxs": idxs}
    if op == "eikonal":
        (dq,) = torch.autograd.grad(f_out.sum(), ins[0], create_graph=True)
        loss = ((dq.norm(dim=-1) - 1.0) ** 2).mean()
        out["dq"] = dq
        out["grads"] = torch.autograd.grad(loss, ins)
    else:
        out["grads"] = torch.autograd.grad(f_out, ins, grad_outputs=state["grad"])
    return out


# -------------------------------------------------------------------- work


def _work(op, Q, P, F, K, size):
    """Bytes (each input read once, each output written once) and operations
    of Q queries against P points: the keys, weights and sums of the K kept
    neighbours, not of the points that a search may skip."""
    points = P * (15 + F) * size  # p, sigma, R, f
    nbytes = Q * 3 * size + points + Q * (F + 2 * K) * size + 8 * Q * K  # q, f_out, w_out, dists, idxs
    flops = Q * K * (26 + 2 * F)
    if op in ("train", "lookup"):
        nbytes += Q * F * size + Q * 3 * size + points  # grad of f_out; the five gradients
        flops += Q * K * (90 + 4 * F)
        if op == "lookup":
            nbytes += 8 * P * K
    elif op == "eikonal":
        nbytes += 2 * Q * 3 * size + points  # dq and the five gradients
        flops += Q * K * (40 + 250) + P * F
    elif op == "ragged":
        nbytes += Q // 2 * 3 * size
        flops += Q // 2 * K * 40
    return nbytes, flops


def work(case):
    size = 8 if case["dtype"] == "float64" else 4
    if case["op"] == "ragged":
        every = [_work("ragged", Q, P, case["F"], K, size) for P, Q, K in zip(*_ragged_sizes(case))]
        return {"bytes": sum(b for b, _ in every), "flops": sum(n for _, n in every)}
    nbytes, flops = _work(case["op"], case["Q"], case["P"], case["F"], case["K"], size)
    return {"bytes": case["B"] * nbytes, "flops": case["B"] * flops}


# ------------------------------------------------------- values in 64 bits


def _keys64(q, p, sigma, R, idx):
    """Keys [n, k] of queries q [n, 3] against the points idx [n, k]."""
    d = q[:, None] - p[idx]
    u = (R[idx] @ d[..., None])[..., 0]
    return (sigma[idx] * u * u).sum(-1)


def _search64(q, p, sigma, R, K):
    """The K points with the smallest keys, ascending: candidates from the
    expanded quadratic form, ranked by their keys."""
    o = p.mean(0)
    pc = p - o
    M = R.transpose(1, 2) @ (sigma[..., None] * R)
    b = (M @ pc[..., None])[..., 0]
    psi = torch.stack([M[:, 0, 0], M[:, 1, 1], M[:, 2, 2], 2 * M[:, 0, 1], 2 * M[:, 0, 2], 2 * M[:, 1, 2],
                       -2 * b[:, 0], -2 * b[:, 1], -2 * b[:, 2], (pc * b).sum(1)])
    n, take, out = max(1, (1 << 28) // p.shape[0]), min(p.shape[0], K + 4), []
    for qc in q.split(n):
        x, y, z = (qc - o).unbind(1)
        phi = torch.stack([x * x, y * y, z * z, x * y, x * z, y * z, x, y, z, torch.ones_like(x)], 1)
        idx = (phi @ psi).topk(take, largest=False, sorted=False).indices
        best = _keys64(qc, p, sigma, R, idx).topk(K, largest=False, sorted=True).indices
        out.append(idx.gather(1, best))
    return torch.cat(out)


def _nearest64(q, p):
    return torch.cat([(qc[:, None] - p[None]).square().sum(-1).argmin(1)
                      for qc in q.split(max(1, (1 << 26) // p.shape[0]))])


def _aggregate64(q, p, f, sigma, R, idx):
    """(f_out, w, keys) at the neighbours idx, differentiable."""
    flat, (n, k) = idx.reshape(-1), idx.shape
    d = q[:, None] - p.index_select(0, flat).view(n, k, 3)
    u = (R.index_select(0, flat).view(n, k, 3, 3) * d[:, :, None, :]).sum(-1)
    s = (sigma.index_select(0, flat).view(n, k, 3) * u * u).sum(-1)
    w = torch.exp(-s)
    return (w[..., None] * f.index_select(0, flat).view(n, k, -1)).sum(1), w, s


def exact(case, seed):
    x = {k: t.double() if t.is_floating_point() else t for k, t in _inputs(case, seed).items()}
    if case["op"] == "ragged":
        Ps, Qs, Ks = _ragged_sizes(case)
        got = {k: [] for k in ("f_out", "w_out", "dists", "dq")}
        a = b = 0
        for s, (P, Q, K) in enumerate(zip(Ps, Qs, Ks)):
            p, f, sigma, R = (x[k][a:a + P] for k in ("p", "f", "sigma", "R"))
            q = x["q"][b:b + Q].clone().requires_grad_(True)
            f_out, w, keys = _aggregate64(q, p, f, sigma, R, _search64(q.detach(), p, sigma, R, K))
            want = s < (len(Ps) + 1) // 2
            dq = torch.autograd.grad(f_out.sum(), q)[0] if want else torch.zeros_like(q)
            for k, t in (("f_out", f_out), ("w_out", w.reshape(-1)), ("dists", keys.reshape(-1)), ("dq", dq)):
                got[k].append(t.detach())
            a, b = a + P, b + Q
        return dict({k: torch.cat(v) for k, v in got.items()}, idxs=None)
    B, Q, K, op = case["B"], case["Q"], case["K"], case["op"]
    names = ("q", "p", "f", "sigma", "R")
    outs = {k: [] for k in ("f_out", "w_out", "dists", "dq")}
    grads = {k: torch.zeros_like(x[k]) for k in names}
    for b in range(B):
        p, f, sigma, R = (x[k][b].clone().requires_grad_(op != "forward") for k in names[1:])
        for at in range(0, Q, 32768):
            rows = slice(at, min(Q, at + 32768))
            q = x["q"][b, rows].clone().requires_grad_(op != "forward")
            with torch.no_grad():
                idx = x["table"][_nearest64(q, p)] if op == "lookup" else _search64(q, p, sigma, R, K)
            f_out, w, keys = _aggregate64(q, p, f, sigma, R, idx)
            if op == "eikonal":
                (dq,) = torch.autograd.grad(f_out.sum(), q, create_graph=True)
                outs["dq"].append(dq.detach())
                got = torch.autograd.grad(((dq.norm(dim=-1) - 1.0) ** 2).sum() / (B * Q), (q, p, f, sigma, R))
            elif op != "forward":
                got = torch.autograd.grad(f_out, (q, p, f, sigma, R), grad_outputs=x["grad"][b, rows])
            for k, t in (("f_out", f_out), ("w_out", w), ("dists", keys)):
                outs[k].append(t.detach())
            if op != "forward":
                grads["q"][b, rows] = got[0]
                for k, t in zip(names[1:], got[1:]):
                    grads[k][b] += t
    result = {k: torch.cat(v).view(B, Q, -1) for k, v in outs.items() if v}
    result["idxs"] = None
    if op != "forward":
        result["grads"] = [grads[k] for k in names]
    return result
