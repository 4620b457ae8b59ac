"""What a program built on this framework has it do, as cases that can be timed and compared.

A case is a dict of plain values. Its "op" names the public call (repulsive_test2_b200.api):

  energy    calculateEnergy: the objective alone, as a line search or a display asks for it
  grad      energyAndGradient: the adjoint gradient with its forward energy
  cgrad     solveConstrainedGradientSet: Gram assembly, factorization and saddle solve
  step      sobolevStepSet: the whole descent step, the call that an application repeats
  batch     Batch.step: one step for each of many curves of uneven size
  bh        bhEnergy: the Barnes-Hut energy of a curve far beyond the dense kernels

Every call takes and returns host arrays, as a program calls it. The curves are the ones that
this repository measures with: jittered trefoils and torus knots, random-walk knots, and
networks of random-walk loops joined at Y-junctions. The topology of a case is fixed; its
positions are moved a little by the seed.
"""
import math

import numpy as np
import torch

from repulsive_test2_b200 import api
from repulsive_test2_b200 import fixtures

EPS = 1e-10
TORUS = ((2, 3), (3, 5), (2, 7))


def listed():
    return [
        # one small curve, the smallest call: a display or a host-side search asks for the energy
        {"name": "energy_v128", "op": "energy", "curve": "trefoil", "V": 128, "alpha": 3.0, "beta": 6.0},
        # a single curve of ordinary size: the raw descent direction and its energy
        {"name": "grad_v2048", "op": "grad", "curve": "walk", "V": 2048, "alpha": 3.0, "beta": 6.0},
        # exponents that a user dialled away from the defaults, and an odd size
        {"name": "grad_v1311_a2", "op": "grad", "curve": "torus", "V": 1311, "alpha": 2.0, "beta": 4.5},
        # 12 loops of 1024 vertices joined at Y-junctions: any topology, the largest gradient
        {"name": "grad_net12288", "op": "grad", "curve": "net", "loops": 12, "V": 1024, "alpha": 3.0, "beta": 6.0},
        # the Sobolev direction of one curve for a caller that runs its own search
        {"name": "cgrad_v777", "op": "cgrad", "curve": "torus", "V": 777, "alpha": 3.0, "beta": 6.0},
        # an interactive editor's curve: defaults, the operator assembled anew at each correction
        {"name": "step_v128", "op": "step", "curve": "trefoil", "V": 128, "set": "length",
         "projection": "reassemble", "precision": "fp64"},
        # a single random-walk knot in double precision, frozen projection
        {"name": "step_v2048", "op": "step", "curve": "walk", "V": 2048, "set": "length",
         "projection": "frozen", "precision": "fp64"},
        # the headline: the largest dense step, mixed precision, batched trials
        {"name": "step_v8192_mixed", "op": "step", "curve": "walk", "V": 8192, "set": "length",
         "projection": "frozen", "precision": "mixed"},
        # every edge length held, a ragged size: the large constraint set's explicit inverses
        {"name": "step_v2500_edges", "op": "step", "curve": "walk", "V": 2500, "set": "edges",
         "projection": "frozen", "precision": "mixed"},
        # a loop network with pins and penalties in double precision: the general assembly
        {"name": "step_net1200", "op": "step", "curve": "net", "loops": 4, "V": 300, "set": "pins",
         "projection": "frozen", "precision": "fp64"},
        # many curves of uneven size at once
        {"name": "batch_64", "op": "batch", "count": 64, "vmin": 256, "vmax": 1500},
        # one very long smooth curve through the edge tree
        {"name": "bh_e131072", "op": "bh", "V": 131072, "theta": 0.5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(("energy", "grad", "grad", "cgrad", "step", "step", "step", "edges", "net", "batch", "bh"))
    curve = rng.choice(("trefoil", "torus", "walk"))
    alpha, beta = rng.choice(((3.0, 6.0), (3.0, 6.0), (2.0, 4.5)))
    if op == "energy":
        return {"op": "energy", "curve": curve, "V": _log(rng, 24, 8192), "alpha": alpha, "beta": beta}
    if op == "grad":
        if rng.random() < 0.3:
            return {"op": "grad", "curve": "net", "loops": rng.randint(2, 12), "V": _log(rng, 24, 1024),
                    "alpha": 3.0, "beta": 6.0}
        return {"op": "grad", "curve": curve, "V": _log(rng, 64, 4096 if alpha == 2.0 else 12000),
                "alpha": alpha, "beta": beta}
    if op == "cgrad":
        return {"op": "cgrad", "curve": rng.choice(("trefoil", "torus")), "V": _log(rng, 64, 800),
                "alpha": 3.0, "beta": 6.0}
    if op == "step":
        if rng.random() < 0.25:
            return {"op": "step", "curve": curve, "V": _log(rng, 32, 512), "set": "length",
                    "projection": "reassemble", "precision": "fp64"}
        precision = rng.choice(("fp64", "mixed"))
        most = 2500 if curve != "walk" else 8192 if precision == "mixed" else 4096
        return {"op": "step", "curve": curve, "V": _log(rng, 128, most), "set": "length",
                "projection": "frozen", "precision": precision}
    if op == "edges":
        return {"op": "step", "curve": curve, "V": _log(rng, 100, 2800), "set": "edges",
                "projection": "frozen", "precision": rng.choice(("fp64", "mixed"))}
    if op == "net":
        return {"op": "step", "curve": "net", "loops": rng.randint(2, 6), "V": _log(rng, 32, 256), "set": "pins",
                "projection": "frozen", "precision": "fp64"}
    if op == "batch":
        return {"op": "batch", "count": rng.randint(4, 40), "vmin": _log(rng, 64, 256), "vmax": _log(rng, 400, 1500)}
    return {"op": "bh", "V": _log(rng, 4096, 131072), "theta": rng.choice((0.25, 0.5))}


# ---- inputs -----------------------------------------------------------------------------

def _curve(kind, n, seed, loops=1, base=1):
    """A curve of the kind (its shape from `base`, as the benchmark's workloads fix theirs), each vertex
    moved by a fiftieth of the mean edge length by `seed`."""
    if kind == "trefoil":
        v, e = fixtures.trefoil(n, jitter=0.01, seed=base)
    elif kind == "torus":
        v, e = fixtures.torus_knot(n, *TORUS[n % 3], jitter=0.01, seed=base)
    elif kind == "walk":
        v, e = fixtures.random_walk_knot(n, seed=7 + base)
    else:
        v, e = fixtures.loop_network(loops=loops, n=n, junctions=min(8, 2 * loops), seed=5)
    # (the first n edges are the first loop's: a network's long bridges follow all loops)
    step = 0.02 * float(api.edgeLengths(v, e[:n]).mean())
    return v + step * fixtures.normals(seed * 8 + 5, v.size).reshape(-1, 3), e


def _blocks(which, v, e):
    out = [api.barycenterBlock(api.barycenterTarget(v, e))]
    if which == "length":
        return out + [api.totalLengthBlock(api.totalLength(v, e))]
    out.append(api.edgeLengthsBlock(api.edgeLengths(v, e)))
    if which == "pins":
        # sixteen pins spread over the network, no two on one edge (their length is held already)
        out += [api.pointBlock(p, v[p]) for p in (k * len(v) // 16 + 2 for k in range(16))]
    return out


def _batch_sizes(case):
    """Log-uniform between vmin and vmax, the same for every seed."""
    u = fixtures.uniforms(3, case["count"])
    return [int(round(case["vmin"] * (case["vmax"] / case["vmin"]) ** float(x))) for x in u]


def prepare(case, seed):
    op = case["op"]
    seed = 1 + seed % 1000003
    if op == "batch":
        curves = [_curve(("trefoil", "torus", "walk")[c % 3], n, seed * 64 + c, base=300 + c)
                  for c, n in enumerate(_batch_sizes(case))]
        return {"op": op, "batch": api.Batch(curves), "xs": [v for v, _ in curves],
                "sets": [_blocks("length", v, e) for v, e in curves],
                "opts": {"projectionMode": "frozen", "precision": "mixed", "trials": 8}}
    if op == "bh":
        # a smooth closed curve: the trefoil with three small harmonics of the seed
        n = case["V"]
        t = np.linspace(0.0, 2.0 * np.pi, n, endpoint=False)
        v = np.stack([np.sin(t) + 2.0 * np.sin(2.0 * t), np.cos(t) - 2.0 * np.cos(2.0 * t), -np.sin(3.0 * t)], axis=1)
        a = fixtures.normals(seed, 9).reshape(3, 3) * 0.02
        v = 0.25 * (v + sum(np.sin((k + 4) * t + k)[:, None] * a[k] for k in range(3)))
        return {"op": op, "v": np.ascontiguousarray(v), "e": fixtures.closed_edges(n), "theta": case["theta"]}
    v, e = _curve(case["curve"], case["V"], seed, case.get("loops", 1))
    state = {"op": op, "v": v, "e": e, "alpha": case.get("alpha", 3.0), "beta": case.get("beta", 6.0)}
    if op == "cgrad":
        state["dE"] = _energy_grad(v, e, state["alpha"], state["beta"])[1]
        state["set"] = _blocks("length", v, e)
    if op == "step":
        state["set"] = _blocks(case["set"], v, e)
        state["opts"] = {"projectionMode": case["projection"], "precision": case["precision"]}
        if case["set"] == "pins":
            state["opts"]["penalties"] = {"totalLength": 1.0, "lengthDiff": 10.0,
                                          "field": {"weight": 5.0, "X": [0.5, 1.0, 0.0]}}
        elif case["projection"] == "frozen":
            # an application's loop hands each step the energy that the last one ended with
            state["opts"]["energyBefore"] = api.calculateEnergy(v, e)
    return state


def _stepped(r):
    # the new curve and what the search decided; its energy is that of these vertices (the energy
    # case), which near contacts of a rough curve make far more sensitive than the vertices are
    return {"vertices": r["vertices"], "tau": r["stats"]["tau"], "accepted": r["accepted"],
            "converged": r["converged"]}


def run(state):
    op = state["op"]
    if op == "energy":
        return {"energy": api.calculateEnergy(state["v"], state["e"], None, state["alpha"], state["beta"], EPS)}
    if op == "grad":
        energy, grad = api.energyAndGradient(state["v"], state["e"], state["alpha"], state["beta"], EPS)
        return {"energy": energy, "grad": grad}
    if op == "cgrad":
        r = api.solveConstrainedGradientSet(state["v"], state["e"], None, state["alpha"], state["beta"], EPS,
                                            state["dE"], state["set"])
        return {"gTilde": r["gTilde"], "lambda": r["lambda"]}
    if op == "step":
        return _stepped(api.sobolevStepSet(state["v"], state["e"], None, state["set"], state["opts"]))
    if op == "batch":
        got = [_stepped(r) for r in state["batch"].step(state["xs"], state["sets"], state["opts"])]
        return {"vertices": np.concatenate([r["vertices"] for r in got]),
                "tau": np.array([r["tau"] for r in got]), "converged": np.array([r["converged"] for r in got]),
                "accepted": np.array([r["accepted"] for r in got])}
    energy, counts = api.bhEnergy(state["v"], state["e"], theta=state["theta"], leafSize=8)
    return {"energy": energy, "counts": counts}


# ---- what a pass cannot do without ------------------------------------------------------

def _step_work(V, E, rows, evals):
    """Bytes and operations of one step: the pair terms of the gradient, the Gram matrix and
    `evals` energies, a Cholesky factorization of A and the solves for the constraint rows."""
    P = 0.5 * E * E
    flops = P * (793 + 278 + 249 * evals) + V ** 3 / 3.0 + 2.0 * V * V * 3 * min(rows + 1, 5)
    if rows > 64:  # the inverse of A and of the rows' Schur complement
        flops += 2.0 * V ** 3 / 3.0 + float(rows) ** 3
    return 8.0 * (6 * V + 2.0 * V * V), flops


def work(case):
    op = case["op"]
    if op == "batch":
        b = f = 0.0
        for n in _batch_sizes(case):
            x, y = _step_work(n, n, 4, 2)
            b, f = b + x, f + y
        return {"bytes": b, "flops": f}
    V = case["V"] * case.get("loops", 1)
    if op == "bh":
        # a tree walk per edge: about 160 visits of some 60 operations
        return {"bytes": 32.0 * V, "flops": 160.0 * 60.0 * V}
    if op == "energy":
        return {"bytes": 32.0 * V, "flops": 249 * 0.5 * V * V}
    if op == "grad":
        return {"bytes": 56.0 * V, "flops": 793 * 0.5 * V * V}
    if op == "cgrad":
        return {"bytes": 8.0 * (9 * V + 2.0 * V * V), "flops": 278 * 0.5 * V * V + V ** 3 / 3.0 + 30.0 * V * V}
    rows = {"length": 4, "edges": 3 + V, "pins": 51 + V}[case["set"]]
    b, f = _step_work(V, V, rows, 2)
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, in plain torch ------------------------------------------------

def _energy_grad(v, e, alpha, beta):
    """The tangent-point energy and its gradient: every edge against every edge that shares
    no vertex with it, four endpoint pairs each, in rows of a few hundred edges."""
    dev = "cuda"
    x = torch.tensor(v, dtype=torch.float64, device=dev)
    i = torch.tensor(np.asarray(e, dtype=np.int64), device=dev)
    n = len(i)
    rows = max(1, min(n, 4_000_000 // n))
    p1, p2 = x[i[:, 0]].requires_grad_(True), x[i[:, 1]].requires_grad_(True)
    energy, g1, g2 = 0.0, torch.zeros_like(p1), torch.zeros_like(p2)
    for r0 in range(0, n, rows):
        r = slice(r0, min(n, r0 + rows))
        share = (i[r, None, :, None] == i[None, :, None, :]).flatten(2).any(-1)
        eI, ell = p2[r] - p1[r], torch.linalg.vector_norm(p2 - p1, dim=1) + EPS
        total = 0.0
        for a in (p1, p2):
            for b in (p1, p2):
                d = a[r, None] - b[None]
                d = torch.where(share[..., None], torch.ones_like(d), d)
                c = torch.linalg.cross(eI[:, None].expand_as(d), d, dim=-1)
                c2 = (c * c).sum(-1)
                flat = c2 < 1e-28
                area = torch.where(flat, torch.zeros_like(c2), torch.where(flat, torch.ones_like(c2), c2).sqrt()) + EPS
                total = total + area ** alpha / ((d * d).sum(-1).sqrt() + EPS) ** beta
        w = torch.where(share, torch.zeros_like(total), total) * ell[r, None] ** (1.0 - alpha) * ell[None]
        part = 0.25 * w.sum() * 0.5
        h1, h2 = torch.autograd.grad(part, (p1, p2))
        energy, g1, g2 = energy + float(part.detach()), g1 + h1, g2 + h2
    # gathered in a fixed order, so that the same inputs give the same bits
    out = np.zeros_like(v)
    np.add.at(out, np.asarray(e)[:, 0], g1.detach().cpu().numpy())
    np.add.at(out, np.asarray(e)[:, 1], g2.detach().cpu().numpy())
    return energy, out


def _saddle(v, e, alpha, beta, dE):
    """The Gram matrix B + B0, the rows of [barycenter, totalLength] and the saddle system."""
    dev = "cuda"
    x = torch.tensor(v, dtype=torch.float64, device=dev)
    i = torch.tensor(np.asarray(e, dtype=np.int64), device=dev)
    V, n = len(v), len(i)
    p = (x[i[:, 0]], x[i[:, 1]])
    raw = torch.linalg.vector_norm(p[1] - p[0], dim=1)
    T, ell = (p[1] - p[0]) / raw[:, None], raw + EPS
    share = (i[:, None, :, None] == i[None, :, None, :]).flatten(2).any(-1)
    s = (beta - 1.0) / alpha
    w, q = torch.zeros(n, n, dtype=torch.float64, device=dev), torch.zeros(n, n, dtype=torch.float64, device=dev)
    for a in p:
        for b in p:
            d = a[:, None] - b[None]
            dn = torch.where(share, torch.ones_like(w), torch.linalg.vector_norm(d, dim=-1)) + EPS
            k = dn ** -(2.0 * (s - 1.0) + 1.0)
            c = torch.linalg.vector_norm(torch.linalg.cross(T[:, None].expand_as(d), d, dim=-1), dim=-1) + EPS
            w += k
            q += c ** 2 / dn ** 4 * k
    keep = (~share).double() * (ell[:, None] * ell[None])
    w, q = 0.25 * w * keep, 0.0625 * q * keep
    w, q = w + w.T, q + q.T
    D = torch.zeros(n, V, dtype=torch.float64, device=dev)
    U = torch.zeros(n, V, dtype=torch.float64, device=dev)
    at = torch.arange(n, device=dev)
    D[at, i[:, 0]], D[at, i[:, 1]] = 1.0, -1.0
    U[at, i[:, 0]], U[at, i[:, 1]] = 1.0, 1.0
    m = -w * (T @ T.T) / (ell[:, None] * ell[None])
    A = D.T @ (torch.diag(w.sum(1) / ell ** 2) + m) @ D + U.T @ (torch.diag(q.sum(1)) - q) @ U
    # constraint rows by differentiating barycenter and total length
    y = x.clone().requires_grad_(True)
    b0, b1 = y[i[:, 0]], y[i[:, 1]]
    le = torch.linalg.vector_norm(b1 - b0, dim=1)
    mid = 0.5 * (b0 + b1)
    x0 = torch.tensor(api.barycenterTarget(v, e), dtype=torch.float64, device=dev)
    phi = [(le[:, None] * (mid - x0)).sum(0)[c] for c in range(3)] + [-le.sum()]
    C = torch.stack([torch.autograd.grad(f, y, retain_graph=True)[0].T.reshape(-1) for f in phi])
    K = torch.zeros(3 * V + 4, 3 * V + 4, dtype=torch.float64, device=dev)
    for c in range(3):
        K[c * V:(c + 1) * V, c * V:(c + 1) * V] = A
    K[3 * V:, :3 * V], K[:3 * V, 3 * V:] = C, C.T
    rhs = torch.zeros(3 * V + 4, dtype=torch.float64, device=dev)
    rhs[:3 * V] = torch.tensor(dE, dtype=torch.float64, device=dev).T.reshape(-1)
    lu = torch.linalg.lu_factor(K)
    z = torch.linalg.lu_solve(*lu, rhs[:, None])[:, 0]
    for _ in range(3):
        z = z + torch.linalg.lu_solve(*lu, (rhs - K @ z)[:, None])[:, 0]
    return z[:3 * V].reshape(3, V).T.contiguous().cpu().numpy(), z[3 * V:].cpu().numpy()


def exact(case, seed):
    op = case["op"]
    if op in ("energy", "grad"):
        s = prepare(case, seed)
        energy, grad = _energy_grad(s["v"], s["e"], s["alpha"], s["beta"])
        return {"energy": energy} if op == "energy" else {"energy": energy, "grad": grad}
    if op == "cgrad":
        s = prepare(case, seed)
        g, lam = _saddle(s["v"], s["e"], s["alpha"], s["beta"], s["dE"])
        return {"gTilde": g, "lambda": lam}
    # a whole step (a search with its projections) and the tree walk take minutes in plain numpy
    return None
