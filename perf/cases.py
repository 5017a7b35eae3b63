"""The work that users of this library have it do, as cases with inputs, one
pass and its outputs.

Each case goes through the public Python view of the C ABI (Context, Mlp,
Surrogate, Batch).  Contexts, networks and their tables are built once per
grid and gain path and kept, as a program that steps many batches keeps them;
a state holds the distributions and the output buffers.  Distributions are
seeded mixtures of 1-4 Maxwellians, the inputs of the library's own runners
and benchmark; lattices are the cubic boxes [-5, 5]^3 of its configurations.

exact() restates the same results in FP64 torch: the gain by walking the pair
sums with the analytic sphere-in-box weights (spherical excess of a cap
octant, inclusion-exclusion over the box's corners), the loss, the projection,
the network and Adam straight from their definitions."""
from __future__ import annotations

import math

import numpy as np
import torch

import gpu_determ_gb300 as gd

DEV = "cuda"
PATHS = {"pair": gd.GAIN_PAIR, "bf16": gd.GAIN_CMATRIX_BF16, "bf16x3": gd.GAIN_CMATRIX_BF16X3,
         "pair_tc": gd.GAIN_PAIR_TC}
COURANT = 0.5
TRAIN_STEPS, TRAIN_LR, TRAIN_WARMUP = 64, 1e-3, 200


def listed():
    return [
        # the space-homogeneous relaxation runner: one cell, one step after another, default gain path
        {"name": "step one cell 20", "do": "step", "path": "pair", "n": 20, "R": 4.8, "cells": 1},
        # the reference program's own run: 16^3 whole box, 256 cells, default gain path
        {"name": "step 256 cells box 16", "do": "step", "path": "pair", "n": 16, "R": 16.5, "cells": 256},
        # nu and the gain for a solver with its own time stepping: a ragged batch on a small lattice, FP32 kernels
        {"name": "collision 1501 cells 12", "do": "collision", "path": "pair", "n": 12, "R": 4.8, "cells": 1501},
        # the benchmark's step: 4096 cells on the 20^3 lattice, BF16x3 collision matrices
        {"name": "step 4096 cells 20 x3", "do": "step", "path": "bf16x3", "n": 20, "R": 4.8, "cells": 4096},
        # the collision-matrix configuration: a batch of 1024 mixtures on 16^3
        {"name": "collision 1024 cells 16 x3", "do": "collision", "path": "bf16x3", "n": 16, "R": 4.8, "cells": 1024},
        # the one-pass matrices, a ragged batch with a padded leading dimension
        {"name": "collision 777 cells 20 bf16", "do": "collision", "path": "bf16", "n": 20, "R": 4.8, "cells": 777},
        # the finest lattice of the uneven batches on the path that serves lattices whose matrices do not fit
        {"name": "collision 512 cells 24 tc", "do": "collision", "path": "pair_tc", "n": 24, "R": 4.8, "cells": 512},
        # conservation projection alone (after a caller's own loss and gain), benchmark size
        {"name": "project 4096 cells 20", "do": "project", "n": 20, "R": 4.8, "cells": 4096},
        # the surrogate's network on the benchmark's batch
        {"name": "network forward 4096", "do": "forward", "n": 20, "R": 4.8, "cells": 4096},
        # an epoch's worth of training steps of the surrogate at its default batch, then the weights read back
        {"name": "network train 1024", "do": "train", "n": 20, "R": 4.8, "cells": 1024},
        # uneven lattices stepped together from one captured graph, every gain in one launch
        {"name": "uneven batch 8 12 16", "do": "batch", "path": "bf16x3", "n": 16, "R": 4.8, "cells": 500},
        # surrogate gain with plain fallback, about half of the cells falling back
        {"name": "surrogate 1024 cells 20", "do": "surrogate", "path": "bf16x3", "n": 20, "R": 4.8, "cells": 1024},
    ]


def draw(rng):
    def cells(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    do = rng.choice(["step", "step", "collision", "collision", "collision", "project", "forward", "train", "batch",
                     "surrogate"])
    c = {"do": do}
    if do in ("step", "collision"):
        c["path"] = rng.choice(["pair", "bf16", "bf16x3", "pair_tc"])
        c["n"] = rng.choice([8, 10, 12, 14, 16, 18, 20] + ([24] if c["path"] == "pair_tc" else []))
        c["R"] = rng.choice([4.8, 4.8, 4.8, 16.5]) if c["n"] <= 16 else 4.8
        hi = {8: 4096, 10: 4096, 12: 4096, 14: 2048, 16: 1024, 18: 512, 20: 512, 24: 256}[c["n"]]
        c["cells"] = cells(1, hi)
    elif do == "project":
        c["n"] = rng.choice([8, 12, 16, 20, 24])
        c["R"] = 4.8
        c["cells"] = cells(1, 4096)
    elif do in ("forward", "train"):
        c["n"] = rng.choice([8, 12, 16, 20])
        c["R"] = 4.8
        c["cells"] = cells(1, 4096) if do == "forward" else 64 * cells(1, 32)
    elif do == "batch":
        c["path"] = "bf16x3"
        c["n"] = rng.choice([12, 14, 16])
        c["R"] = 4.8
        c["cells"] = cells(4, 500)
    else:
        c["path"] = rng.choice(["bf16x3", "pair"])
        c["n"] = rng.choice([8, 12, 16])
        c["R"] = 4.8
        c["cells"] = cells(64, 1024)
    return c


# ---- lattice and inputs ----------------------------------------------------------
_kept = {}


def kept(key, make):
    if key not in _kept:
        _kept[key] = make()
    return _kept[key]


def lattice(n, R):
    """Packed in-sphere nodes [ns][3] of [-5, 5]^3, their velocities (FP64 of
    the stored floats), the box -> node map and the step."""
    def make():
        d = np.float32(10.0) / np.float32(n)
        t = np.float32(10.0) * (2 * np.arange(n) + 1 - n).astype(np.float32)
        m = (t.astype(np.float64) / 2.0 / n).astype(np.float32)      # the membership test's centres
        r2 = m[:, None, None] * m[:, None, None] + m[None, :, None] * m[None, :, None]
        r2 = (r2 + m[None, None, :] * m[None, None, :]).astype(np.float32)
        box = np.argwhere(r2 < np.float32(R) * np.float32(R))
        cmap = np.full((n, n, n), -1, np.int64)
        cmap[tuple(box.T)] = np.arange(len(box))
        v = (-5.0 + float(d) * (2.0 * np.arange(n) + 1.0) / 2.0).astype(np.float32).astype(np.float64)
        d3v = np.float32(np.float32(d * d) * d)
        return box, v[box], cmap, float(d), float(d3v)
    return kept(("lattice", n, R), make)


def ld_of(cells):
    """Leading dimension of a batch: the cells rounded up to four."""
    return (cells + 3) // 4 * 4


def mixtures(n, R, cells, seed):
    """float32 [ns][ld] on the device: per cell 1-4 Maxwellians, Dirichlet(1)
    weights, u ~ N(0, I), T ~ U[0.5, 2]."""
    rng = np.random.default_rng(seed)
    k = rng.integers(1, 5, cells)
    w = rng.dirichlet(np.ones(4), cells) * (np.arange(4)[None, :] < k[:, None])
    w /= w.sum(axis=1, keepdims=True)
    u, T = rng.normal(0.0, 1.0, (cells, 4, 3)), rng.uniform(0.5, 2.0, (cells, 4))
    X = torch.from_numpy(lattice(n, R)[1]).to(DEV)
    W, U, TT = (torch.from_numpy(a).to(DEV) for a in (w, u, T))
    out = torch.zeros((len(X), ld_of(cells)), dtype=torch.float32, device=DEV)
    for c0 in range(0, cells, 1024):
        c1 = min(cells, c0 + 1024)
        acc = torch.zeros((len(X), c1 - c0), dtype=torch.float64, device=DEV)
        for j in range(4):
            c2 = sum((X[:, a, None] - U[None, c0:c1, j, a]) ** 2 for a in range(3))
            acc += W[None, c0:c1, j] * (math.pi * TT[None, c0:c1, j]) ** -1.5 * torch.exp(-c2 / TT[None, c0:c1, j])
        out[:, c0:c1] = acc.float()
    return out


def project_inputs(case, seed):
    """f, nu and a gain near f nu, as a caller's own collision step leaves them."""
    f = mixtures(case["n"], case["R"], case["cells"], seed)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    v2 = torch.from_numpy((lattice(case["n"], case["R"])[1] ** 2).sum(1)).to(DEV).float()[:, None]
    nu = (20.0 + 4.0 * v2).sqrt() * (1.0 + 0.1 * torch.rand(f.shape[1], generator=gen, device=DEV)[None, :])
    gain = f * nu * (1.0 + 0.02 * torch.randn(f.shape, generator=gen, device=DEV))
    return f, nu.contiguous(), gain


def shapes(n_in, n_out):
    p, q = (n_in + 63) // 64 * 64, (n_out + 63) // 64 * 64
    return [(256, p), (512, 256), (512, 512), (256, 512), (q, 256)]


def weights(n_in, n_out, which):
    """A network's parameters (W_k [out][in], b_k): uniform fan-in weights as
    the library starts from, zero in the padding."""
    rng = np.random.default_rng(1000 + which)
    out = []
    for k, (o, i) in enumerate(shapes(n_in, n_out)):
        fan = n_in if k == 0 else i
        W = rng.uniform(-1.0, 1.0, (o, i)) / math.sqrt(fan)
        b = np.zeros(o)
        if k == 0:
            W[:, n_in:] = 0.0
        if k == 4:
            W[n_out:] = 0.0
        out.append((W.astype(np.float32), b.astype(np.float32)))
    return out


IN_GAIN, OUT_GAIN = 0.3, 2.0


def network(n_in, n_out, cap, flags, which):
    net = gd.Mlp(n_in, n_out, cap, flags=flags, seed=which)
    net.set_io_scale(IN_GAIN, OUT_GAIN if n_out > 1 else 1.0)
    net.set_params(np.concatenate([np.concatenate([W.ravel(), b]) for W, b in weights(n_in, n_out, which)]))
    return net


def context(n, R, path):
    def make():
        ctx = gd.Context(gd.GridSpec(n, R=R))
        ctx.set_gain_path(PATHS[path])
        assert ctx.n_pnt == len(lattice(n, R)[0])
        return ctx
    return kept(("context", n, R, path), make)


FORWARD = gd.MLP_SCALE_INPUT | gd.MLP_SCALE_OUTPUT
TRAIN = FORWARD | gd.MLP_LOSS_BATCH


def batch_cells(case):
    """(lattice, cells) of the groups of an uneven batch."""
    return [(8, case["cells"]), (case["n"] - 2 if case["n"] < 16 else 12, case["cells"]), (case["n"], case["cells"])]


# ---- the state before a call ---------------------------------------------------------
def prepare(case, seed):
    n, R, cells, do = case["n"], case["R"], case["cells"], case["do"]
    ns, ld = len(lattice(n, R)[0]), ld_of(cells)
    s = {"case": case}
    if do == "batch":
        # a captured graph keeps its contexts' buffers: the batch has its own contexts
        s["groups"], s["batch"] = [], gd.Batch()
        for k, (m, nc) in enumerate(batch_cells(case)):
            ctx = gd.Context(gd.GridSpec(m, R=R))
            ctx.set_gain_path(PATHS[case["path"]])
            f = mixtures(m, R, nc, seed + 100 * k)
            t = torch.zeros(1, dtype=torch.float32, device=DEV)
            s["batch"].add(ctx, f, nc, f.shape[1], gd.DT_COURANT, COURANT, time=t)
            s["groups"].append((f, t))
        s["batch"].set_mode(gd.BATCH_FUSED_CMATRIX)
        return s
    if do == "project":
        s["ctx"] = context(n, R, "pair")
        s["f"], s["nu"], s["gain"] = project_inputs(case, seed)
        s["nuc"] = torch.zeros_like(s["f"])
        s["q"] = torch.zeros(s["f"].shape, dtype=torch.float64, device=DEV)
        s["x"] = torch.zeros((cells, 5), dtype=torch.float64, device=DEV)
        return s
    s["f"] = mixtures(n, R, cells, seed)
    if do in ("step", "collision"):
        s["ctx"] = context(n, R, case["path"])
        s["nu"], s["gain"] = torch.zeros_like(s["f"]), torch.zeros_like(s["f"])
        s["dt"] = torch.zeros(1, dtype=torch.float32, device=DEV)
    elif do == "forward":
        s["net"] = kept(("net", n, R, cells), lambda: network(ns, ns, (cells + 63) // 64 * 64, FORWARD, 1))
        s["y"] = torch.zeros((ns, ld), dtype=torch.float32, device=DEV)
    elif do == "train":
        s["net"] = network(ns, ns, cells, TRAIN, 2)
        s["f"] = mixtures(n, R, 4 * cells, seed)     # four batches, in turn
        s["t"] = targets(s["f"])
        s["loss"] = torch.zeros(1, dtype=torch.float32, device=DEV)
        s["step"] = 0
    else:
        cap = (cells + 63) // 64 * 64
        s["net"] = kept(("snet", n, R, cap), lambda: network(ns, ns, cap, FORWARD, 3))
        s["est"] = kept(("sest", n, R, cap),
                        lambda: network(ns, 1, cap, gd.MLP_SCALE_INPUT | gd.MLP_LOSS_MSE, 4))
        s["ctx"] = context(n, R, case["path"])
        s["sur"] = kept(("sur", n, R, cap, case["path"]), lambda: gd.Surrogate(s["ctx"], s["net"], s["est"], cap))
        s["nu"], s["gain"] = torch.zeros_like(s["f"]), torch.zeros_like(s["f"])
        s["e"] = torch.zeros(cells, dtype=torch.float32, device=DEV)
        # the tolerance that about half of the cells miss
        s["sur"].gain(s["f"], cells, ld, float("inf"), s["nu"], s["gain"], s["e"])
        v = s["e"].cpu().numpy().astype(np.float64)
        v.sort()
        s["tol"] = float(10.0 ** (0.5 * (v[(cells - 1) // 2] + v[cells // 2])))
    return s


def targets(f):
    """What the training cases fit: a smooth quadratic functional of f."""
    m = f.mean(dim=0, keepdim=True)
    return (f * m - 0.25 * f * f).contiguous()


# ---- one pass ----------------------------------------------------------------------------
def run(s):
    case = s["case"]
    cells, do = case["cells"], case["do"]
    if do == "step":
        ld = s["f"].shape[1]
        s["ctx"].step(s["f"], cells, ld, gd.DT_COURANT, COURANT, nu=s["nu"], gain=s["gain"], dt=s["dt"])
        return {"f": s["f"], "nu": s["nu"], "gain": s["gain"], "dt": s["dt"]}
    if do == "collision":
        s["ctx"].collision(s["f"], cells, s["f"].shape[1], s["nu"], s["gain"])
        return {"nu": s["nu"], "gain": s["gain"]}
    if do == "project":
        s["ctx"].project(s["f"], s["nu"], s["gain"], cells, s["f"].shape[1], s["nuc"], s["q"], s["x"])
        return {"nu": s["nuc"], "q": s["q"], "x": s["x"]}
    if do == "forward":
        s["net"].forward(s["f"], s["f"].shape[1], cells, s["y"], s["y"].shape[1])
        return {"y": s["y"]}
    if do == "train":
        ld = s["f"].shape[1]
        for _ in range(TRAIN_STEPS):
            b = s["step"] % 4 * cells
            s["net"].train_step(s["f"][:, b:], ld, s["t"][:, b:], ld, cells, lr_at(s["step"]), loss=s["loss"])
            s["step"] += 1
        return {"params": s["net"].get_params(), "loss": s["loss"]}
    if do == "batch":
        s["batch"].step(True)
        return {"%s%d" % (k, i): v for i, g in enumerate(s["groups"]) for k, v in (("f", g[0]), ("time", g[1]))}
    nfb = s["sur"].gain(s["f"], cells, s["f"].shape[1], s["tol"], s["nu"], s["gain"], s["e"])
    return {"nu": s["nu"], "gain": s["gain"], "estimate": s["e"], "fallback": nfb}


def lr_at(step):
    return TRAIN_LR * min(1.0, (step + 1) / TRAIN_WARMUP)


# ---- what a pass cannot do without ------------------------------------------------------------
def collision_work(n, R, cells):
    ns = len(lattice(n, R)[0])
    pairs, terms, updates = plan(n, R)[1]
    return {"bytes": 12.0 * ns * cells, "flops": cells * (2.0 * pairs + 2.0 * terms + updates + 2.0 * ns * ns)}


def network_flops(ns, n_out):
    return 2.0 * sum(o * i for o, i in shapes(ns, n_out))


def work(case):
    n, R, cells, do = case["n"], case["R"], case["cells"], case["do"]
    ns = len(lattice(n, R)[0])
    values = float(ns) * cells
    if do in ("collision", "step"):
        w = collision_work(n, R, cells)
        # a step also projects (about 25 sums and 7 operations per value) and updates f
        return w if do == "collision" else {"bytes": w["bytes"] + 4 * values, "flops": w["flops"] + 60 * values}
    if do == "project":
        return {"bytes": (12 + 4 + 8) * values, "flops": 60 * values}
    if do == "forward":
        return {"bytes": 8 * values + 4.0 * sum(o * i for o, i in shapes(ns, ns)), "flops": cells * network_flops(ns, ns)}
    if do == "train":
        params = float(sum(o * i + o for o, i in shapes(ns, ns)))
        # per step: both batches once; parameters and two Adam moments read and written
        return {"bytes": TRAIN_STEPS * (8 * values + 24 * params) + 4 * params,
                "flops": TRAIN_STEPS * 3 * cells * network_flops(ns, ns)}
    if do == "batch":
        t = {"bytes": 0.0, "flops": 0.0}
        for m, nc in batch_cells(case):
            w, v = collision_work(m, R, nc), float(len(lattice(m, R)[0])) * nc
            t["bytes"] += 8 * v
            t["flops"] += w["flops"] + 60 * v
        return t
    w = collision_work(n, R, (cells + 1) // 2)
    return {"bytes": 12 * values, "flops": w["flops"] + cells * (network_flops(ns, 1) + 2.0 * ns * ns)
            + cells / 2 * network_flops(ns, ns)}


# ---- FP64 restatement ----------------------------------------------------------------------------
def octant_cap(A, B, C):
    """Area of {x >= A, y >= B, z >= C} on the unit sphere, A, B, C >= 0, by
    Gauss-Bonnet: 2 pi less the turning at the three corners and the geodesic
    curvature along the three circles."""
    live = A * A + B * B + C * C < 1.0
    A, B, C = (np.where(live, v, 0.0) for v in (A, B, C))
    sa, sb, sc = (np.sqrt(1.0 - v * v) for v in (A, B, C))

    def turn(x, y, sx, sy):
        return np.arccos(np.clip(-x * y / (sx * sy), -1.0, 1.0))

    def arc(x, y, r):
        return np.arccos(np.clip(y / r, -1.0, 1.0)) - np.arcsin(np.clip(x / r, -1.0, 1.0))

    area = (2.0 * math.pi - turn(A, B, sa, sb) - turn(B, C, sb, sc) - turn(A, C, sa, sc)
            - A * arc(B, C, sa) - B * arc(A, C, sb) - C * arc(A, B, sc))
    return np.where(live, area, 0.0)


def weight_class(n, p, d, d3v):
    """w(g, n') for the distinct |g| of one parity class and its offsets n',
    [rows][h^3], with the row of each g: 2 |g| d3v times the area of the unit
    sphere inside the box (n' - 1 .. n' + 1) / |g|."""
    h = n // 2
    ax = [2 * np.arange(h) + p[a] for a in range(3)]
    G = np.stack(np.meshgrid(*ax, indexing="ij"), -1).reshape(-1, 3)
    uniq, inv = np.unique((G * G).sum(1), return_inverse=True)
    rows = np.zeros((len(uniq), h ** 3))
    for r, u in enumerate(uniq):
        if u == 0:
            continue
        gg = math.sqrt(u)
        edges = [(np.maximum(a - 1, 0) / gg, (a + 1) / gg) for a in ax]
        lo_hi = [np.stack(e) for e in edges]
        T = octant_cap(lo_hi[0].reshape(2, 1, 1, h, 1, 1), lo_hi[1].reshape(1, 2, 1, 1, h, 1),
                       lo_hi[2].reshape(1, 1, 2, 1, 1, h))
        area = sum((-1) ** (i + j + k) * T[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1))
        area = area.reshape(-1)
        rows[r] = np.where(area < 1e-10, 0.0, area) * (2.0 * gg * d * d3v)
    return rows.astype(np.float32).astype(np.float64), inv.reshape(-1)


def plan(n, R):
    """Per box sum D in the low octant: its pairs, weights and targets, and
    the counts (pair products, weight terms, updates) per cell over the whole
    lattice.  Nodes outside the sphere have index ns."""
    def make():
        box, _, cmap, d, d3v = lattice(n, R)
        ns, h = len(box), n // 2
        cm = np.where(cmap < 0, ns, cmap)
        W = {p: weight_class(n, p, d, d3v) for p in np.ndindex(2, 2, 2)}
        items, pairs, terms, updates = [], 0, 0, 0
        for D in np.ndindex(n, n, n):
            p = tuple(x & 1 for x in D)
            h_a = [np.arange(D[a] // 2 + 1) for a in range(3)]
            H = np.stack(np.meshgrid(*h_a, indexing="ij"), -1).reshape(-1, 3)
            cls = (H[:, 0] * h + H[:, 1]) * h + H[:, 2]
            N = 2 * H + np.array(p)
            hi, lo = (np.array(D) + N) // 2, (np.array(D) - N) // 2
            at = {s: cm[np.where(s[0], hi[:, 0], lo[:, 0]), np.where(s[1], hi[:, 1], lo[:, 1]),
                        np.where(s[2], hi[:, 2], lo[:, 2])] for s in np.ndindex(2, 2, 2)}
            prod = [(at[s], at[tuple(1 - x for x in s)]) for s in ((1, 1, 1), (1, 0, 0), (1, 1, 0), (1, 0, 1))]
            have = np.zeros(len(N), bool)
            for a, b in prod:
                have |= (a < ns) & (b < ns)
            want = np.zeros(len(N), bool)
            tgt, src = [], []
            for s in np.ndindex(2, 2, 2):
                ok = at[s] < ns
                for a in range(3):
                    if s[a] == 0:
                        ok &= N[:, a] != 0
                want |= ok
                tgt.append(at[s][ok])
                src.append(np.flatnonzero(ok))
            mult = 1
            for a in range(3):
                mult *= 1 if D[a] == n - 1 else 2
            updates += mult * sum(len(t) for t in tgt)
            if not have.any() or not want.any():
                continue
            rows, row_of = W[p]
            used, pos = np.unique(np.where(want, row_of[cls], -1), return_inverse=True)
            pos = pos.reshape(-1) - (1 if used[0] < 0 else 0)
            Wd = rows[used[used >= 0]][:, cls[have]]
            pairs += mult * sum(int(((a < ns) & (b < ns)).sum()) for a, b in prod)
            terms += mult * int(np.count_nonzero(Wd))
            items.append((D, [(a[have], b[have]) for a, b in prod], Wd, np.concatenate(tgt),
                          pos[np.concatenate(src)]))
        return items, (pairs, terms, updates)
    return kept(("plan", n, R), make)


def exact_gain(n, R, f):
    box, _, cmap, _, _ = lattice(n, R)
    ns, cells = len(box), f.shape[1]
    refl = []
    for r in range(8):
        b = box.copy()
        for a in range(3):
            if r >> a & 1:
                b[:, a] = n - 1 - b[:, a]
        refl.append(cmap[tuple(b.T)])
    P = [torch.from_numpy(r).to(DEV) for r in refl]
    out = torch.zeros((ns, cells), dtype=torch.float64, device=DEV)
    for c0 in range(0, cells, 1024):
        c1 = min(cells, c0 + 1024)
        F = torch.zeros((8, ns + 1, c1 - c0), dtype=torch.float64, device=DEV)
        for r in range(8):
            F[r, :ns] = f[P[r], c0:c1].double()
        I = torch.zeros_like(F)
        for D, prod, Wd, tgt, src in plan(n, R)[0]:
            rs = [r for r in range(8) if all(not (r >> a & 1) or D[a] != n - 1 for a in range(3))]
            ix = np.concatenate([np.concatenate(ab) for ab in prod] + [tgt, src])
            ix = torch.from_numpy(ix).to(DEV)
            k, t = len(prod[0][0]), len(tgt)
            rr = slice(None) if len(rs) == 8 else None
            X = (F if rr else F[rs])[:, ix[:8 * k]].view(len(rs), 4, 2, k, -1) if rr else \
                F[torch.tensor(rs, device=DEV)[:, None], ix[None, :8 * k]].view(len(rs), 4, 2, k, -1)
            Pr = (X[:, :, 0] * X[:, :, 1]).sum(1)
            C = torch.from_numpy(Wd).to(DEV) @ Pr
            to, fr = ix[8 * k:8 * k + t], ix[8 * k + t:]
            if rr:
                I[:, to] += C[:, fr]
            else:
                I[torch.tensor(rs, device=DEV)[:, None], to[None, :]] += C[:, fr]
        for r in range(8):
            out[P[r], c0:c1] += I[r, :ns]
    return out


def exact_loss(n, R, f):
    box, _, _, d, d3v = lattice(n, R)
    X = torch.from_numpy(box.astype(np.float64)).to(DEV) * d
    B = 4.0 * math.pi * d3v * torch.cdist(X, X, compute_mode="donot_use_mm_for_euclid_dist")
    return B @ f.double()


def exact_project(n, R, f, nu, gain):
    """nu', Q and X of the conservation projection."""
    v = torch.from_numpy(lattice(n, R)[1]).to(DEV)
    phi = torch.cat([torch.ones_like(v[:, :1]), v, (v * v).sum(1, keepdim=True)], 1)
    f, nu, gain = f.double(), nu.double(), gain.double()
    fn = f * nu
    A = torch.einsum("ic,ik,il->ckl", fn, phi, phi) if f.shape[1] < 64 else \
        ((phi[:, :, None] * phi[:, None, :]).reshape(len(v), 25).T @ fn).T.reshape(-1, 5, 5)
    B = ((gain - fn).T @ phi)
    X = torch.linalg.solve(A, B)
    nuc = nu * (1.0 + phi @ X.T)
    return nuc, gain - f * nuc, X


def padded(v, ld):
    out = torch.zeros((v.shape[0], ld), dtype=v.dtype, device=v.device)
    out[:, :v.shape[1]] = v
    return out


def exact_step(n, R, f):
    nu, gain = exact_loss(n, R, f), exact_gain(n, R, f)
    nuc, q, _ = exact_project(n, R, f, nu, gain)
    dt = COURANT / nuc.max()
    return f.double() + dt * q, nuc, gain, dt.reshape(1)


def layers64(n_in, n_out, which):
    return [[torch.from_numpy(a).to(DEV).double() for a in wb] for wb in weights(n_in, n_out, which)]


def net64(L, x, flags, out_gain):
    """x [n_in][cells] -> y [n_out][cells] (padded outputs) and the cells' scale."""
    n_in = x.shape[0]
    s = x.mean(dim=0)
    X = torch.zeros((x.shape[1], L[0][0].shape[1]), dtype=torch.float64, device=DEV)
    X[:, :n_in] = x.T * (float(np.float32(IN_GAIN)) / s)[:, None]
    h0 = X @ L[0][0].T + L[0][1]
    g = torch.nn.functional.gelu
    h2 = g(g(h0 @ L[1][0].T + L[1][1]) @ L[2][0].T + L[2][1])
    z = h2 @ L[3][0].T + L[3][1] + h0
    return (z @ L[4][0].T + L[4][1]), s


def exact(case, seed):
    n, R, cells, do = case["n"], case["R"], case["cells"], case["do"]
    ns, ld = len(lattice(n, R)[0]), ld_of(cells)
    if do == "project":
        f, nu, gain = project_inputs(case, seed)
        r = exact_project(n, R, f[:, :cells], nu[:, :cells], gain[:, :cells])
        return {"nu": padded(r[0], ld), "q": padded(r[1], ld), "x": r[2]}
    if do == "batch":
        out = {}
        for k, (m, nc) in enumerate(batch_cells(case)):
            f = mixtures(m, R, nc, seed + 100 * k)
            r = exact_step(m, R, f[:, :nc])
            out["f%d" % k], out["time%d" % k] = padded(r[0], f.shape[1]), r[3]
        return out
    if do == "train":
        f = mixtures(n, R, 4 * cells, seed)
        t = targets(f)
        L = layers64(ns, ns, 2)
        flat = [p.requires_grad_(True) for wb in L for p in wb]
        m, v = [torch.zeros_like(p) for p in flat], [torch.zeros_like(p) for p in flat]
        og = float(np.float32(OUT_GAIN))
        for k in range(TRAIN_STEPS):
            b = k % 4 * cells
            y, s = net64(L, f[:, b:b + cells].double(), TRAIN, og)
            tt = t[:, b:b + cells].double().T / (s * s)[:, None] / og
            loss = ((y[:, :ns] - tt) ** 2).sum(1).mean() / (tt * tt).sum(1).mean()
            g = torch.autograd.grad(loss, flat)
            with torch.no_grad():
                for p, gg, mm, vv in zip(flat, g, m, v):
                    mm.mul_(0.9).add_(gg, alpha=0.1)
                    vv.mul_(0.999).addcmul_(gg, gg, value=0.001)
                    c1, c2 = 1.0 - 0.9 ** (k + 1), 1.0 - 0.999 ** (k + 1)
                    p -= lr_at(k) * (mm / c1) / ((vv / c2).sqrt() + 1e-8)
        return {"params": torch.cat([p.detach().reshape(-1) for p in flat]).cpu().numpy(),
                "loss": loss.detach().reshape(1)}
    f = mixtures(n, R, cells, seed)
    if do == "forward":
        y, s = net64(layers64(ns, ns, 1), f[:, :cells].double(), FORWARD, OUT_GAIN)
        return {"y": padded(y[:, :ns].T * (s * s)[None, :] * float(np.float32(OUT_GAIN)), ld)}
    nu = exact_loss(n, R, f[:, :cells])
    if do == "surrogate":
        # which cells fall back, and so the gain, hangs on the estimate's own rounding
        y, _ = net64(layers64(ns, 1, 4), f[:, :cells].double(), FORWARD, 1.0)
        return {"nu": padded(nu, ld), "gain": None, "estimate": y[:, 0].contiguous(), "fallback": None}
    if do == "collision":
        return {"nu": padded(nu, ld), "gain": padded(exact_gain(n, R, f[:, :cells]), ld)}
    r = exact_step(n, R, f[:, :cells])
    return {"f": padded(r[0], ld), "nu": padded(r[1], ld), "gain": padded(r[2], ld), "dt": r[3]}
