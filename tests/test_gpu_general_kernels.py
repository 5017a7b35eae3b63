"""The kernels that serve lattices of more than 1024 orbits (loss_kernel,
gain_pair_kernel, pair_tc_kernel, the BF16x3 matrices from 512 nodes on), on small
lattices: Context.use_general_kernels() takes the orbit kernels away.  Checked against
the FP64 oracle and against the orbit kernels, which share no code with them.  Also
the multi-grid launches, which batches of small lattices no longer reach otherwise.

Tolerances: the FP32 pair gain 1e-5 in relative L2 (its chains of up to some thousand
FP32 additions, as in the parity tests), the tensor-core pair gain 2e-5 (BF16 hi/lo
products, 2^-17 per operand), the loss per node 66 x 2^-24 = 3.9e-6 (chains of 64
non-negative products, one rounding of b, one of the sum), the BF16x3 matrices 1e-5."""
import ctypes as C

import numpy as np
import pytest

from gpu_determ_gb300 import inputs
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def _general(gd, dims, R, path=None):
    ctx = gd.Context(gd.GridSpec(*dims, R=R))
    ctx.use_general_kernels()
    ctx.set_gain_path(gd.GAIN_PAIR if path is None else path)
    return ctx


def _collision(torch, ctx, f, nc, ld):
    ft = torch.full((ctx.n_pnt, ld), float("nan"), dtype=torch.float32, device="cuda")   # padding is not read
    ft[:, :nc] = torch.from_numpy(f).cuda() if isinstance(f, np.ndarray) else f
    out = [torch.full_like(ft, -1.0) for _ in range(4)]
    for nu, gain in (out[:2], out[2:]):
        ctx.collision(ft, nc, ld, nu, gain)
    ctx.check()
    assert torch.equal(out[0], out[2]) and torch.equal(out[1], out[3])        # bitwise reproducible
    assert all(bool((o[:, nc:] == -1.0).all()) for o in out)                  # padding columns untouched
    return out[0][:, :nc], out[1][:, :nc]


def _rel(a, b):
    a, b = (x.cpu().numpy().astype(np.float64) if hasattr(x, "cpu") else x for x in (a, b))
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("path,tol", [("pair", 1e-5), ("pair_tc", 2e-5), ("x3", 1e-5)])
@pytest.mark.parametrize("dims,R,nc,ld", [((2, 2, 2), 16.5, 1, 1), ((4, 2, 6), 16.5, 33, 35), ((8, 8, 8), 16.5, 129, 131),
                                          ((12, 10, 8), 4.2, 64, 65), ((12, 12, 12), 4.8, 31, 31)])
def test_loss_and_gain_match_oracle(cuda, gdlib, dims, R, nc, ld, path, tol):
    paths = {"pair": gdlib.GAIN_PAIR, "pair_tc": gdlib.GAIN_PAIR_TC, "x3": gdlib.GAIN_CMATRIX_BF16X3}
    ctx = _general(gdlib, dims, R, paths[path])
    f = inputs.mixtures(ctx.spec.fill(), nc, seed=sum(dims) + nc)
    nu, gain = _collision(cuda, ctx, f, nc, ld)
    o = Oracle(*dims, R=R)
    box = o.to_box(f)
    ref = o.loss_f64(box)
    worst = np.max(np.abs(nu.cpu().numpy() - ref) / ref)
    assert worst <= 3.9e-6, worst      # ld odd: the FP32 loss on every path
    rel = _rel(gain, o.gain_f64(box))
    assert rel <= tol, rel


@pytest.mark.parametrize("path,tol", [("pair", 1e-5), ("pair_tc", 2e-5)])
@pytest.mark.parametrize("n,nc", [(16, 300), (24, 130)])
def test_gain_matches_the_orbit_kernel(cuda, gdlib, n, nc, path, tol):
    """24^3: class boxes with up to 412 row groups, two passes of at most 256."""
    torch = cuda
    ref_ctx = gdlib.Context(gdlib.GridSpec(n, R=4.8))
    f = torch.from_numpy(inputs.dirichlet_mixtures(ref_ctx.spec.fill(), nc, seed=n)).cuda()
    ref = torch.empty_like(f)
    ref_ctx.collision(f, nc, nc, None, ref)
    ctx = _general(gdlib, (n, n, n), 4.8, gdlib.GAIN_PAIR if path == "pair" else gdlib.GAIN_PAIR_TC)
    _, gain = _collision(torch, ctx, f, nc, nc)
    rel = _rel(gain, ref)
    assert 0.0 < rel <= tol, rel       # another kernel, so other roundings


def test_pair_tc_bits_scale_and_batch(cuda, gdlib):
    """64-bit fixed-point sums: exact under powers of two, the same bits alone and in
    a batch; a non-finite cell gets NaN alone."""
    torch = cuda
    nc = 160
    ctx = _general(gdlib, (12, 12, 12), 4.8, gdlib.GAIN_PAIR_TC)
    f = torch.from_numpy(inputs.dirichlet_mixtures(ctx.spec.fill(), nc, seed=5)).cuda()
    _, base = _collision(torch, ctx, f, nc, nc)
    g = f.clone()
    g[:, 3] *= 2.0 ** 20
    g[:, 7] *= 2.0 ** -8
    g[5, 11] = float("nan")
    g[9, 140] = float("inf")
    out = torch.empty_like(g)
    ctx.collision(g, nc, nc, None, out)
    assert torch.equal(out[:, 3], base[:, 3] * 2.0 ** 40)
    assert torch.equal(out[:, 7], base[:, 7] * 2.0 ** -16)
    assert bool(torch.isnan(out[:, 11]).all()) and bool(torch.isnan(out[:, 140]).all())
    keep = [c for c in range(nc) if c not in (3, 7, 11, 140)]
    assert torch.equal(out[:, keep], base[:, keep])
    for first, count in ((0, 1), (5, 129), (100, 60)):
        _, part = _collision(torch, ctx, f[:, first:first + count], count, count)
        assert torch.equal(part, base[:, first:first + count])


STEPS = 3


@pytest.mark.parametrize("mode,path,general,specs", [
    ("BATCH_FUSED_PAIR_TC", "GAIN_PAIR_TC", True, [(8, 200), (12, 300), (16, 130)]),
    ("BATCH_FUSED_CMATRIX", "GAIN_CMATRIX_BF16X3", True, [(8, 33), (12, 300), (10, 1)]),
    ("BATCH_FUSED_CMATRIX", "GAIN_CMATRIX_BF16X3", False, [(8, 200), (10, 37), (6, 129)]),
    ("BATCH_FUSED_CMATRIX", "GAIN_CMATRIX_BF16", False, [(12, 100), (8, 17), (16, 40), (10, 1)]),
    # one group by the FP32 kernel, the others in one launch
    ("BATCH_FUSED_CMATRIX", "GAIN_CMATRIX_BF16X3", False, [(8, 50), (12, 100), (10, 37)])])
def test_one_launch_over_several_grids_matches_single_steps(cuda, gdlib, mode, path, general, specs):
    torch = cuda
    groups = []
    for n, cells in specs:
        ctx = _general(gdlib, (n, n, n), 4.8) if general else gdlib.Context(gdlib.GridSpec(n, R=4.8))
        ctx.set_gain_path(getattr(gdlib, path))
        groups.append((ctx, inputs.mixtures(ctx.spec.fill(), cells, seed=n + cells), cells))
    single = []
    for ctx, f0, cells in groups:
        f = torch.from_numpy(f0).cuda()
        t = torch.zeros(1, dtype=torch.float32, device="cuda")
        for _ in range(STEPS):
            ctx.step(f, cells, cells, gdlib.DT_COURANT, 0.5, time=t)
        single.append((f, t))
    for use_graph in (False, True):
        b = gdlib.Batch()
        batch = []
        for ctx, f0, cells in groups:
            f = torch.from_numpy(f0).cuda()
            t = torch.zeros(1, dtype=torch.float32, device="cuda")
            b.add(ctx, f, cells, cells, gdlib.DT_COURANT, 0.5, time=t)
            batch.append((f, t))
        b.set_mode(getattr(gdlib, mode))
        for _ in range(STEPS):
            b.step(use_graph)
        b.check()
        b.close()
        torch.cuda.synchronize()
        for (f, t), (g, u) in zip(single, batch):
            assert torch.equal(f, g) and torch.equal(t, u) and float(t) > 0


# the fixed array holds gd_collision's chunks in the second case
@pytest.mark.parametrize("n,nc,ld,bitwise", [(12, 40, 44, False), (12, 256, 256, True), (16, 300, 301, False)])
def test_noalloc_gain_of_the_pair_kernel(cuda, gdlib, n, nc, ld, bitwise):
    torch = cuda
    ctx = _general(gdlib, (n, n, n), 4.8)
    f = inputs.mixtures(ctx.spec.fill(), nc, seed=n)
    _, ref = _collision(torch, ctx, f, nc, ld)
    ft = torch.zeros((ctx.n_pnt, ld), dtype=torch.float32, device="cuda")
    ft[:, :nc] = torch.from_numpy(f).cuda()
    out = torch.full_like(ft, -1.0)
    assert gdlib.lib().gd_gain_noalloc(ctx._h, C.c_void_p(ft.data_ptr()), nc, ld, C.c_void_p(out.data_ptr()), None) == 0
    torch.cuda.synchronize()
    assert bool((out[:, nc:] == -1.0).all())
    assert torch.equal(out[:, :nc], ref) if bitwise else _rel(out[:, :nc], ref) <= 1e-6


def test_step_by_the_general_kernels(cuda, gdlib):
    """A whole step on both kinds of kernels: the same time step and distribution to
    the FP32 kernels' accuracy."""
    torch = cuda
    nc = 50
    ctxs = [gdlib.Context(gdlib.GridSpec(12, R=4.8)), _general(gdlib, (12, 12, 12), 4.8)]
    f0 = inputs.mixtures(ctxs[0].spec.fill(), nc, seed=2)
    out = []
    for ctx in ctxs:
        f = torch.from_numpy(f0).cuda()
        t = torch.zeros(1, dtype=torch.float32, device="cuda")
        ctx.step(f, nc, nc, gdlib.DT_COURANT, 0.5, time=t)
        ctx.check()
        out.append((f, float(t)))
    assert out[0][1] == pytest.approx(out[1][1], rel=1e-5)
    assert _rel(out[0][0], out[1][0]) <= 1e-5
