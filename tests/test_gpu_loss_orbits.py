"""The FP32 loss frequency of cells whose mirrors differ widely: all mass on one
node, on a node and its mirrors, narrow beams far from the origin.

nu is a sum of non-negative products b f: chains of 32 of them (a rounding of
2^-24 at most each, of a partial sum that only grows), compensated sums of the
chains and one rounding of b, so every node's own nu is within 36 x 2^-24 =
2.2e-6 of the FP64 sum, however small it is beside its mirrors', never negative,
and exactly zero where the only filled node is the node itself (b(0) = 0)."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def _cells(spec, n):
    """[n_pnt][cells]: one node each, a node with three mirrors, beams."""
    g = spec.fill()
    rng = np.random.default_rng(n)
    nodes = rng.choice(n, min(n, 60), replace=False)
    f = np.zeros((n, len(nodes) + 6), np.float32)
    f[nodes, np.arange(len(nodes))] = rng.uniform(0.5, 2.0, len(nodes)).astype(np.float32)
    v = np.stack(inputs.node_velocities(g))
    m = int(nodes[0])
    for k, s in enumerate(((-1, 1, 1), (1, -1, 1), (1, 1, -1))):
        mirror = np.argmin(np.abs(v - (v[:, m] * np.array(s))[:, None]).sum(0))
        f[mirror, len(nodes)] = 10.0 ** -k
    f[m, len(nodes)] = 1.0
    for k, (u, T) in enumerate((((2.5, 2.5, 2.5), 0.1), ((2.0, -2.0, 2.0), 0.5), ((-3.0, 0.4, 0.4), 0.05),
                                ((4.0, 0.0, 0.0), 0.2), ((1.0, 1.0, -3.5), 0.1))):
        f[:, len(nodes) + 1 + k] = inputs.maxwellian(g, 1.0, u, T)
    return np.ascontiguousarray(f), nodes


@pytest.mark.parametrize("dims,R", [((2, 2, 2), 16.5), ((8, 8, 8), 16.5), ((12, 10, 8), 4.2), ((12, 12, 12), 4.8)])
def test_loss_of_concentrated_cells(cuda, gdlib, dims, R):
    torch = cuda
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    f, nodes = _cells(spec, ctx.n_pnt)
    f = np.maximum(f, np.where(f > 0, 1e-25, 0)).astype(np.float32)   # products stay normal numbers
    ft = torch.from_numpy(f).cuda()
    nc = f.shape[1]
    nu = torch.full_like(ft, -1.0)
    ctx.collision(ft, nc, nc, nu, None)
    got = nu.cpu().numpy().astype(np.float64)
    o = Oracle(*dims, R=R)
    ref = o.loss_f64(o.to_box(f))
    assert np.all(got >= 0.0)
    assert np.all(got[nodes, np.arange(len(nodes))] == 0.0)
    full = ref > 0.0
    assert np.max(np.abs(got[full] - ref[full]) / ref[full]) <= 2.2e-6


def test_one_node_cell_is_recorded_as_singular(cuda, gdlib):
    """nu vanishes on the only filled node, so the conservation system is zero."""
    torch = cuda
    spec = gdlib.GridSpec(12, R=4.8)
    ctx = gdlib.Context(spec)
    f = inputs.mixtures(spec.fill(), 40, seed=3)
    rng = np.random.default_rng(8)
    for node in rng.choice(ctx.n_pnt, 40, replace=False):
        g = f.copy()
        g[:, 7] = 0.0
        g[node, 7] = 0.7
        gt = torch.from_numpy(g).cuda()
        ctx.step(gt, 40, 40, gdlib.DT_FIXED, 1e-3)
        with pytest.raises(gdlib.GDError) as e:
            ctx.check()
        assert "singular" in str(e.value) and "cell 7" in str(e.value)
