"""Singular conservation systems are recognised from the size of what the
elimination leaves, not from an exact zero: a cell with all its mass on one node has
a system of rank one, whichever node it is and whatever its value, and gets X = 0
and a record.  Cells with little spread but more nodes than that are solved."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,R", [(8, 16.5), (12, 4.8), (20, 4.8)])
def test_one_node_cells_have_no_correction(cuda, gdlib, n, R):
    torch = cuda
    spec = gdlib.GridSpec(n, R=R)
    ctx = gdlib.Context(spec)
    ns = ctx.n_pnt
    for value, rate in ((1.0, 2.0), (0.7, 1.3), (123.4, 0.37), (1e-3, 3.1)):
        f = torch.diag(torch.full((ns,), value, dtype=torch.float32, device="cuda")).contiguous()
        nu = torch.full((ns, ns), rate, dtype=torch.float32, device="cuda")
        gain = torch.full((ns, ns), 0.21, dtype=torch.float32, device="cuda")
        x = torch.full((ns, 5), -1.0, dtype=torch.float64, device="cuda")
        q = torch.empty((ns, ns), dtype=torch.float64, device="cuda")
        nuc = torch.empty_like(nu)
        ctx.project(f, nu, gain, ns, ns, nuc, q, x)
        with pytest.raises(gdlib.GDError) as e:
            ctx.check()
        assert "singular" in str(e.value) and "cell 0" in str(e.value)
        assert int(torch.count_nonzero(x)) == 0, value
        assert torch.equal(nuc, nu)


@pytest.mark.parametrize("n,T", [(12, 0.05), (20, 0.03), (20, 0.1)])
def test_narrow_cells_are_solved(cuda, gdlib, n, T):
    torch = cuda
    spec = gdlib.GridSpec(n, R=4.8)
    ctx = gdlib.Context(spec)
    g = spec.fill()
    rng = np.random.default_rng(n)
    f = np.stack([inputs.maxwellian(g, 1.0, rng.uniform(-2.0, 2.0, 3), T) for _ in range(40)], 1).astype(np.float32)
    nu = rng.uniform(1.0, 3.0, f.shape).astype(np.float32)
    gain = (f * nu * rng.uniform(0.7, 1.4, f.shape)).astype(np.float32)
    t = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (f, nu, gain)]
    x = torch.zeros((40, 5), dtype=torch.float64, device="cuda")
    q = torch.empty(f.shape, dtype=torch.float64, device="cuda")
    ctx.project(*t, 40, 40, torch.empty_like(t[0]), q, x)
    ctx.check()
    X, Q = x.cpu().numpy(), q.cpu().numpy()
    assert np.all(np.abs(X).max(axis=1) > 0)
    # what is left of the moments: rounding of sums whose terms are I and f nu (1 + X.phi)
    v = np.stack(inputs.node_velocities(g))
    phi = np.vstack([np.ones((1, ctx.n_pnt)), v, (v * v).sum(0, keepdims=True)])
    terms = np.abs(phi) @ (np.abs(gain) + np.abs(f * nu) * (1.0 + (np.abs(X) @ np.abs(phi)).T))
    assert np.all(np.abs(phi @ Q) <= 1e-12 * terms)
