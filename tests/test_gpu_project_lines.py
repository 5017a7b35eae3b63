"""The projection's per-line sums over few and many cells (one, eight or 32
cells per warp, one to eight CTAs per group of cells): X, nu' and Q against the
FP64 projection of the same FP32 inputs, moments of Q at rounding level.

Sums of n_pnt terms in FP64 (1.1e-16) lose at most n_pnt roundings, so B and A
are good to 1e-12 of the sums of absolute terms; X is B / A with B at least
1e-3 of those sums here, so 1e-8 holds with room, and Q is within that of
I and f nu."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,R,nc,ld", [((4, 2, 2), 16.5, 1, 1), ((12, 10, 8), 4.2, 8, 9), ((12, 12, 12), 4.8, 9, 9),
                                          ((12, 12, 12), 4.8, 513, 515), ((8, 8, 8), 16.5, 512, 512),
                                          ((6, 6, 6), 16.5, 6000, 6000)])
def test_project_over_cell_counts(cuda, gdlib, dims, R, nc, ld):
    torch = cuda
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    g = spec.fill()
    rng = np.random.default_rng(nc)
    base = inputs.mixtures(g, min(nc, 64), seed=3)
    f = np.tile(base, (1, -(-nc // base.shape[1])))[:, :nc] * rng.uniform(0.5, 2.0, nc).astype(np.float32)
    nu = rng.uniform(1.0, 3.0, f.shape).astype(np.float32)
    gain = (f * nu * rng.uniform(0.7, 1.4, f.shape)).astype(np.float32)
    t = [torch.full((ctx.n_pnt, ld), float("nan"), dtype=torch.float32, device="cuda") for _ in range(3)]
    for a, b in zip(t, (f, nu, gain)):
        a[:, :nc] = torch.from_numpy(b).cuda()
    nuc = torch.full_like(t[0], -1.0)
    q = torch.full(t[0].shape, -1.0, dtype=torch.float64, device="cuda")
    x = torch.zeros((nc, 5), dtype=torch.float64, device="cuda")
    ctx.project(*t, nc, ld, nuc, q, x)
    torch.cuda.synchronize()
    ctx.check()
    assert bool((nuc[:, nc:] == -1.0).all()) and bool((q[:, nc:] == -1.0).all())
    v = np.stack(inputs.node_velocities(g))
    phi = np.vstack([np.ones((1, ctx.n_pnt)), v, (v * v).sum(0, keepdims=True)])
    X = x.cpu().numpy()
    f64, nu64, g64 = (a.astype(np.float64) for a in (f, nu, gain))
    ref_nuc = nu64 * (1.0 + (X @ phi).T)
    ref_q = g64 - f64 * ref_nuc
    assert np.allclose(nuc[:, :nc].cpu().numpy(), ref_nuc, rtol=1.3e-7, atol=0.0)
    assert np.max(np.abs(q[:, :nc].cpu().numpy() - ref_q) / g64.max(axis=0)) <= 1e-12
    fn = f64 * nu64
    A = np.einsum("ic,ki,li->ckl", fn, phi, phi)
    B = (phi @ (g64 - fn)).T
    sol = np.linalg.solve(A, B[:, :, None])[:, :, 0]
    assert np.max(np.abs(X - sol) / np.abs(sol).max(axis=1, keepdims=True)) <= 1e-8
    mom = np.abs(phi @ q[:, :nc].cpu().numpy())
    assert np.all(mom <= 1e-12 * (np.abs(phi) @ np.abs(g64)))
