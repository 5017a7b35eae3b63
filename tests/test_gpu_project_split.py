"""The projection's split of lines and cells over the chip (one, eight or 32
cells per warp, one to eight CTAs per group of cells, by the number of SMs and the
lattice) over cell counts where it changes: every split sums the same FP64 terms in another order, so a cell's Q agrees between batches to n_pnt
roundings, 1e-12 of its largest I.  An empty cell is left alone without a
record, a cell whose system is singular is recorded."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs

pytestmark = pytest.mark.gpu


def _project(torch, ctx, f, nu, gain, nc):
    t = [torch.from_numpy(np.ascontiguousarray(np.tile(a, (1, -(-nc // a.shape[1])))[:, :nc])).cuda()
         for a in (f, nu, gain)]
    nuc = torch.empty_like(t[0])
    q = torch.empty(t[0].shape, dtype=torch.float64, device="cuda")
    x = torch.zeros((nc, 5), dtype=torch.float64, device="cuda")
    ctx.project(*t, nc, nc, nuc, q, x)
    torch.cuda.synchronize()
    return nuc.cpu().numpy(), q.cpu().numpy()


@pytest.mark.parametrize("dims,R", [((8, 8, 8), 4.8), ((2, 2, 4), 16.5), ((10, 12, 14), 4.4)])
def test_batches_around_the_splits_agree(cuda, gdlib, dims, R):
    torch = cuda
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    rng = np.random.default_rng(7)
    f = inputs.mixtures(spec.fill(), 7, seed=3)
    nu = rng.uniform(1.0, 3.0, f.shape).astype(np.float32)
    gain = (f * nu * rng.uniform(0.7, 1.4, f.shape)).astype(np.float32)
    ref_nu, ref_q = _project(torch, ctx, f, nu, gain, 7)
    scale = gain.astype(np.float64).max(axis=0)
    for nc in (sms // 2 + 1, sms, sms + 1, 2 * sms + 5, 4 * sms, 4 * sms + 1, 8 * sms, 8 * sms + 1, 20 * sms + 3):
        got_nu, got_q = _project(torch, ctx, f, nu, gain, nc)
        ctx.check()
        cols = np.arange(nc) % 7
        assert np.max(np.abs(got_q - ref_q[:, cols]) / scale[cols]) <= 1e-12, nc
        assert np.allclose(got_nu, ref_nu[:, cols], rtol=1.3e-7, atol=0.0), nc


@pytest.mark.parametrize("nc", [3, 200, 700, 1300])
def test_empty_and_singular_cells(cuda, gdlib, nc):
    torch = cuda
    spec = gdlib.GridSpec(8, R=4.8)
    ctx = gdlib.Context(spec)
    f = inputs.mixtures(spec.fill(), nc, seed=1)
    nu = np.full_like(f, 2.0)
    gain = (f * 2.5).astype(np.float32)
    f[:, 1] = 0.0
    gain[:, 1] = 0.0
    _, q = _project(torch, ctx, f, nu, gain, nc)
    ctx.check()                       # the empty cell is no fault
    assert not q[:, 1].any() and np.abs(q[:, 2]).max() > 0
    f[1:, 2] = 0.0                    # all mass on one node: a system of rank one
    _project(torch, ctx, f, nu, gain, nc)
    with pytest.raises(gdlib.GDError) as e:
        ctx.check()
    assert "singular" in str(e.value) and "cell 2" in str(e.value)
    ctx.check()
