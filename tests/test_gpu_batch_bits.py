"""A cell's results do not depend on the batch that it is in: alone, in a shard of
the batch or in the whole batch (more cells than a launch takes at once among
them), at an odd place in it, they are the same bits.  So a batch split over
ranks repeats the unsplit one."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs

pytestmark = pytest.mark.gpu


def _batch(torch, spec, nc, seed=2):
    f = inputs.mixtures(spec.fill(), 41, seed=seed)
    return torch.from_numpy(np.ascontiguousarray(np.tile(f, (1, -(-nc // 41)))[:, :nc])).cuda()


# 8-cell and 4-cell tiles; batches below and above a CTA per SM; 20^3: two launches
@pytest.mark.parametrize("n,nc", [(8, 1300), (12, 1300), (20, 1000), (22, 41)])
def test_gain_bits_do_not_depend_on_the_batch(cuda, gdlib, n, nc):
    torch = cuda
    spec = gdlib.GridSpec(n, R=4.8)
    ctx = gdlib.Context(spec)
    f = _batch(torch, spec, nc)
    for path in (gdlib.GAIN_PAIR, gdlib.GAIN_PAIR_TC, gdlib.GAIN_CMATRIX_BF16X3):
        if path == gdlib.GAIN_CMATRIX_BF16X3 and n == 22:
            continue      # as GAIN_PAIR_TC on this lattice
        ctx.set_gain_path(path)
        whole = torch.empty_like(f)
        ctx.collision(f, nc, nc, None, whole)
        for first, count in ((0, 1), (5, 1), (3, 9), (0, nc // 2), (nc // 2, nc - nc // 2)):
            part = f[:, first:first + count].contiguous()
            out = torch.empty_like(part)
            ctx.collision(part, count, count, None, out)
            assert torch.equal(out, whole[:, first:first + count]), (path, first, count)
        ctx.check()


@pytest.mark.parametrize("n,nc", [(2, 700), (6, 2500), (8, 2500), (12, 1300), (20, 1100), (24, 600)])
def test_projection_bits_do_not_depend_on_the_batch(cuda, gdlib, n, nc):
    """nu', Q, X and the step's moments over cell counts on both sides of every
    split of the work (a line per thread; 8, 16 or 32 cells per warp)."""
    torch = cuda
    spec = gdlib.GridSpec(n, R=4.8 if n > 2 else 16.5)
    ctx = gdlib.Context(spec)
    rng = np.random.default_rng(n)
    f = _batch(torch, spec, nc)
    nu = torch.from_numpy(rng.uniform(1.0, 3.0, f.shape).astype(np.float32)).cuda()
    gain = f * nu * torch.from_numpy(rng.uniform(0.7, 1.4, f.shape).astype(np.float32)).cuda()

    def project(first, count):
        part = [a[:, first:first + count].contiguous() for a in (f, nu, gain)]
        out = (torch.empty_like(part[0]), torch.empty(part[0].shape, dtype=torch.float64, device="cuda"),
               torch.empty((count, 5), dtype=torch.float64, device="cuda"))
        ctx.project(*part, count, count, *out)
        return out

    def moments(first, count):
        g = f[:, first:first + count].clone(memory_format=torch.contiguous_format)
        m5 = torch.empty((count, 5), dtype=torch.float64, device="cuda")
        ctx.step(g, count, count, gdlib.DT_FIXED, 1e-3, m5=m5)
        return g, m5

    whole, stepped = project(0, nc), moments(0, nc)
    for first, count in ((0, 1), (7, 2), (1, 40), (2, 200), (3, 350), (0, nc // 2), (nc // 2, nc - nc // 2)):
        cols = slice(first, first + count)
        got = project(first, count)
        assert torch.equal(got[0], whole[0][:, cols]) and torch.equal(got[1], whole[1][:, cols]), (first, count)
        assert torch.equal(got[2], whole[2][cols]), (first, count)
        got = moments(first, count)
        assert torch.equal(got[0], stepped[0][:, cols]) and torch.equal(got[1], stepped[1][cols]), (first, count)


# one orbit; tiles of 4 and of 16 orbits on both sides of the change
@pytest.mark.parametrize("n,nc", [(2, 50), (12, 1300), (20, 300)])
def test_loss_bits_do_not_depend_on_the_batch(cuda, gdlib, n, nc):
    torch = cuda
    spec = gdlib.GridSpec(n, R=4.8 if n > 2 else 16.5)
    ctx = gdlib.Context(spec)
    f = _batch(torch, spec, nc)
    whole = torch.empty_like(f)
    ctx.collision(f, nc, nc, whole, None)
    for first, count in ((0, 1), (5, 9), (3, nc // 2), (nc // 2, nc - nc // 2)):
        part = f[:, first:first + count].contiguous()
        out = torch.empty_like(part)
        ctx.collision(part, count, count, out, None)
        assert torch.equal(out, whole[:, first:first + count]), (first, count)
