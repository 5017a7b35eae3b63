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
