"""The collision-matrix gain's tiles of 16 cells under eight reflections: cell
counts around a tile and a pair of tiles, and more cells than one group of
tiles whose rows stay in L2.  Cells are independent and every row of a tile is
accumulated in the same order, so a cell's gain is bitwise the same in any
batch; against FP64 the operands' rounding bounds it."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,tol", [(0, 2e-3), (1, 1e-5)])
@pytest.mark.parametrize("dims,nc", [((8, 8, 8), 1), ((8, 8, 8), 16), ((12, 10, 8), 17), ((8, 8, 8), 33)])
def test_tile_edges(cuda, gdlib, dims, nc, mode, tol):
    torch = cuda
    spec = gdlib.GridSpec(*dims, R=4.2)
    ctx = gdlib.Context(spec)
    f = inputs.mixtures(spec.fill(), 40, seed=nc)
    all_cells = torch.from_numpy(f).cuda()
    cm = gdlib.CollisionMatrix(ctx, mode)
    base = torch.full_like(all_cells, -1.0)
    cm.gain(all_cells, 40, 40, base)
    ld = nc + 3
    ft = torch.full((ctx.n_pnt, ld), float("nan"), device="cuda")   # padding is not read
    ft[:, :nc] = all_cells[:, 7:7 + nc]
    out = torch.full_like(ft, -1.0)
    cm.gain(ft, nc, ld, out)
    ctx.check()
    assert torch.equal(out[:, :nc], base[:, 7:7 + nc])
    assert bool((out[:, nc:] == -1.0).all())
    o = Oracle(*dims, R=4.2)
    ref = o.gain_f64(o.to_box(f))
    assert np.linalg.norm(base.cpu().numpy() - ref) <= tol * np.linalg.norm(ref)
    cm.close()
    ctx.close()


def test_groups_of_tiles(cuda, gdlib):
    """12^3 (840 nodes): 2000 cells' rows are 82 MB in one BF16 pass, two groups."""
    torch = cuda
    spec = gdlib.GridSpec(12, R=4.8)
    ctx = gdlib.Context(spec)
    cm = gdlib.CollisionMatrix(ctx, 0)
    f = torch.from_numpy(inputs.mixtures(spec.fill(), 100, seed=3)).cuda()
    out = torch.zeros_like(f)
    cm.gain(f, 100, 100, out)
    many = f.repeat(1, 20).contiguous()
    got = torch.full_like(many, -1.0)
    cm.gain(many, 2000, 2000, got)
    assert torch.equal(got, out.repeat(1, 20))
    cm.close()
    ctx.close()
