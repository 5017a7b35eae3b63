"""The FP32 gain with all eight reflections of a pair sum at once (the default
gain path wherever its rows fit a CTA) against the FP64 oracle.

Every output is a sum of non-negative FP32 terms: three roundings per pair
product, a contraction chain of at most ~500 weights, runs of at most 64
targets and ~2000 runs.  With independent roundings of half an ulp (6e-8) the
relative error of an output grows with the root of the roundings on its path,
sqrt(3 + 500 + 64 + 2000) 6e-8 = 3e-6, which bounds the relative L2 error; a
single output may lie a few times above."""
import numpy as np
import pytest

from gpu_determ_gb300 import inputs
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


def _gain(gdlib, torch, dims, R, nc, ld, seed):
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    f = inputs.mixtures(spec.fill(), nc, seed=seed)
    ft = torch.full((ctx.n_pnt, ld), float("nan"), dtype=torch.float32, device="cuda")  # padding is not read
    ft[:, :nc] = torch.from_numpy(f).cuda()
    out = [torch.full_like(ft, -1.0) for _ in range(2)]
    for o in out:
        ctx.collision(ft, nc, ld, None, o)
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1])               # bitwise reproducible
    assert bool((out[0][:, nc:] == -1.0).all())      # padding columns untouched
    return f, out[0][:, :nc].cpu().numpy().astype(np.float64)


# lattices with one, two and many orbits per warp, unequal axes, odd cell
# counts around the tile width; 22^3 has more orbits than eight-cell tiles hold
@pytest.mark.parametrize("dims,R,nc,ld", [((2, 2, 2), 16.5, 1, 1), ((4, 2, 6), 16.5, 9, 11), ((8, 8, 8), 16.5, 7, 7),
                                          ((12, 10, 8), 4.2, 8, 8), ((12, 12, 12), 4.8, 65, 67),
                                          ((20, 20, 20), 4.8, 3, 3), ((22, 22, 22), 4.8, 5, 6)])
def test_orbit_gain_matches_oracle(cuda, gdlib, dims, R, nc, ld):
    f, got = _gain(gdlib, cuda, dims, R, nc, ld, seed=sum(dims) + nc)
    o = Oracle(*dims, R=R)
    ref = o.gain_f64(o.to_box(f))
    assert np.linalg.norm(got - ref) <= 3e-6 * np.linalg.norm(ref)
    big = ref > 1e-30   # below, FP32 products are subnormal
    assert np.max(np.abs(got[big] - ref[big]) / ref[big]) <= 1.2e-5


@pytest.mark.parametrize("nc", [1, 40, 1300])
def test_orbit_gain_of_a_cell_does_not_depend_on_its_neighbours(cuda, gdlib, nc):
    """Cells are independent: a non-finite cell stays alone, and a cell's gain
    is the same in every column (chunks of the walk depend on the count only)."""
    torch = cuda
    spec = gdlib.GridSpec(12, R=4.8)
    ctx = gdlib.Context(spec)
    one = torch.from_numpy(inputs.mixtures(spec.fill(), 1, seed=9)).cuda()
    f = one.repeat(1, nc).contiguous()
    if nc > 1:
        f[5, 1] = float("nan")
        f[7, 2] = float("inf")
    out = torch.empty_like(f)
    ctx.collision(f, nc, nc, None, out)
    torch.cuda.synchronize()
    keep = [c for c in range(nc) if c not in (1, 2)] if nc > 1 else [0]
    assert torch.equal(out[:, keep], out[:, :1].expand(-1, len(keep)))
    assert bool(torch.isfinite(out[:, 0]).all())
    if nc > 1:
        assert not bool(torch.isfinite(out[:, 1]).all()) and not bool(torch.isfinite(out[:, 2]).all())


# 1, 4, 105 and 512 orbits (the tiles are 32 orbits by 8 or 32 cells, steps of 16
# orbits); cells around the tile width and, in the last, enough for the wide tile
@pytest.mark.parametrize("dims,R,nc,ld", [((2, 2, 2), 16.5, 1, 1), ((4, 4, 4), 16.5, 8, 9), ((12, 12, 12), 4.8, 33, 33),
                                          ((12, 10, 8), 4.2, 9, 12), ((16, 16, 16), 16.5, 31, 31),
                                          ((16, 16, 16), 16.5, 321, 324)])
def test_folded_loss_matches_oracle(cuda, gdlib, dims, R, nc, ld):
    """The loss with f and b folded by the lattice's reflections.  Each
    character's sum takes chains of 16 products (16 roundings of 6e-8 at most),
    compensated sums of them, three roundings in the fold and one at the end:
    1.3e-6 of the largest frequency among a node's mirrors if all roundings add
    up, and those frequencies differ by a factor below 4; independent roundings
    stay near the root of that count, 3e-7 in relative L2."""
    torch = cuda
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    f = inputs.mixtures(spec.fill(), nc, seed=nc)
    ft = torch.full((ctx.n_pnt, ld), float("nan"), dtype=torch.float32, device="cuda")
    ft[:, :nc] = torch.from_numpy(f).cuda()
    out = [torch.full_like(ft, -1.0) for _ in range(2)]
    for o in out:
        ctx.collision(ft, nc, ld, o, None)
    torch.cuda.synchronize()
    assert torch.equal(out[0], out[1]) and bool((out[0][:, nc:] == -1.0).all())
    got = out[0][:, :nc].cpu().numpy().astype(np.float64)
    o = Oracle(*dims, R=R)
    ref = o.loss_f64(o.to_box(f))
    assert np.max(np.abs(got - ref) / ref) <= 5e-6
    assert np.linalg.norm(got - ref) <= 3e-7 * np.linalg.norm(ref)


# lattices whose gain the FP32 kernel computes on the tensor-core paths too; up
# to 1216 cells of eight (tiles x 152) run in chunks of the walk, then in one
@pytest.mark.parametrize("dims,R,nc,ld", [((8, 8, 8), 16.5, 1216, 1216), ((12, 10, 8), 4.2, 7, 9),
                                          ((12, 12, 12), 4.8, 65, 67), ((22, 22, 22), 4.8, 3, 3)])
def test_orbit_gain_serves_the_tensor_core_paths(cuda, gdlib, dims, R, nc, ld):
    """The FP32 path's gain bit for bit; a cell with a non-finite f gets NaN
    alone; a cell scaled by 2^+-50, whose products would leave FP32's range,
    gets the exactly scaled gain, rounded once."""
    torch = cuda
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    f = torch.full((ctx.n_pnt, ld), float("nan"), dtype=torch.float32, device="cuda")
    # no product of f itself is subnormal
    f[:, :nc] = torch.from_numpy(np.maximum(inputs.dirichlet_mixtures(spec.fill(), nc, seed=5), 1e-12)).cuda()
    ref = torch.full_like(f, -1.0)
    ctx.collision(f, nc, ld, None, ref)
    g = f.clone()
    g[3, 1] = float("inf")
    g[:, 2] *= 2.0 ** -50
    g[:, 0] *= 2.0 ** 50
    paths = [gdlib.GAIN_PAIR_TC] + ([gdlib.GAIN_CMATRIX_BF16X3] if ctx.n_pnt >= 512 else [])
    for path in paths:
        ctx.set_gain_path(path)
        out = [torch.full_like(f, -1.0) for _ in range(2)]
        for x, o in zip((f, g), out):
            ctx.collision(x, nc, ld, None, o)
        ctx.check()
        assert torch.equal(out[0], ref)
        assert torch.equal(out[1][:, 3:], ref[:, 3:]) and bool(torch.isnan(out[1][:, 1]).all())
        r = ref.cpu().numpy().astype(np.float64)
        assert np.array_equal(out[1][:, 0].cpu().numpy(), np.ldexp(r[:, 0], 100).astype(np.float32))
        assert np.array_equal(out[1][:, 2].cpu().numpy(), np.ldexp(r[:, 2], -100).astype(np.float32))
