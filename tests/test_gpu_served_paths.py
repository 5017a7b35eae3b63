"""Gain paths whose gain the FP32 kernel computes (GD_GAIN_PAIR_TC, and
GD_GAIN_CMATRIX_BF16X3 from 512 nodes on): choosing one builds no table that no
result uses, the weight table is there for the call that reads it, and the injected
time-out is one of the kernel that runs."""
import pytest

from gpu_determ_gb300 import inputs

pytestmark = pytest.mark.gpu


def test_choosing_a_served_path_takes_no_memory(cuda, gdlib):
    torch = cuda
    ctx = gdlib.Context(gdlib.GridSpec(20, R=4.8))
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for path in (gdlib.GAIN_PAIR_TC, gdlib.GAIN_CMATRIX_BF16X3):
        ctx.set_gain_path(path)     # a weight table of 0.6 GB, a loss matrix of 53 MB otherwise
        assert free - torch.cuda.mem_get_info()[0] <= 8 << 20, path
    ctx.set_gain_path(gdlib.GAIN_PAIR_TC)
    assert ctx.pair_tc_table()["wh"].any()
    ctx.set_gain_path(gdlib.GAIN_PAIR)
    with pytest.raises(gdlib.GDError) as e:
        ctx.pair_tc_table()
    assert e.value.code == 4


@pytest.mark.parametrize("late", [False, True])
@pytest.mark.parametrize("cells", [1, 300])
def test_timed_out_wait_of_the_fp32_gain_is_reported_once(cuda, gdlib, cells, late):
    """The kernel's own bounded wait runs out with its first copies in flight:
    they land before the CTA leaves, and the next call is bitwise the clean one."""
    torch = cuda
    spec = gdlib.GridSpec(12, R=4.8)
    ctx = gdlib.Context(spec)
    f = torch.from_numpy(inputs.mixtures(spec.fill(), cells, seed=4)).cuda()
    ctx.set_gain_path(gdlib.GAIN_CMATRIX_BF16X3)
    nu0, g0, nu1, g1, nu2, g2 = (torch.empty_like(f) for _ in range(6))
    ctx.collision(f, cells, cells, nu0, g0)
    ctx.check()
    ctx.inject_timeout(256, late=late)
    ctx.collision(f, cells, cells, nu1, g1)
    with pytest.raises(gdlib.GDError) as e:
        ctx.check()
    assert e.value.code == 2 and "FP32 gain kernel" in str(e.value) and "timed out" in str(e.value)
    ctx.check()
    assert torch.equal(nu1, nu0)       # the loss is not the stalled kernel's
    ctx.collision(f, cells, cells, nu2, g2)
    ctx.check()
    assert torch.equal(nu2, nu0) and torch.equal(g2, g0)
    ctx.set_gain_path(gdlib.GAIN_PAIR_TC)
    with pytest.raises(gdlib.GDError) as e:
        ctx.inject_timeout(256)
    assert e.value.code == 4


@pytest.mark.parametrize("dims,R", [((2, 2, 2), 16.5), ((4, 2, 6), 16.5), ((12, 12, 12), 4.8)])
def test_gain_work(cuda, gdlib, dims, R):
    """The executed operations are at most those of the whole class boxes, and at
    least one update for every pair of in-sphere nodes (its pair sum's shell holds the
    pair itself); a batch beyond a launch's scratch takes more launches."""
    ctx = gdlib.Context(gdlib.GridSpec(*dims, R=R))
    flop, launches = ctx.gain_work(8)
    i = ctx.info
    assert ctx.n_pnt ** 2 <= flop <= 7 * i["pair_products"] + 2 * i["contraction_terms"] + i["scatter_terms"]
    assert launches in (3, 4) and ctx.gain_work(1)[1] == launches
    assert ctx.gain_work(1 << 28)[1] > launches
    ctx.use_general_kernels()
    assert ctx.gain_work(8)[0] >= flop
