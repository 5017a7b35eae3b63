"""A bounded wait that runs out in an epilogue, while copies and MMAs are in flight:
the CTA leaves when these are done, the time-out is reported once by the check, and
the next call is bitwise the clean one.  Sizes with a K loop longer than the
pipeline's stages, and with more tiles than CTAs."""
import pytest

from gpu_determ_gb300 import inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,batch", [(12, 64), (20, 1024), (20, 4096)])
@pytest.mark.parametrize("polls", [1, 300])
def test_late_timeout_of_a_network_gemm(cuda, gdlib, n, batch, polls):
    torch = cuda
    spec = gdlib.GridSpec(n, R=4.8)
    f = torch.from_numpy(inputs.mixtures(spec.fill(), 64, seed=4)).cuda().repeat(1, batch // 64).contiguous()
    net = gdlib.Mlp(f.shape[0], f.shape[0], batch_cap=batch)
    y0, y1, y2 = (torch.empty_like(f) for _ in range(3))
    net.forward(f, batch, batch, y0, batch)
    net.check()
    net.inject_timeout(polls, late=True)
    net.forward(f, batch, batch, y1, batch)
    with pytest.raises(gdlib.GDError) as e:
        net.check()
    assert e.value.code == 2 and "timed out" in str(e.value)
    net.check()
    net.forward(f, batch, batch, y2, batch)
    net.check()
    assert torch.equal(y2, y0)
    with pytest.raises(gdlib.GDError):
        net.inject_timeout(0, late=True)


@pytest.mark.parametrize("cells", [64, 300])
def test_late_timeout_of_the_loss_gemm(cuda, gdlib, cells):
    torch = cuda
    spec = gdlib.GridSpec(12, R=4.8)
    ctx = gdlib.Context(spec)
    f = torch.from_numpy(inputs.mixtures(spec.fill(), cells, seed=4)).cuda()
    ctx.set_gain_path(gdlib.GAIN_CMATRIX_BF16)
    nu0, nu1, nu2, g = (torch.empty_like(f) for _ in range(4))
    ctx.collision(f, cells, cells, nu0, None)
    ctx.check()
    ctx.inject_timeout(300, late=True)
    ctx.collision(f, cells, cells, nu1, g)    # the gain kernel sees the record and does no work
    with pytest.raises(gdlib.GDError) as e:
        ctx.check()
    assert e.value.code == 2 and "timed out" in str(e.value)
    ctx.check()
    ctx.collision(f, cells, cells, nu2, None)
    ctx.check()
    assert torch.equal(nu2, nu0)
