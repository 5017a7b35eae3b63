"""The FP32 gain of distributions whose products leave FP32's range: every output is
the FP64 gain rounded to FP32 within the kernel's error, infinite only where that
exceeds FP32, zero or subnormal where it is below; no output of such a cell is NaN,
and the other cells keep their bits.  Same sums as at ordinary scale, times a power
of two: the tolerance is the one of the ordinary scale (3e-6 in relative L2, 1.2e-5
for one output)."""
import ctypes as C

import numpy as np
import pytest

from gpu_determ_gb300 import inputs
from oracle.pyoracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("dims,R", [((8, 8, 8), 16.5), ((12, 10, 8), 4.2)])
def test_gain_beyond_the_range_of_products(cuda, gdlib, dims, R, noalloc):
    torch = cuda
    spec = gdlib.GridSpec(*dims, R=R)
    ctx = gdlib.Context(spec)
    nc = 21
    f = np.maximum(inputs.mixtures(spec.fill(), nc, seed=6), 1e-6).astype(np.float32)
    o = Oracle(*dims, R=R)
    ref = o.gain_f64(o.to_box(f))
    power = np.zeros(nc, int)
    power[[2, 3, 5, 9]] = 58, 64, 70, -64
    g = np.ldexp(f, power[None, :]).astype(np.float32)

    def gain(x):
        t = torch.from_numpy(np.ascontiguousarray(x)).cuda()
        out = torch.full_like(t, -1.0)
        if noalloc:
            rc = gdlib.lib().gd_gain_noalloc(ctx._h, C.c_void_p(t.data_ptr()), nc, nc, C.c_void_p(out.data_ptr()), None)
            assert rc == 0
        else:
            ctx.collision(t, nc, nc, None, out)
        torch.cuda.synchronize()
        return out.cpu().numpy()

    base, got = gain(f), gain(g)
    keep = power == 0
    assert np.array_equal(got[:, keep], base[:, keep])
    assert not np.isnan(got).any()
    with np.errstate(over="ignore"):
        for c in np.flatnonzero(power):
            want = np.ldexp(ref[:, c], 2 * power[c])
            big = np.finfo(np.float32).max
            sure = np.abs(want / big - 1.0) > 1e-4       # clear of the border itself
            assert np.array_equal(np.isinf(got[sure, c]), want[sure] > big), c
            ok = np.isfinite(got[:, c]) & (want > 1e-30) & (want < big)
            rel = np.abs(got[ok, c] - want[ok]) / want[ok]
            assert rel.size == 0 or rel.max() <= 1.2e-5, c
            # the exactly scaled gain of ordinary size
            assert np.array_equal(got[:, c], np.ldexp(base[:, c].astype(np.float64), 2 * power[c]).astype(np.float32))
