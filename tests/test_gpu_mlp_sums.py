"""The network's per-cell scale: one FP32 chain of additions over the nodes in
order, whatever the copies ahead of it look like.  With all weights zero and the
decoder's bias one, the output is the squared scale times the gain, so the scale
can be compared bit for bit with the same chain on the host."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# rows around a stage of 128 and around the whole ring of 1024; full and partial
# blocks of 32 cells, strides and starts with and without 16-byte alignment
@pytest.mark.parametrize("n", [1, 31, 128, 129, 300, 1100])
@pytest.mark.parametrize("batch,ld,first", [(1, 1, 0), (33, 33, 0), (64, 64, 0), (64, 68, 1), (96, 100, 4)])
def test_scale_is_the_ordered_sum(cuda, gdlib, n, batch, ld, first):
    torch = cuda
    net = gdlib.Mlp(n, n, 128, flags=gdlib.MLP_SCALE_INPUT | gdlib.MLP_SCALE_OUTPUT, seed=1)
    p = np.zeros_like(net.get_params())
    p[-net.info["n_out_padded"]:] = 1.0
    net.set_params(p)
    rng = np.random.default_rng(n + batch)
    x = rng.random((n, ld + first), dtype=np.float32) + 0.1
    xt = torch.from_numpy(x).cuda()[:, first:]
    y = torch.zeros((n, ld), dtype=torch.float32, device="cuda")
    net.forward(xt, ld + first, batch, y, ld)
    net.check()
    s = np.zeros(batch, dtype=np.float32)
    for i in range(n):
        s += x[i, first:first + batch]
    s /= np.float32(n)
    assert np.array_equal(y.cpu().numpy()[:, :batch], np.repeat((s * s)[None], n, axis=0))
    net.close()
