"""The network's GEMM tiles and launches at the sizes where their choice
changes, against the FP64 oracle with the same BF16 rounding points: a K of at
most eight steps (narrow tiles, two CTAs per SM) and a longer one, whose tiles
are 32, 64, 128 or 256 columns by the batch; the weights' gradients of all
layers in one launch; the transposes that the epilogues, the input's copy, the
loss gradient and Adam write.  Tolerances as for the other gradients: FP32 sums
in another order and single BF16 roundings the other way, 2e-3."""
import numpy as np
import pytest

from oracle import mlp_ref as M

pytestmark = pytest.mark.gpu
FLAGS = M.SCALE_INPUT | M.SCALE_OUTPUT


def _rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("n_in,n_out,B", [
    (70, 130, 64),       # every K short
    (600, 33, 512),      # the first layer's K long, the batch's short
    (600, 200, 576),     # both long, 32 columns
    (640, 64, 2560),     # 64 columns in the first layer
    (600, 700, 5120),    # 128
    (600, 64, 9984),     # 256
])
def test_gradients_after_an_adam_step(gdlib, cuda, n_in, n_out, B):
    torch = cuda
    rng = np.random.default_rng(B)
    x = rng.uniform(0.05, 1.0, (n_in, B)).astype(np.float32)
    t = rng.normal(0, 1.0, (n_out, B)).astype(np.float32)
    xd = torch.zeros((n_in, B + 5), dtype=torch.float32, device="cuda")
    td = torch.zeros((n_out, B + 1), dtype=torch.float32, device="cuda")
    xd[:, :B], td[:, :B] = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    net = gdlib.Mlp(n_in, n_out, batch_cap=B, flags=FLAGS, seed=3)
    net.set_params(M.init_like_library(n_in, n_out, seed=11))
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    row = torch.zeros(B, dtype=torch.float32, device="cuda")
    net.train_step(xd, B + 5, td, B + 1, B, lr=1e-3)           # the BF16 copies are Adam's from here on
    net.train_step(xd, B + 5, td, B + 1, B, lr=0.0, loss=loss)
    g = net.get_grads()
    net.loss(xd, B + 5, td, B + 1, B, row)
    net.check()
    p = net.get_params()
    ref_loss, _, ref = M.loss_and_grads(M.unpack(p, n_in, n_out), x, t, FLAGS, n_out, bf16=True)
    assert float(loss.item()) == pytest.approx(ref_loss, rel=2e-3)
    assert float(loss.item()) == pytest.approx(float(row.double().mean().item()), rel=1e-6)
    for k, ((gw, gb), (rw, rb)) in enumerate(zip(M.unpack(g, n_in, n_out), ref)):
        assert _rel(gw, rw) < 2e-3, f"layer {k} weights"
        assert _rel(gb, rb) < 2e-3, f"layer {k} bias"
    net.close()
