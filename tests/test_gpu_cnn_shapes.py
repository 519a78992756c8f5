"""The training step's data-movement kernels at their edges: pixel counts that are no multiple of 8 at the coarse
levels, images smaller than a block's tile, rows that straddle tiles, one image and several, with and without a mask;
every gradient tensor against the CPU oracle.  2e-2: where fp32 and float64 sums round to neighbouring bf16 values an
entry is 2^-8 off, and a ReLU whose input is within that of zero switches a pixel's whole share of a tensor, one in
about 2^8 of the some hundred pixels that the coarsest gradients here average over (the larger images of
test_gpu_cnn.py hold 1e-2)."""
import numpy as np
import pytest

from test_gpu_cnn import _inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,W,masked", [(1, 16, 16, True), (13, 16, 24, True), (11, 24, 16, False), (2, 40, 48, True)])
def test_gradients_at_odd_sizes(B, H, W, masked):
    from oracle import cnn_oracle as co
    from octo_b200.learned import FieldCorrectionNet
    net = FieldCorrectionNet(H, W, max_batch=B, seed=11)
    p = net.get_params()
    p = p + (0.01 * np.random.default_rng(3).standard_normal(p.size)).astype(np.float32)
    net.set_params(p)
    xb, t, mask = _inputs(B, H, W, 5)
    mask = mask if masked else None
    loss, g = net.train_step(xb, t, mask, update=False, want_grads=True)
    ref = co.Net(p.astype(np.float64), rounding=True)
    loss_ref, g_ref = ref.loss_and_grads(xb.float().cpu().numpy().astype(np.float64), t.cpu().numpy().astype(np.float64),
                                         None if mask is None else mask.cpu().numpy())
    assert abs(loss / loss_ref - 1) < 2e-3, (loss, loss_ref)
    off = 0
    for k, (cin, cout, _, _) in enumerate(co.LAYERS):
        live = 2 if cout == 8 else cout  # the head's unused channels carry no loss
        n = cout * 9 * cin
        for a, b in ((g[off:off + live * 9 * cin], g_ref[off:off + live * 9 * cin]),
                     (g[off + n:off + n + live], g_ref[off + n:off + n + live])):
            assert np.linalg.norm(a - b) <= 2e-2 * np.linalg.norm(b), (k, np.linalg.norm(a - b) / np.linalg.norm(b))
        off += n + cout
    net.close()


@pytest.mark.parametrize("B,H,W", [(20, 48, 48), (64, 32, 32), (64, 16, 16), (3, 16, 64)])
def test_forward_of_bands_that_fill_shared_memory(B, H, W):
    """Batches at which the widest decoder layer takes bands of up to 226 KB (one CTA an SM), and small ones."""
    from oracle import cnn_oracle as co
    from octo_b200.learned import FieldCorrectionNet
    net = FieldCorrectionNet(H, W, max_batch=B, seed=11)
    p = net.get_params()
    p = p + (0.01 * np.random.default_rng(3).standard_normal(p.size)).astype(np.float32)
    net.set_params(p)
    xb, _, _ = _inputs(B, H, W, 5)
    out = net.forward(xb).cpu().numpy()
    ref = co.Net(p.astype(np.float64), rounding=True).forward(xb.float().cpu().numpy().astype(np.float64))[..., :2]
    assert np.linalg.norm(out - ref) <= 1e-2 * np.linalg.norm(ref)  # the bound of test_gpu_cnn.py
    net.close()


@pytest.mark.parametrize("W", [344, 1024, 2304])
def test_gradients_where_no_band_fits(W):
    """Wide images, whose forward layers and input gradients run as GEMMs: one, half of them, all."""
    test_gradients_at_odd_sizes(1, 16, W, True)
