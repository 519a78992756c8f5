"""The band convolutions of the network's forward pass against the same layers as im2col GEMMs of the same tensor cores
(octo_gemm_bf16): K is taken 16 at a time, tap by tap and channel by channel, and where the GEMM would split K its parts
are summed in order, so every layer's fp32 sums, and with them the bf16 activations and the output, agree to the bit.
Infinities and NaN too: an input pixel reaches the outputs whose nine taps hold it and no other."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


def _parts(M, cin):
    """Parts of K of a layer of M pixels: enough that the 128-row tiles fill the GPU twice, no shorter than 128."""
    tiles, chunks = (M + 127) // 128, (9 * cin + 63) // 64
    return max(1, min(chunks // 2, (296 + tiles - 1) // tiles)) if tiles < 148 and chunks >= 4 else 1


def _layer(x, w, b, relu, head):
    import torch
    from octo_b200 import _lib
    B, H, W, cin = x.shape
    cout, M = w.shape[0], B * H * W
    d = _lib.OctoGemmDesc()
    d.M, d.N, d.K, d.a_mode, d.H, d.W, d.C = M, cout, 9 * cin, 1, H, W, cin
    d.A, d.B, d.ldb, d.splits = x.data_ptr(), w.data_ptr(), 9 * cin, 1 if head else _parts(M, cin)
    out = torch.empty((d.splits, M, cout), device="cuda")
    d.out, d.ldc = out.data_ptr(), cout
    rc = _lib.lib().octo_gemm_bf16(0, C.byref(d), C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _lib.OCTO_OK, rc
    v = out[0]
    for z in range(1, out.shape[0]):
        v = v + out[z]
    v = v + b
    if relu:
        v = torch.where(v > 0, v, torch.zeros_like(v))  # a NaN becomes zero, as in the maximum with zero
    return (v if head else v.to(torch.bfloat16)).reshape(B, H, W, cout)


def _forward(params, x):
    import torch
    from oracle.cnn_oracle import LAYERS
    ws, off = [], 0
    p = torch.from_numpy(params).cuda()
    for cin, cout, _, _ in LAYERS:
        n = cout * 9 * cin
        ws.append((p[off:off + n].to(torch.bfloat16).reshape(cout, 3, 3, cin).contiguous(), p[off + n:off + n + cout]))
        off += n + cout

    def conv(k, t):
        return _layer(t.contiguous(), *ws[k], LAYERS[k][3], k == len(LAYERS) - 1)

    def pool(t):
        f = t.float()
        return (0.25 * (f[:, 0::2, 0::2] + f[:, 0::2, 1::2] + f[:, 1::2, 0::2] + f[:, 1::2, 1::2])).to(torch.bfloat16)

    def up(t, skip):
        return torch.cat([t.repeat_interleave(2, 1).repeat_interleave(2, 2), skip], 3)

    s1 = conv(1, conv(0, x))
    s2 = conv(3, conv(2, pool(s1)))
    s3 = conv(5, conv(4, pool(s2)))
    t = conv(6, pool(s3))
    for k, skip in ((7, s3), (8, s2), (9, s1)):
        t = conv(k, up(t, skip))
    return conv(10, t)[..., :2]


def _check(B, H, W, odd):
    import numpy as np
    import torch
    from test_gpu_cnn import _inputs
    from octo_b200.learned import FieldCorrectionNet
    net = FieldCorrectionNet(H, W, max_batch=B, seed=11)
    p = net.get_params()
    p = p + (0.01 * np.random.default_rng(3).standard_normal(p.size)).astype(np.float32)
    net.set_params(p)
    x, _, _ = _inputs(B, H, W, 5)
    if odd:  # inside, on the last column, on the first row, in the last pixel
        x[0, H // 2, W // 2, 0] = float("inf")
        x[0, 3, W - 1, 1] = float("-inf")
        x[B - 1, 0, 5, 0] = float("nan")
        x[B - 1, H - 1, W - 1, 2] = float("inf")
    got, want = net.forward(x), _forward(p, x)
    net.close()
    assert torch.equal(got.isnan(), want.isnan())
    same = (got == want) | want.isnan()
    assert bool(same.all()), (int((~same).sum()), same.numel(), float((got - want)[~same].abs().max()))


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("B,H,W", [(74, 128, 128), (400, 64, 48)])
def test_layers_whose_tiles_fill_the_device(B, H, W, odd):
    _check(B, H, W, odd)


@pytest.mark.parametrize("odd", [False, True])
@pytest.mark.parametrize("B,H,W", [(20, 48, 48), (1, 48, 48), (64, 32, 32), (1, 16, 16), (5, 40, 24), (3, 16, 64),
                                   (70, 48, 48)])
def test_layers_in_parts(B, H, W, odd):
    _check(B, H, W, odd)


def test_more_images_than_a_grid_axis_takes():
    _check(65537, 16, 16, False)


@pytest.mark.parametrize("W", [344, 512, 1024, 2304])
def test_images_too_wide_for_bands(W):
    """From 344 columns on the widest decoder layer's band no longer fits shared memory and it runs as a GEMM, split over
    K; at 1024 half of the layers do, at 2304 all of them, the pooled ones on a pooled copy of their input."""
    _check(2, 16, W, True)
