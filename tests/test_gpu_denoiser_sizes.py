"""The tcgen05 convolutions and the weight gradients at the sizes where their
pipelines can go wrong: images of one 8x8 block, rows shorter and longer than
a 128-pixel segment, fewer rows than the ring of stages or the ring of
accumulators holds, more rows than one pass of either, several images.

Bars: those of test_gpu_denoiser.py for the same comparisons (tcgen05 against
mma.sync: max 1e-2 and rms 5e-4 of the scale; gradients in the linear regime:
relative L2 error at most 2e-2 and cosine at least 0.9998 per layer), for the
same reason: products are added in FP32 in another order, and a stored value
may round to the neighbouring BF16.
"""
import ctypes

import numpy as np
import pytest
import torch

import arbor_b200 as ab
from test_gpu_denoiser import SPEC, Net, random_inputs, reference_forward, to_dev_bf16, unpack

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 8), (136, 8), (8, 264), (128, 40), (264, 104), (1288, 16)])
def test_forward_sizes(cuda, w, h):
    net = Net(1, w, h, seed=w + h)
    try:
        feat, noisy, _ = random_inputs(1, w, h, seed=3)
        f, n = to_dev_bf16(feat), noisy.contiguous().cuda()
        outs = {}
        for tc in (1, 0):
            assert net.lib.arbor_denoiser_set_backend(net.h, tc) == ab.OK
            out = torch.full((h * w * 4,), float("nan"), device="cuda")
            assert net.lib.arbor_denoiser_infer(net.h, f.data_ptr(), n.data_ptr(), out.data_ptr(), w, h) == ab.OK, ab.last_error()
            assert net.lib.arbor_denoiser_check(net.h) == ab.OK, ab.last_error()
            outs[tc] = out.cpu().view(h, w, 4)
        assert torch.isfinite(outs[1]).all() and (outs[1][..., 3] == 1.0).all()
        err, scale = (outs[1] - outs[0]).abs(), outs[0].abs().max().item()
        assert err.max().item() <= 1e-2 * max(1.0, scale)
        assert err.pow(2).mean().sqrt().item() <= 5e-4 * max(1.0, scale)
    finally:
        net.close()


@pytest.mark.parametrize("batch,w,h", [(1, 8, 8), (3, 24, 40), (2, 136, 72)])
def test_gradient_sizes(cuda, batch, w, h):
    """Against FP32 autograd where every pre-activation is positive and every
    loss term keeps its sign (as in test_gradient_in_the_linear_regime)."""
    net = Net(batch, w, h, seed=5)
    try:
        g = torch.Generator().manual_seed(9)
        flat = []
        for cin, cout, _ in SPEC:
            flat.append((torch.randn(cout, cin, 3, 3, generator=g) * 0.2 * (2.0 / (9 * cin)) ** 0.5).permute(0, 2, 3, 1).reshape(-1))
            flat.append(torch.full((cout,), 4.0))
        p0 = torch.cat(flat).contiguous()
        pn = p0.numpy()
        assert net.lib.arbor_denoiser_set_params(net.h, pn.ctypes.data, pn.size) == ab.OK, ab.last_error()
        feat, noisy, target = random_inputs(batch, w, h, seed=1)
        params = [t.clone().requires_grad_(True) for pair in unpack(p0.clone()) for t in pair]
        layers = [(params[2 * i], params[2 * i + 1]) for i in range(len(SPEC))]
        out = reference_forward(layers, feat.permute(0, 3, 1, 2))[:, :3].permute(0, 2, 3, 1)
        resid = torch.log1p(noisy[..., :3].clamp(min=0)) + out - torch.log1p(target[..., :3].clamp(min=0))
        assert bool((resid > 0.5).all()), "every loss term must keep its sign"
        resid.abs().mean().backward()
        gref = torch.cat([torch.cat([params[2 * i].grad.permute(0, 2, 3, 1).reshape(-1), params[2 * i + 1].grad]) for i in range(len(SPEC))])
        grad, loss = np.full(net.count, np.nan, np.float32), ctypes.c_float()
        f, n, t = to_dev_bf16(feat), noisy.contiguous().cuda(), target.contiguous().cuda()
        assert net.lib.arbor_denoiser_gradient(net.h, f.data_ptr(), n.data_ptr(), t.data_ptr(), batch, w, h, grad.ctypes.data, grad.size,
                                               ctypes.byref(loss)) == ab.OK, ab.last_error()
        got, off = torch.from_numpy(grad).double(), 0
        for cin, cout, _ in SPEC:
            k = cout * 9 * cin + cout
            a, b = got[off:off + k], gref[off:off + k].double()
            assert float((a @ b) / (a.norm() * b.norm() + 1e-30)) >= 0.9998
            assert float((a - b).norm() / (b.norm() + 1e-30)) <= 2e-2
            off += k
    finally:
        net.close()
