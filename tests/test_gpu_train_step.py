"""spx_mlp_train_step against the same step made of single calls (spx_gemm_bf16, spx_mlp_loss_grad,
spx_rowsum_bf16, spx_adamw): batches below, at and past the row tile and the K-block, ragged ones among
them. A product's elements are accumulated over K in one order whatever the tile and the launch, so
weights, gradients and bf16 copies are the same bits; and a row's outputs do not depend on the batch.
The loss is an FP64 sum in another order (1e-12)."""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _single_calls(net, x, xt, t, weights, lr, wd):
    import torch

    from imageprocessor_new_b200 import _device as dev
    from imageprocessor_new_b200 import _lib
    from imageprocessor_new_b200.warmstart import HID, IN, OUT, OUT_PAD, _gemm

    b, bf, s, p, err = x.shape[0], torch.bfloat16, dev.stream_ptr(), net.p, net.err
    y, (h1, h1t, h2, h2t) = net.forward(x, keep=True)
    loss = torch.zeros(1, dtype=torch.float64, device="cuda")
    dy, dyt = dev.empty((b, OUT_PAD), bf), dev.empty((OUT_PAD, b), bf)
    _lib.call("spx_mlp_loss_grad", y.data_ptr(), t.data_ptr(), weights.data_ptr(), b, OUT, OUT_PAD, dy.data_ptr(),
              dyt.data_ptr(), loss.data_ptr(), s)
    dh2, dh2t, dh1t = dev.empty((b, HID), bf), dev.empty((HID, b), bf), dev.empty((HID, b), bf)
    _gemm(dyt, h2t, OUT, HID, b, out_f32=p["w3"].g, ld_f32=HID, err=err)
    _gemm(dy, net.w3t, b, HID, OUT_PAD, mask=h2, ld_mask=HID, out_bf16=dh2, ld_bf16=HID, out_t=dh2t, ld_t=b, err=err)
    _gemm(dh2t, h1t, HID, HID, b, out_f32=p["w2"].g, ld_f32=HID, err=err)
    _gemm(dh2, net.w2t, b, HID, HID, mask=h1, ld_mask=HID, out_t=dh1t, ld_t=b, err=err)
    _gemm(dh1t, xt, HID, IN, b, out_f32=p["w1"].g, ld_f32=IN, err=err)
    for src, rows, name in ((dyt, OUT, "b3"), (dh2t, HID, "b2"), (dh1t, HID, "b1")):
        _lib.call("spx_rowsum_bf16", src.data_ptr(), rows, b, p[name].g.data_ptr(), s)
    net.step += 1
    for name, out, out_rows, out_t, ld_t in (("w1", net.w1, HID, None, 0), ("w2", net.w2, HID, net.w2t, HID),
                                             ("w3", net.w3, OUT_PAD, net.w3t, OUT_PAD), ("b1", None, 0, None, 0),
                                             ("b2", None, 0, None, 0), ("b3", None, 0, None, 0)):
        q = p[name]
        rows, cols = (q.w.shape[0], q.w.shape[1]) if q.w.dim() == 2 else (1, q.w.shape[0])
        f = ctypes.c_float
        _lib.call("spx_adamw", q.w.data_ptr(), q.g.data_ptr(), q.m.data_ptr(), q.v.data_ptr(), rows, cols, net.step,
                  f(lr), f(0.9), f(0.999), f(1e-8), f(wd if name.startswith("w") else 0.0),
                  None if out is None else out.data_ptr(), out_rows, None if out_t is None else out_t.data_ptr(), ld_t, s)
    return loss


@pytest.mark.parametrize("batch", [8, 120, 128, 136, 1000, 2056])
def test_train_step_is_its_single_calls(batch):
    import torch

    from imageprocessor_new_b200 import warmstart as ws

    g = torch.Generator(device="cuda").manual_seed(batch)
    x = torch.rand((batch, ws.IN), device="cuda", generator=g).to(torch.bfloat16)
    xt, t = x.t().contiguous(), torch.randn((batch, ws.OUT), device="cuda", generator=g)
    weights = torch.rand(ws.OUT, device="cuda", generator=g)
    one, many = ws.WarmStartNet(seed=3), ws.WarmStartNet(seed=3)
    for _ in range(2):
        la = one.train_step(x, xt, t, weights, lr=1e-3, weight_decay=0.01)
        lb = _single_calls(many, x, xt, t, weights, 1e-3, 0.01)
        np.testing.assert_allclose(float(la), float(lb), rtol=1e-12)
    one.check_errors()
    many.check_errors()
    for name in one.p:
        for field in ("w", "g", "m", "v"):
            assert torch.equal(getattr(one.p[name], field), getattr(many.p[name], field)), (name, field)
    for name in ("w1", "w2", "w2t", "w3", "w3t"):
        assert torch.equal(getattr(one, name), getattr(many, name)), name


def test_rows_do_not_depend_on_the_batch():
    """Outputs of the first rows of batches whose tiles are 16 to 256 columns wide."""
    import torch

    from imageprocessor_new_b200 import warmstart as ws

    net = ws.WarmStartNet.load()
    x = torch.rand((40000, ws.IN), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)).to(torch.bfloat16)
    want = net.forward(x)
    for rows in (1, 100, 2000, 9000):
        assert torch.equal(net.forward(x[:rows]), want[:rows]), rows


def test_train_step_refuses_a_ragged_batch():
    import torch

    from imageprocessor_new_b200 import _lib
    from imageprocessor_new_b200 import warmstart as ws

    net = ws.WarmStartNet(seed=0)
    x = torch.zeros((12, ws.IN), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(_lib.LibraryError, match="multiple of 8"):
        net.train_step(x, x.t().contiguous(), torch.zeros((12, ws.OUT), device="cuda"), torch.ones(ws.OUT, device="cuda"),
                       lr=0.0)
    assert net.step == 0
