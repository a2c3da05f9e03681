"""vfps_ws_forward / vfps_ws_backward on networks of any hidden width, through
the C ABI, against the float64 restatement (oracle/warmstart_ref.py)."""
import ctypes as C

import numpy as np
import pytest
import torch

from inovesa_gb300 import _lib
from oracle import warmstart_ref as R

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
NLAT = 32


class Net:
    """Random weights of a network and buffers for B samples."""

    def __init__(self, ctx, nin, nh, npix, B, seed=0):
        self.ctx, self.dims, self.B = ctx, (nin, nh, NLAT, npix), B
        g = torch.Generator(device=DEV).manual_seed(seed)

        def rnd(*s, scale=1.0):
            return torch.randn(*s, generator=g, device=DEV) * scale
        self.shapes = dict(w1=(nh, nin), b1=(nh,), w2=(nh, nh), b2=(nh,),
                           w3=(NLAT, nh), b3=(NLAT,), wd=(NLAT, npix),
                           bd=(npix,))
        fan = dict(w1=nin, w2=nh, w3=nh, wd=NLAT)
        self.w = {k: rnd(*s, scale=fan.get(k, 100) ** -0.5)
                  for k, s in self.shapes.items()}
        for k in fan:
            self.w[k] = self.w[k].bfloat16()
        self.grad = {k: torch.full(s, 7.0, device=DEV)
                     for k, s in self.shapes.items()}
        self.x, self.target = rnd(B, nin), rnd(B, npix)
        z = dict(h1=nh, h2=nh, z=NLAT, g=npix, dz=NLAT, d1=nh, d2=nh)
        self.buf = {k: torch.zeros(B, c, device=DEV) for k, c in z.items()}
        self.lp = torch.zeros(256, dtype=torch.float64, device=DEV)

    def struct(self, t):
        return _lib.WsNet(*self.dims, *(t[k].data_ptr() for k in self.shapes))

    def forward(self):
        torch.cuda.synchronize()
        net, b = self.struct(self.w), self.buf
        rc = _lib.lib().vfps_ws_forward(
            self.ctx.handle, C.byref(net), self.x.data_ptr(), self.B,
            b["h1"].data_ptr(), b["h2"].data_ptr(), b["z"].data_ptr(), None,
            self.target.data_ptr(), b["g"].data_ptr(), self.lp.data_ptr(),
            256)
        self.ctx.synchronize()
        return rc

    def backward(self):
        torch.cuda.synchronize()
        net, grad, b = self.struct(self.w), self.struct(self.grad), self.buf
        rc = _lib.lib().vfps_ws_backward(
            self.ctx.handle, C.byref(net), C.byref(grad), self.x.data_ptr(),
            self.B, *(b[k].data_ptr()
                      for k in ("h1", "h2", "z", "g", "dz", "d1", "d2")))
        self.ctx.synchronize()
        return rc

    def loss(self):
        return float(self.lp.sum().item()) / self.target.numel()

    def want(self):
        w = {k: v.double().cpu().numpy() for k, v in self.w.items()}
        return R.loss_and_grads(w, self.x.cpu().numpy(),
                                self.target.cpu().numpy())


# a unit, the width on either side of 48 KiB for eight slices of a layer's
# sums, and the widest that the forward pass takes
@pytest.mark.parametrize("nin,nh", [(3, 1), (3, 1134), (3, 1135), (2, 1536),
                                    (1, 6143)])
def test_hidden_width(gpu_ctx, nin, nh):
    """FP32 sums of nh terms in slices: within 1e-4 of the largest entry, as
    for the 128 units of the network in use (an error of sqrt(nh / 8) eps / 2
    of the sum of magnitudes at most)."""
    net = Net(gpu_ctx, nin, nh, 300, 3, seed=nh)
    assert net.forward() == 0
    assert net.backward() == 0
    loss, grads = net.want()
    assert abs(net.loss() - loss) <= 1e-5 * loss
    for k, g in grads.items():
        got = net.grad[k].double().cpu().numpy()
        assert np.abs(got - g).max() <= 1e-4 * np.abs(g).max(), k


# wider layers than the forward pass takes, from buffers of the caller: fewer
# slices; and past the backward pass's own limit: refused before anything is
# written
@pytest.mark.parametrize("nh,taken", [(6200, True), (12256, True),
                                      (12257, False)])
def test_hidden_width_limits(gpu_ctx, nh, taken):
    net = Net(gpu_ctx, 1, nh, 64, 1)
    net.buf["z"].normal_()
    net.buf["g"].normal_()
    rc = net.backward()
    if not taken:
        assert rc != 0
        for v in net.grad.values():
            assert bool((v == 7.0).all())
        return
    assert rc == 0
    # (h1 = h2 = 0: d2 = W3^T dz, d1 = W2^T d2)
    w = {k: v.double() for k, v in net.w.items()}
    dz = net.buf["g"].double() @ w["wd"].T
    d2 = dz @ w["w3"]
    d1 = d2 @ w["w2"]
    for k, v in (("dz", dz), ("d2", d2), ("d1", d1)):
        err = (net.buf[k].double() - v).abs().max()
        assert float(err) <= 1e-4 * float(v.abs().max()), k


def test_loss_range(gpu_ctx):
    """The loss is summed in 64 bits: squares of residuals that FP32 cannot
    hold, large and small, count."""
    for scale in (1e25, 1e-25):
        net = Net(gpu_ctx, 3, 16, 300, 5)
        net.target = torch.randn(5, 300, device=DEV) * scale
        for k in ("w3", "b3", "bd"):
            net.w[k].zero_()     # y = 0: the residual is the target
        assert net.forward() == 0
        want = float((net.target.double() ** 2).mean())
        assert abs(net.loss() - want) <= 1e-14 * want


def test_latent_gradient_cancels(gpu_ctx):
    """dz adds FP32 sums of 32 pixels in 64 bits: sums of 1, 2^-25, 2^-51, -1
    and -2^-25 leave 2^-51 (a pair of FP32 numbers loses it beside 2^-25)."""
    net = Net(gpu_ctx, 1, 4, 300, 1)
    net.w["wd"].fill_(1.0)
    g = net.buf["g"][0]
    for k, v in enumerate((1.0, 2.0 ** -25, 2.0 ** -51, -1.0, -2.0 ** -25)):
        g[32 * k] = v
    assert net.backward() == 0
    assert bool((net.buf["dz"] == 2.0 ** -51).all())


def test_scratch_is_bounded():
    """Growing minibatches in turn: the context's scratch for the backward
    pass stays within twice the largest call's (32 MB for 384 samples of
    78000 pixels or more; its powers of two add up to 64 MB), and goes with
    the context."""
    from inovesa_gb300 import vfps as V
    npix, largest = 304 * 256, 384
    ctx = V.Context(0)
    net = Net(ctx, 1, 4, npix, largest)
    net.backward()      # whatever else the first call loads
    ctx.close()
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    ctx = V.Context(0)
    net.ctx = ctx
    for net.B in list(range(1, 200, 3)) + [largest]:
        assert net.backward() == 0
    held = before - torch.cuda.mem_get_info()[0]
    assert held <= (64 + 8) << 20, held
    ctx.close()
    assert before - torch.cuda.mem_get_info()[0] <= 8 << 20
