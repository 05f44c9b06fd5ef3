"""The drag network's loss, gradient and forward kernels at the edges of their tiles (64 samples, two groups of
256 threads per CTA), against torch in 64 bits.  Tolerance: a sum of up to n products in FP32 with partial sums
of at most 64 terms per tile; the 2-norm of its error over that of the gradient was below 1e-6 for every n
here, the bound is 5e-6."""
import pytest
import torch

from gpuimogen_b200 import learned_drag as ld

pytestmark = pytest.mark.gpu


def _net(ib, p, x):
    o, H = ib.MLP_OFF, ib.MLP_HID
    h = torch.relu(x @ p[o["W1"]:o["B1"]].view(H, 16).T + p[o["B1"]:o["W2"]])
    h = torch.relu(h @ p[o["W2"]:o["B2"]].view(H, H).T + p[o["B2"]:o["W3"]])
    h = torch.relu(h @ p[o["W3"]:o["B3"]].view(H, H).T + p[o["B3"]:o["W4"]])
    return h @ p[o["W4"]:o["B4"]] + p[o["B4"]]


@pytest.mark.parametrize("n", [1, 5, 63, 64, 65, 127, 129, 64 * 148 - 1, 64 * 148 + 1, 2 * 64 * 148 + 70, 70001])
@pytest.mark.parametrize("shift", [0, 1])
def test_loss_gradient_and_forward(cuda, ib, n, shift):
    import gpuimogen_b200.imogen as im
    g = torch.Generator().manual_seed(n)
    buf = torch.randn(n * 16 + shift, generator=g).cuda()
    x = buf[shift:].view(n, 16)          # shift: rows that are not 16-byte aligned
    t = torch.randn(n, generator=g).cuda()
    p = ld.init_params(3)
    p += 0.05 * torch.randn(p.numel(), generator=g).cuda()   # biases and padding columns count too
    q = p.double().requires_grad_()
    y = _net(im, q, x.double())
    loss = ((y - t.double()) ** 2).mean()
    grad, = torch.autograd.grad(loss, q)
    tr = ld.Trainer(p, batch=n)
    got, l = tr.loss_grad(x, t)
    torch.cuda.synchronize()
    assert abs(float(l) - float(loss)) <= 5e-6 * float(loss)
    assert float((got.double() - grad).norm()) <= 5e-6 * float(grad.norm())
    again, _ = ld.Trainer(p, batch=n).loss_grad(x, t)
    assert torch.equal(got, again)       # the sums are taken in a fixed order
    f = ld.forward_fp32(p, x)
    assert float((f.double() - y.detach()).norm()) <= 5e-6 * float(y.detach().norm())
