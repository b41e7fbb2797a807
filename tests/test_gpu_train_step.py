"""The fused training step (forward, loss, backward and weight gradients of 128
rows per CTA in one launch, Adam in another) against the GEMM path and the numpy
oracle, its lost-wait path, and the target statistics."""
import numpy as np
import pytest
import torch

from oracle import mlp_oracle as mo
from pycompute_gb300 import synth
from pycompute_gb300.warmstart import HID, WarmStartMLP

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _net(n, seed, nout=4):
    w = synth.ivim(synth.ivim_b16(), name="ivim16")
    true, data, *_ = w.generate(n, seed=seed)
    net = WarmStartMLP(16, nout, [0, 1, 2, 2][:nout], w.lb[:nout], w.ub[:nout], DEV, seed=seed)
    sig, lab = torch.from_numpy(data).to(DEV), torch.from_numpy(true[:nout].copy()).to(DEV)
    net.fit_normalisation(sig, lab)
    x, _, t = net._prepare(sig, lab)
    return net, x, t, sig, lab


@pytest.mark.parametrize("B,nout", [(128, 4), (512, 4), (8192, 4), (384, 1), (256, 3)])
def test_gradients_equal_the_gemm_path_and_the_oracle(B, nout):
    net, x, t, _, _ = _net(B, 3, nout)
    net._alloc_batch(B)
    net.bx.copy_(x)
    net.bt.copy_(t)
    net._forward_train()
    net._backward(k_split=128)
    want = [L.grad.clone() for L in net.layers]
    loss = float(net.loss_sum.item())
    for L in net.layers:
        L.grad.zero_()
    net.loss_sum.zero_()
    net._fused_steps(x, t, 1, B, 0, 1, 1e-3, torch.ones(3, device=DEV), update=False)
    torch.cuda.synchronize()
    assert net.gemm_status() == 0
    assert abs(float(net.loss_sum.item()) - loss) <= 1e-5 * loss
    # the same bf16 operands: fp32 sums over rows in another order, and through it an occasional bf16 rounding of a
    # later layer's operand (2^-9 of that entry) flips
    for L, g in zip(net.layers, want):
        assert float((L.grad - g).norm() / g.norm()) < 1e-3
    dims = [(16, HID), (HID, HID), (HID, HID), (HID, nout)]
    grads, _, ref_loss = mo.backward(x[:, :16].float().cpu().numpy().astype(np.float64),
                                     t.cpu().numpy().astype(np.float64), [L.master.cpu().numpy() for L in net.layers],
                                     dims, nout)
    for L, ref in zip(net.layers, grads):
        g = L.grad.cpu().numpy().astype(np.float64)
        assert np.linalg.norm(g - ref) < 1e-2 * np.linalg.norm(ref)


def test_training_equals_the_gemm_path():
    n, B = 128 * 9 + 5, 256
    nets = []
    for fused in (True, False):
        net, _, _, sig, lab = _net(n, 5)
        net._fused_steps = net._fused_steps if fused else None
        net.gemm_impl = "tcgen05" if fused else "mma"
        net.train(sig, lab, epochs=3, batch=B, lr=1e-3, log_every=2)
        nets.append(net)
    a, b = nets
    assert a.step == b.step == 12 and a.gemm_status() == 0
    np.testing.assert_allclose(a.losses, b.losses, rtol=2e-2)
    for x, y in zip(a.layers, b.layers):
        assert float((x.master - y.master).norm() / y.master.norm()) < 2e-2
        assert torch.equal(x.wbf, x.master.to(torch.bfloat16)) and float(x.grad.abs().max()) == 0.0


def test_lost_wait_sets_status_frees_tmem_and_returns():
    """CTA 1 never issues its first stage (no tensor-core work of it is in
    flight), so its wait runs out: the call returns, the status is set, the other
    CTAs' gradients are there, and a normal step right after equals the GEMM
    path, which it could not if CTA 1 had kept its tensor memory (all 512
    columns)."""
    B = 512
    net, x, t, _, _ = _net(B, 7)
    net.loss_sum = torch.zeros(1, device=DEV)
    one = torch.ones(3, device=DEV)
    net._fused_steps(x, t, 1, B, 0, 1, 1e-3, one, wait_limit=1 << 10, skip_block=1, update=False)
    torch.cuda.synchronize()
    assert net.gemm_status() == 1
    part = [L.grad.clone() for L in net.layers]
    for L in net.layers:
        L.grad.zero_()
    net._gemm_status.zero_()
    for lo in (0, 256, 384):
        net._fused_steps(x[lo:lo + 128], t[lo:lo + 128], 1, 128, 0, 1, 1e-3, one, update=False)
    torch.cuda.synchronize()
    for L, g in zip(net.layers, part):  # the mean runs over 128 rows here and over 512 there
        assert float((L.grad / 4 - g).norm() / g.norm()) < 1e-2
    assert net.gemm_status() == 0


@pytest.mark.parametrize("n", [1, 255, 257, 300001])
def test_target_statistics_equal_numpy(n):
    g = torch.Generator(device=DEV).manual_seed(n)
    sig = torch.rand((16, n), generator=g, device=DEV) * 1000
    sig[:, 0] = 0.0  # the largest signal is clamped from below
    par = torch.rand((4, n), generator=g, device=DEV) * torch.tensor([[1000.0], [0.3], [0.05], [1e-3]], device=DEV)
    par[2, -1] = 0.0  # and so is the argument of the logarithm
    if n > 1:
        par[0, 0] = 1e-18
    net = WarmStartMLP(16, 4, [0, 1, 2, 2], [0] * 4, [1] * 4, DEV)
    net.fit_normalisation(sig, par)
    got = net.mean.copy(), net.std.copy()
    net.fit_normalisation(sig.cpu(), par.cpu())  # numpy
    np.testing.assert_allclose(got[0], net.mean, rtol=3e-7, atol=1e-30)
    np.testing.assert_allclose(got[1], net.std, rtol=1e-6)
