"""Training after a wait for the tensor cores ran out: no step learns from the incomplete gradients, and train() says so."""
import pytest
import torch

from pycompute_gb300 import synth
from pycompute_gb300.warmstart import WarmStartMLP

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _net(n, seed):
    w = synth.ivim(synth.ivim_b16(), name="ivim16")
    true, data, *_ = w.generate(n, seed=seed)
    net = WarmStartMLP(16, 4, [0, 1, 2, 2], w.lb, w.ub, DEV, seed=seed)
    return net, torch.from_numpy(data).to(DEV), torch.from_numpy(true).to(DEV)


def _weights(net):
    return [t.clone() for L in net.layers for t in (L.master, L.m, L.v, L.wbf)]


def test_a_lost_step_leaves_the_weights_and_the_next_call_trains():
    """One CTA of two never issues its first stage (nothing of it is in flight), so its bounded wait runs out."""
    B = 256
    net, sig, lab = _net(B, 3)
    net.fit_normalisation(sig, lab)
    x, _, t = net._prepare(sig, lab)
    net.loss_sum = torch.zeros(1, device=DEV)
    corr = torch.tensor([[0.1, 0.001, 1.0]] * 3, device=DEV)
    before = _weights(net)
    net._fused_steps(x, t, 1, B, 0, 3, 1e-3, corr, wait_limit=1 << 10, skip_block=1)
    torch.cuda.synchronize()
    assert net.gemm_status() == 1
    assert all(torch.equal(a, b) for a, b in zip(before, _weights(net)))
    assert all(float(L.grad.abs().max()) == 0.0 for L in net.layers)
    net._gemm_status.zero_()
    net._fused_steps(x, t, 1, B, 0, 1, 1e-3, corr)
    torch.cuda.synchronize()
    assert net.gemm_status() == 0
    assert not any(torch.equal(a, b) for a, b in zip(before[::4], _weights(net)[::4]))


def test_train_raises_and_can_be_called_again():
    net, sig, lab = _net(1024, 5)
    steps = net._fused_steps
    net._fused_steps = lambda *a, **k: steps(*a, wait_limit=1 << 10, skip_block=0, **k)
    with pytest.raises(RuntimeError, match="ran out"):
        net.train(sig, lab, epochs=1, batch=256)
    assert net.gemm_status() == 1
    net._fused_steps = steps
    net.train(sig, lab, epochs=1, batch=256)
    assert net.gemm_status() == 0
