"""Tile schedule of the tcgen05 network: which CTA gets a tile never shows in a
voxel's result."""
import numpy as np
import pytest
import torch

from pycompute_gb300 import synth
from pycompute_gb300.warmstart import WarmStartMLP

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("per_sm,extra", [(1, -1), (1, 0), (1, 1), (4, 0), (4, 1), (9, 3)])
def test_tiles_of_a_large_call_equal_small_calls(per_sm, extra):
    """Around one tile per SM, four (all tensor memory in use) and several
    rounds: equal bit for bit to calls of 13 tiles, since a voxel's arithmetic
    reads nothing of its neighbours."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 128 * (per_sm * sms + extra) - 5
    w = synth.ivim(synth.ivim_b16(), name="ivim16")
    true, data, *_ = w.generate(n, seed=17)
    sig = torch.from_numpy(np.ascontiguousarray(data)).to(DEV)
    net = WarmStartMLP(16, 4, [0, 1, 2, 2], w.lb, w.ub, DEV, seed=3, log_in=True)
    net.fit_normalisation(sig, torch.from_numpy(np.ascontiguousarray(true)).to(DEV))
    whole = net.infer(sig, impl="tcgen05")
    step = 128 * 13
    parts = [net.infer(sig[:, i:i + step].contiguous(), impl="tcgen05") for i in range(0, n, step)]
    torch.cuda.synchronize()
    assert net.tc_status() == 0
    assert torch.equal(whole, torch.cat(parts, dim=1))
