"""What setup() finds out about a protocol or bounds array on the device (shared or
per voxel, and the shared values), and the state it starts a fit from."""
import numpy as np
import pytest
import torch

from pycompute_gb300 import SecondOrderLevenbergMarquardt, synth
from pycompute_gb300.lsqnonlin import _shared_many

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64, torch.float16, torch.int64])
@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 300001])
def test_rows_are_classified_as_by_comparing_columns(dtype, n):
    rng = np.random.default_rng(n)
    first = torch.from_numpy(rng.integers(1, 50, 21)).to(DEV).to(dtype)
    tiled = first[:, None].expand(21, n)
    odd = tiled.clone()
    odd[20, n - 1] += 1  # the last entry of the last row
    args = [(tiled, 21, "a"), (odd, 21, "b"), (first[:4].clone(), 4, "c")]
    (t, stride, vals), (_, stride2, vals2), (_, stride3, vals3) = _shared_many(args, n, True)
    assert t is tiled and stride == 0 and vals == first.double().tolist()
    if n == 1:  # one column is always equal to itself
        assert stride2 == 0 and vals2 == odd[:, 0].double().tolist()
    else:
        assert stride2 == n and vals2 is None
    assert stride3 == 0 and vals3 == first[:4].double().tolist()
    if n > 1:
        assert _shared_many(args[:1], n, False)[0][1:] == (n, None)
    if dtype.is_floating_point:
        nan = tiled.clone()
        nan[3] = float("nan")  # equal to nothing, itself included
        assert _shared_many([(nan, 21, "d")], n, True)[0][1:] == (n, None)


def test_wrong_shapes_are_refused():
    a = torch.zeros(5, 7, device=DEV)
    for rows, n in ((4, 7), (5, 6)):
        with pytest.raises(RuntimeError):
            _shared_many([(a, rows, "a")], n, True)


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("n", [0, 1, 257, 1100003])
def test_setup_starts_every_state_array(dtype, n):
    w = synth.ivim()
    s = SecondOrderLevenbergMarquardt(w.expr, w.pars, w.consts, ndata=w.M, dtype=dtype)
    s.setup(torch.ones(4, n, dtype=dtype, device=DEV), list(w.protocol), torch.ones(10, n, dtype=dtype, device=DEV),
            list(w.lb), list(w.ub))
    for t, v, dt in ((s.lam_t, 5, dtype), (s.step_t, 0, dtype), (s.f_t, 0, dtype), (s.step_type_t, 1, torch.int8),
                     (s.iters_t, 0, torch.int32)):
        assert t.dtype == dt and t.shape[1] == n and bool((t == v).all())
