"""The flow schedule of mixed-model batches: a warp that keeps the lanes of one chunk alive while it claims the next,
hands a chunk of another job back, and leaves the models that do not flow to the grid. Per voxel the results are those
of fits too short to flow, run one after the other."""
import ctypes

import pytest
import torch

from pycompute_gb300 import Expr, _lib, synth
from pycompute_gb300.multi import MultiJob, MultiModelFitter, _Job

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
WORKLOADS = [synth.vfa_t1, synth.t2star, synth.ivim, synth.biexp_t2]
GRID, BLOCK = 2, 128  # 256 threads, 448 voxels to flow: many claims per warp, across the jobs' borders


def _inputs(sizes):
    out = []
    for k, (f, n) in enumerate(zip(WORKLOADS, sizes)):
        w = f()
        _, data, init, lb, ub, prot = w.generate(max(n, 1), seed=60 + k)
        data, init = torch.from_numpy(data)[:, :n].contiguous().to(DEV), torch.from_numpy(init)[:, :n].contiguous().to(DEV)
        data[:, 5::101] = float("nan")
        data[:, 6::103] = 0.0
        out.append((data, init, prot, lb, ub))
    return out


def _jobs(inputs):
    jobs = []
    for data, init, prot, lb, ub in inputs:
        j = MultiJob(init.clone(), data, prot, lb, ub)
        j.step_type[::17] = 0   # converged before the call
        j.step_type[1::17] = 4  # left by an earlier run after a rejected step
        j.lam[2::19] = 1e20     # a damping from which every step is too small
        jobs.append(j)
    return jobs


def _bits(t):
    return t.view(torch.int32) if t.dtype == torch.float32 else t


@pytest.mark.parametrize("lanes", [[1, 1, 1, 1], [1, 2, 1, 2]])
@pytest.mark.parametrize("sizes,order", [
    ((1500, 700, 2049, 300), [2, 0, 3, 1]),  # all but the third model of the order flow
    ((1, 31, 4000, 33), [0, 1, 2, 3]),       # one does, between jobs smaller than a chunk
    ((0, 447, 448, 64), [3, 2, 1, 0])])      # the least that does, beside one voxel less and an empty job
@pytest.mark.parametrize("iters", [64, 100, 150])
def test_flow_equals_shorter_runs(lanes, sizes, order, iters):
    models = [(Expr(w.expr, w.pars, w.consts), w.M) for w in (f() for f in WORKLOADS)]
    fitter = MultiModelFitter(models, block=BLOCK, lanes=lanes)
    prog = fitter.build()
    inputs = _inputs(sizes)
    for k, n in enumerate(sizes):
        want = n >= 448 and k != 3 and lanes[k] == 1
        assert _lib.lib().pcgb_multi_schedule(prog, k, n, iters, GRID) == int(want)
        assert _lib.lib().pcgb_multi_schedule(prog, k, n, 63, GRID) == 0
    flow, parts = _jobs(inputs), _jobs(inputs)
    fitter.fit(flow, iters, grid=GRID, order=order)
    first = None
    left = iters
    while left:
        k = min(left, 50)
        fitter.fit(parts, k, grid=GRID, order=order)
        if first is None:
            torch.cuda.synchronize()
            first = [j.first_f.clone() for j in parts]
        left -= k
    noalloc = _jobs(inputs)
    arr = (_Job * len(noalloc))(*[j.ctype() for j in noalloc])
    _lib.check("pcgb_multi_run_noalloc", _lib.lib().pcgb_multi_run_noalloc(
        prog, arr, len(noalloc), (ctypes.c_int * 4)(*order), iters, 1e-8, 0.25, 0.75, 0.2, 2.0, 64, GRID,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    for a, b, c, f0 in zip(flow, parts, noalloc, first):
        for name in ("pars", "lam", "step_type", "f", "last_f", "iters"):
            x, y, z = (_bits(getattr(j, name)) for j in (a, b, c))
            assert torch.equal(x, y) and torch.equal(x, z), name
        assert torch.equal(_bits(a.first_f), _bits(f0)) and torch.equal(_bits(c.first_f), _bits(f0))
