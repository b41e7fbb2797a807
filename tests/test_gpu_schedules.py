"""The launch schedules agree bit for bit: the flow schedule of long fits of many
voxels with the grid schedule (which runs every iteration), and the random
search with its draws side by side with one thread per voxel."""
import pytest
import torch

from pycompute_gb300 import Expr, SecondOrderLevenbergMarquardt, SecondOrderRandomSearch, pipeline, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _state(s):
    return {k: getattr(s, k) for k in ("pars_t", "first_f", "last_f", "f_t", "lam_t", "step_type_t", "step_t", "iters_t")}


def _same(a, b):
    for k in a:
        x, y = a[k], b[k]
        x, y = (v.view(torch.int32) if v.dtype == torch.float32 else v for v in (x, y))
        assert torch.equal(x, y), (k, int((x != y).sum()))


@pytest.mark.parametrize("workload,iters,kw", [
    (synth.ivim, 100, {}), (synth.ivim, 130, dict(dec=1.0)), (synth.ivim, 120, dict(dec=3.7, acc=0.5)),
    (synth.ivim, 110, dict(dec=0.7)), (synth.t2star, 100, dict(tol=1e-30)), (synth.vfa_t1, 150, {}),
    (synth.ivim, 260, dict(mu=0.0, eta=0.1)), (synth.biexp_t2, 100, {})])
def test_flow_equals_grid(workload, iters, kw):
    w = workload()
    n = 262147  # 128 voxel-iterations past the 40th per resident thread, ragged
    _, data = pipeline.synth_gpu(w, n, seed=3, device=DEV)
    data[:, 5::1001] = float("nan")
    data[:, 6::1003] = 0.0
    got = []
    for block in (0, 128):  # a block size asks for the grid schedule
        s = SecondOrderLevenbergMarquardt(Expr(w.expr, w.pars, w.consts), None, w.M, torch.float32)
        s.setup(pipeline.init_constant(data, w.init_values), list(w.protocol), data, list(w.lb), list(w.ub))
        s.step_type_t[0, ::17] = 0   # converged before the call
        s.step_type_t[0, 1::17] = 4  # left by an earlier run after a rejected step
        s.lam_t[0, 2::19] = 1e20     # a damping from which every step is too small
        s.run(iters, block=block, **kw)
        torch.cuda.synchronize()
        got.append(_state(s))
    _same(*got)


@pytest.mark.parametrize("draws,lm_iters", [(1, 4), (3, 0), (7, 3), (130, 0)])
def test_search_draws_side_by_side_equal_one_thread(draws, lm_iters):
    w = synth.ivim()
    n = 1 << 20
    _, data = pipeline.synth_gpu(w, n, seed=4, device=DEV)
    got = []
    for m in (n, 701):  # many voxels: one thread each; few: the draws side by side
        rs = SecondOrderRandomSearch(Expr(w.expr, w.pars, w.consts), w.M, torch.float32)
        rs.setup(list(w.protocol), data[:, :m].contiguous(), list(w.lb), list(w.ub))
        for seed in (11, 12):  # the second starts from the first one's best
            rs.run(draws, lm_iters=lm_iters, seed=seed)
        torch.cuda.synchronize()
        got.append({"p": rs.best_pars_t[:, :701].contiguous(), "f": rs.best_f_t[:, :701].contiguous()})
    _same(*got)


@pytest.mark.parametrize("workload,solve", [(synth.vfa_t1, torch.float64), (synth.vfa_t1, torch.float32),
                                            (synth.t2star, torch.float64), (synth.t2star, torch.float32)])
def test_search_of_few_parameters_equals_refined_starts(workload, solve):
    """A draw refined by the search against the fitter started from that draw: with one draw, the parameters that the
    search without refinement returns."""
    w = workload()
    n, iters = 4099, 20
    _, data = pipeline.synth_gpu(w, n, seed=6, device=DEV)
    got = []
    for lm_iters in (0, iters):
        rs = SecondOrderRandomSearch(Expr(w.expr, w.pars, w.consts), w.M, torch.float32, solve_dtype=solve)
        rs.setup(list(w.protocol), data, list(w.lb), list(w.ub))
        rs.run(1, lm_iters=lm_iters, seed=21)
        got.append((rs.best_pars_t, rs.best_f_t.reshape(-1)))
    p = got[0][0].clone()
    s = SecondOrderLevenbergMarquardt(Expr(w.expr, w.pars, w.consts), None, w.M, torch.float32, solve_dtype=solve)
    s.setup(p, list(w.protocol), data, list(w.lb), list(w.ub))
    s.run(iters, block=128)
    f = s.cost().reshape(-1)
    torch.cuda.synchronize()
    same = (got[1][0].view(torch.int32) == p.view(torch.int32)).all(0)
    # the same arithmetic from the same start; a draw whose refinement stopped at the search's own start cost is kept
    better = f < torch.finfo(torch.float32).max / 5
    assert bool(same[better].all()), int((~same[better]).sum())
    assert torch.equal(got[1][1][better].view(torch.int32), f[better].view(torch.int32))
