"""Which fits run the flow schedule, and what their programs compile: the kernel is there for the models that keep its
register cap, nothing is compiled for a model that does not, and pcgb_fitter_compile leaves a run nothing to compile."""
import ctypes
import os

import pytest
import torch

from pycompute_gb300 import Expr, SecondOrderLevenbergMarquardt, SecondOrderRandomSearch, _lib, codegen, pipeline, synth

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _fitter(w, solve=torch.float64, dtype=torch.float32):
    return SecondOrderLevenbergMarquardt(Expr(w.expr, w.pars, w.consts), None, w.M, dtype, solve_dtype=solve)


def _schedule(s, n, iters):
    rc = _lib.lib().pcgb_lm_schedule(s.build().handle, n, iters, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc in (0, 1), _lib.lib().pcgb_last_error()
    return "flow" if rc else "grid"


def _least(iters):  # voxels from which a fit of that many iterations may flow
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return -(-128 * 128 * 6 * sms // (iters - 40))


@pytest.mark.parametrize("workload,flows", [
    (synth.ivim, True), (lambda: synth.ivim(synth.ivim_b16(), name="ivim16"), True), (synth.t2star, True),
    (synth.vfa_t1, True), (synth.biexp_t2, False)])
def test_schedule_of_a_fit(workload, flows):
    w = workload()
    s = _fitter(w)
    want = "flow" if flows else "grid"
    for iters in (64, 100, 260):
        n = _least(iters)
        assert _schedule(s, n, iters) == want and _schedule(s, n - 1, iters) == "grid"
    assert _schedule(s, 1 << 30, 63) == "grid"
    assert _schedule(_fitter(w, torch.float32), 1 << 30, 100) == "grid"
    assert _schedule(_fitter(w, dtype=torch.float64), 1 << 30, 100) == "grid"


@pytest.mark.parametrize("iters", [64, 100])
def test_flow_equals_grid_in_16_samples(iters):
    w = synth.ivim(synth.ivim_b16(), name="ivim16")
    n = _least(iters) + 3
    _, data = pipeline.synth_gpu(w, n, seed=8, device=DEV)
    data[:, 5::1001] = float("nan")
    got = []
    for block in (0, 128):  # a block size asks for the grid schedule
        s = _fitter(w)
        s.setup(pipeline.init_constant(data, w.init_values), list(w.protocol), data, list(w.lb), list(w.ub))
        assert _schedule(s, n, iters) == "flow"
        s.run(iters, block=block)
        got.append([getattr(s, k) for k in ("pars_t", "first_f", "last_f", "f_t", "lam_t", "step_type_t", "step_t",
                                            "iters_t")])
    for a, b in zip(*got):
        a, b = (x.view(torch.int32) if x.dtype == torch.float32 else x for x in (a, b))
        assert torch.equal(a, b)


# per model: one whose fits flow; one that keeps no cap; one whose samples alone are more local memory than the cap allows
@pytest.mark.parametrize("expr,pars,M,solve", [
    ("S*exp(-x*k)", ["S", "k"], 9, torch.float64), ("a+b*x+c*x**2+d*x**3+e*x**4", ["a", "b", "c", "d", "e"], 6, torch.float64),
    ("a+b*x", ["a", "b"], 70, torch.float64), ("a+b*x", ["a", "b"], 71, torch.float32)])
def test_a_compiled_model_has_nothing_left_to_compile(tmp_path, monkeypatch, expr, pars, M, solve):
    monkeypatch.setenv("PCGB_CACHE_DIR", str(tmp_path))
    gm = codegen.generate(expr, pars, ["x"])
    rc = _lib.lib().pcgb_fitter_compile(gm.source.encode(), gm.struct_name.encode(), gm.P, gm.C, M, 0,
                                        int(solve == torch.float64), str(tmp_path).encode(), None, 0)
    assert rc == 0
    programs = set(os.listdir(tmp_path))
    x = torch.linspace(0.1, 1.0, M, device=DEV)
    n = _least(64)
    data = (torch.rand(n, device=DEV) + 1.0) * torch.exp(-x[:, None])
    P = len(pars)
    s = SecondOrderLevenbergMarquardt(Expr(expr, pars, ["x"]), None, M, torch.float32, solve_dtype=solve)
    p = torch.ones((P, n), device=DEV)
    s.setup(p, x, data, [-100.0] * P, [100.0] * P)
    s.run(64)
    s.run(2, schedule="refill")
    s.run_fresh(2, 1.0)
    which, one, cost, backup = (torch.empty(k, device=DEV, dtype=t) for k, t in (
        (n, torch.int32), (n, torch.float32), (n, torch.float32), ((P, n), torch.float32)))
    count = torch.zeros(2, dtype=torch.int32, device=DEV)
    s.run_check(1, [1.0] * P, 5.0, cost, backup, one, which, count)
    s.run_select(1, cost, backup, one, which, count)
    r = SecondOrderRandomSearch(Expr(expr, pars, ["x"]), M, torch.float32, solve_dtype=solve)
    r.setup(x, data[:, :100].contiguous(), [-1.0] * P, [1.0] * P)
    r.run(2, lm_iters=2, seed=1)
    torch.cuda.synchronize()
    assert set(os.listdir(tmp_path)) == programs


def test_rest_in_long_fits_equals_grid():
    """A damping that grows slowly: a voxel at rest has far more iterations left than its growth may span, until it has few
    enough."""
    w = synth.ivim()
    iters = 1500
    n = _least(iters) + 5
    _, data = pipeline.synth_gpu(w, n, seed=9, device=DEV)
    got = []
    for block in (0, 128):
        s = _fitter(w)
        s.setup(pipeline.init_constant(data, w.init_values), list(w.protocol), data, list(w.lb), list(w.ub))
        assert _schedule(s, n, iters) == "flow"
        s.run(iters, dec=1.1, block=block)
        got.append([getattr(s, k) for k in ("pars_t", "first_f", "last_f", "f_t", "lam_t", "step_type_t", "step_t",
                                            "iters_t")])
    for a, b in zip(*got):
        a, b = (x.view(torch.int32) if x.dtype == torch.float32 else x for x in (a, b))
        assert torch.equal(a, b)
