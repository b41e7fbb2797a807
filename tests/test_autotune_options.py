"""The mixed-model autotuner's options and cache key: a choice timed with another library is not used, and no two timed
options are the same launch."""
import pytest

from pycompute_gb300 import Expr, _lib, multi, synth


def test_tuned_choice_belongs_to_one_library(monkeypatch):
    w = synth.vfa_t1()
    f = multi.MultiModelFitter([(Expr(w.expr, w.pars, w.consts), w.M)])
    monkeypatch.setattr(multi, "_library_id", lambda: "a")
    key = multi._tune_key("gpu", f, 20, (1, 2))
    assert key == multi._tune_key("gpu", f, 20, (1, 2)) != multi._tune_key("gpu", f, 100, (1, 2))
    monkeypatch.setattr(multi, "_library_id", lambda: "b")
    assert key != multi._tune_key("gpu", f, 20, (1, 2))


@pytest.mark.parametrize("block", [64, 128, 256])
def test_blocks_of_a_program(block):
    blocks = lambda r, dt=0, P=5: _lib.lib().pcgb_multi_blocks(P, dt, r, block)  # noqa: E731
    assert blocks(0) == blocks(96) == 640 // block  # the same program: one of them is timed
    assert blocks(128) == 512 // block and blocks(255) == max(1, 256 // block) == max(1, blocks(255, 1))
    assert blocks(0, P=7) == blocks(128, P=7) == 512 // block and blocks(0, 1) == 1 and blocks(-1) < 0


@pytest.mark.gpu
def test_no_option_is_timed_twice():
    import torch

    w = synth.t2star()
    n = 4096
    _, data, init, lb, ub, prot = w.generate(n, seed=3)
    jobs = lambda: [multi.MultiJob(torch.from_numpy(init.copy()).cuda(), torch.from_numpy(data).cuda(), prot, lb, ub)]  # noqa: E731
    models = [(Expr(w.expr, w.pars, w.consts), w.M)]
    best = multi.autotune(models, jobs, iters=64, blocks=(64, 256), maxrregs=(0, 96, 255), chunks=(32, 256, 4096),
                          use_cache=False, lane_options=(1,))
    seen = [(t["block"], _lib.lib().pcgb_multi_blocks(3, 0, t["maxrreg"], t["block"]), tuple(t["order"])) for t in best["trials"]]
    assert len(seen) == len(set(seen)) == 4  # two blocks, two programs each; a few voxels cut every chunk to 32
    assert best["chunk"] == 32
