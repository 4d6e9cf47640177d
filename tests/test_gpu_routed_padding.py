"""Routed experts of 32-bit models: slots behind an expert's last row are padding that nothing writes, and nothing may depend on it."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

import logesun_util as lu
from gpu_util import have_b200
from mdlarc_scale_b200 import registry
from mdlarc_scale_b200.layered import Segment
from oracle import logesun as lo

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]


def session(eng, rows, fill):
    s = eng.new_session(rows, 40, 1, 2048, stop_on_end=False)
    s.workspace.fill_(fill)                      # bytes 0xff: every number of it is NaN, in 16 bits and in 32
    return s


def scores(s, toks):
    slots = [s.acquire() for _ in toks]
    out = torch.cat(s.step([Segment(k, t, list(range(len(t)))) for k, t in zip(slots, toks)]))
    s.poll()
    for k in slots:
        s.release(k)
    return out


# experts with one row, with many, with more than a tile of them, and without any
@pytest.mark.parametrize("experts,top,lens", [(7, 3, [1]), (33, 4, [5, 9]), (9, 2, [33, 40, 17, 2]), (2, 2, [39, 39, 39, 39]), (64, 1, [3])])
@pytest.mark.parametrize("fmt", ["f32", "f16"])
def test_results_do_not_depend_on_the_workspace(experts, top, lens, fmt):
    cfg = lu.config(200, 100, [lu.latent(3, 24, 16, 40, 56, 72, 33, lu.moe(experts, top, 40, shared=72))])
    eng = registry.build_engine(cfg, lo.random_weights(cfg, 3), "cuda:0", fmt)
    toks = [lu.tokens(cfg, n, i) for i, n in enumerate(lens)]
    clean, dirty = (scores(session(eng, len(lens), fill), toks) for fill in (0, 255))
    assert bool(torch.isfinite(clean).all()) and torch.equal(clean, dirty)


def test_time_does_not_depend_on_the_workspace():
    cfg = lu.config(640, 100, [lu.latent(3, 24, 16, 40, 56, 72, 33, lu.moe(32, 4, 448))])
    eng = registry.build_engine(cfg, lo.random_weights(cfg, 3), "cuda:0", "f32")
    toks = [lu.tokens(cfg, 30, 1)]
    spent = []
    for fill in (0, 255):
        scores(session(eng, 1, fill), toks)
        fresh = [session(eng, 1, fill) for _ in range(5)]
        with profile(activities=[ProfilerActivity.CUDA]) as p:
            for s in fresh:
                scores(s, toks)
            torch.cuda.synchronize()
        spent.append(sum(e.self_device_time_total for e in p.key_averages() if "gemm_split" in e.key))
    assert 0 < spent[1] < 1.5 * spent[0]         # sums by multiply-adds take several times as long
