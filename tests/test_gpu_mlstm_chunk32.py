"""Recurrence of 32-bit models with 64-wide heads by chunks of 64 tokens, against the oracle in 64 bits and the recurrence
token by token."""
import pytest
import torch

from gpu_util import have_b200
from mdlarc_scale_b200 import registry
from mdlarc_scale_b200.layered import Segment
from oracle import vodavik as vo
from vodavik_util import config, mlstm, oracle_logits, rel_error, tokens

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]
# A chunk's result is a sum of at most 64 + 64 products of 64 terms, each rounded to 2^-24 of the largest: below 2^-24 * 2 * 64,
# 8e-6 of the layer's output; two layers and the projections around them leave 3e-5, what every 32-bit result of these
# models is held to.
TOL = 3e-5


def portions(eng, toks, sizes):
    s = eng.new_session(3, len(toks), 1, 4096, stop_on_end=False)
    other, slot, at, rows = s.acquire(), s.acquire(), 0, []
    for n in sizes:
        # beside another sequence of the same lengths, so that a call holds more than one segment
        seg = [Segment(k, toks[at:at + n], list(range(n))) for k in (slot, other)]
        rows.append(s.step(seg)[0])
        at += n
    s.poll()
    s.close()
    return torch.cat(rows)


@pytest.mark.parametrize("sizes", [[1], [2], [63], [64], [65], [128], [130], [64, 64], [1, 64, 1], [65, 63, 2], [200, 131]], ids=str)
@pytest.mark.parametrize("heads,dim,vdim", [(3, 64, 64), (2, 40, 56)])
@pytest.mark.parametrize("bias", [-9.0, 0.0, 9.0])
def test_chunks(sizes, heads, dim, vdim, bias):
    """Portions that end on, ahead of and behind a chunk, from an empty and from a carried state; forget gates that drop
    everything at once, the usual ones, and ones that keep everything."""
    cfg = config(160, 200, [mlstm(heads, dim, vdim), mlstm(heads, dim, vdim)])
    w = vo.random_weights(cfg, 7)
    for name in [n for n in w if n.endswith(".mix.f.b")]:
        w[name] = w[name] + bias
    toks = tokens(cfg, sum(sizes), 3)
    got = portions(registry.build_engine(cfg, w, "cuda:0", "f32"), toks, sizes)
    assert rel_error(got, oracle_logits(cfg, w, toks)) < TOL
    assert rel_error(got, portions(registry.build_engine(cfg, w, "cuda:0", "f32", mlstm_path="step"), toks, sizes)) < 2 * TOL


@pytest.mark.parametrize("n", [40, 64, 65, 150])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_later_tokens_leave_earlier_ones_alone(n, value):
    """One token of a prompt whose embedding is no number: the rows ahead of it keep every bit."""
    cfg = config(160, 200, [mlstm(3, 64, 64), mlstm(2, 40, 56)])
    w = vo.random_weights(cfg, 7)
    w["embed"][199] = value
    eng = registry.build_engine(cfg, w, "cuda:0", "f32")
    toks = [t % 199 for t in tokens(cfg, n, 3)]
    clean = portions(eng, toks, [n])
    for at in {0, 1, 3, 30, n - 1, min(n - 1, 63), min(n - 1, 64), min(n - 1, 66)}:
        got = portions(eng, toks[:at] + [199] + toks[at + 1:], [n])
        assert torch.equal(got[:at], clean[:at]) and bool(torch.isfinite(got[:at]).all()), at
        assert bool(got[at].isnan().all())


@pytest.mark.parametrize("n,chunked", [(1, 0), (36, 0), (37, 37), (63, 63), (64, 64), (65, 64), (88, 64), (89, 89), (128, 128), (152, 128), (153, 153)])
def test_few_tokens_are_walked(n, chunked):
    """Rows up to the first chunk's length, and few behind the last whole one, by the walk; the others by chunks."""
    cfg = config(160, 200, [mlstm(3, 64, 64)])
    w = vo.random_weights(cfg, 7)
    toks = tokens(cfg, n, 3)
    eng, step = (registry.build_engine(cfg, w, "cuda:0", "f32", mlstm_path=path) for path in ("auto", "step"))
    got, walked = portions(eng, toks, [n]), portions(step, toks, [n])
    assert rel_error(got, oracle_logits(cfg, w, toks)) < TOL
    if chunked == 0:
        assert torch.equal(got, walked)
    else:                      # sums in another order: not one row in eight has the walk's bits all over
        assert int((got[:chunked] == walked[:chunked]).all(dim=1).sum()) <= chunked // 8
    # what is walked behind chunks is what a portion of its own gets (one token alone is a decode step)
    if 0 < chunked < n - 1:
        assert torch.equal(got, portions(eng, toks, [chunked, n - chunked]))
