"""Prefill attention of the layered models, whose CTAs walk over query blocks and heads: many items of unequal sizes, against
the general attention path, and twice."""
import pytest
import torch

import logesun_util as lu
import vodavik_util as vu
from gpu_util import have_b200
from mdlarc_scale_b200 import registry
from mdlarc_scale_b200.layered import Segment
from oracle import logesun as lo
from oracle import vodavik as vo

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]
# one key tile and more, blocks without rows in the second query tile, blocks of one row, several blocks
EDGES = [1, 2, 127, 128, 129, 255, 256, 257, 384, 385, 513, 700]
# each head size has a kernel of its own; the windows let the second query tile skip key tiles of the first
MODELS = {
    **{f"heads_{d}_{u}": (vo, vu.config(128, 100, [vu.attention(6, 2, d, u)])) for d, u in [(64, 64), (64, 128), (128, 64), (128, 128)]},
    **{f"latent_{d}_{u}_{w}": (lo, lu.config(128, 100, [lu.latent(6, d, 32, u, 128, 128, w)]))
       for d, u, w in [(64, 64, 1000), (64, 128, 200), (128, 64, 130), (128, 128, 128)]},
}
TOL = {"f16": 1e-2, "bf16": 7e-2}        # of each path from the oracle, as everywhere for these formats


@pytest.mark.parametrize("fmt", ["f16", "bf16"])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_items_of_all_sizes(name, fmt):
    """324 items for 148 CTAs, in two calls, the second on top of keys that the first left."""
    oracle, cfg = MODELS[name]
    w = oracle.random_weights(cfg, 5)
    toks = [vu.tokens(cfg, n, 50 + i) for i, n in enumerate(EDGES * 3)]

    def logits(eng, prompts):
        s = eng.new_session(len(prompts), 700, 1, 16384, stop_on_end=False)
        slots = [s.acquire() for _ in prompts]
        out = [[] for _ in prompts]
        for part in (lambda t: t[:len(t) // 2], lambda t: t[len(t) // 2:]):
            live = [i for i, t in enumerate(prompts) if part(t)]
            got = s.step([Segment(slots[i], part(prompts[i]), list(range(len(part(prompts[i]))))) for i in live])
            for i, g in zip(live, got):
                out[i].append(g)
        s.poll()
        s.close()
        return [torch.cat(o) for o in out]

    eng = registry.build_engine(cfg, w, "cuda:0", fmt)
    among = logits(eng, toks)
    assert all(torch.equal(a, b) for a, b in zip(logits(eng, toks), among))      # the counter is back at its start
    plain = logits(registry.build_engine(cfg, w, "cuda:0", fmt, attn_path="stream"), toks)
    for n, a, b in zip(EDGES * 3, among, plain):
        assert vu.rel_error(a, b) < 2 * TOL[fmt], n
