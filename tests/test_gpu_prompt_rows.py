"""A prompt's logits do not depend on what else its call holds: its rows are summed in one order, bit for bit, whether they come
alone (a few dozen rows) or among thousands."""
import numpy as np
import pytest
import torch

import logesun_util as lu
import vodavik_util as vu
from gpu_util import have_b200
from mdlarc_scale_b200 import forward_logits, registry
from mdlarc_scale_b200.engine import Engine
from mdlarc_scale_b200.layered import Segment
from oracle import arc_model as om
from oracle import logesun as lo
from oracle import vodavik as vo

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]
LENS = [1, 40, 64, 65, 300]      # few rows in tiles of their own, one more than 64, more than a tile


@pytest.mark.parametrize("act", ["f16", "bf16"])
@pytest.mark.parametrize("size", ["tiny", "small"])
def test_grid_prompts_alone_and_among_others(size, act):
    cfg = om.make_config(size, max_seq_len=4096)
    eng = Engine(om.round_bf16(om.perturb_state(om.init_state(cfg, seed=0), seed=1)), cfg, "cuda:0", act_format=act)
    g = np.random.default_rng(3)
    n, width = len(LENS) + 40, 300
    lens = np.array(LENS + [100] * 40)
    ids = torch.from_numpy(g.integers(0, 14, (n, width)))
    pos = torch.from_numpy(np.stack([g.integers(0, m, (n, width)) for m in (30, 30, 5)], -1))
    mask = torch.from_numpy(np.arange(width)[None] < lens[:, None])
    among = forward_logits(eng, ids.cuda(), pos.cuda(), None, mask.cuda())
    for i, k in enumerate(LENS):
        alone = forward_logits(eng, ids[i:i + 1, :k].cuda(), pos[i:i + 1, :k].cuda())
        assert torch.equal(alone[0], among[i, :k]), k


# attention and recurrence; latent attention with a loop, dense and without feed-forwards (a routed layer of few rows chooses
# its experts with a kernel of its own)
MODELS = {
    "vodavik": (vo, vu.config(640, 500, [vu.attention(10, 2, 64, 64, ff=700), vu.mlstm(4, 64, 64)])),
    "logesun": (lo, lu.config(640, 500, [lu.latent(10, 64, 32, 64, 256, 128, 200, lu.dense(700)), lu.latent(5, 64, 32, 64, 256, 128, 60)],
                              loop=(0, 1, 2))),
}


@pytest.mark.parametrize("fmt", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("name", sorted(MODELS))
def test_layered_prompts_alone_and_among_others(name, fmt):
    oracle, cfg = MODELS[name]
    eng = registry.build_engine(cfg, oracle.random_weights(cfg, 5), "cuda:0", fmt)
    toks = [vu.tokens(cfg, n, 50 + i) for i, n in enumerate(LENS + [200] * 14)]

    def logits(prompts):
        s = eng.new_session(len(prompts), 320, 1, 4096, stop_on_end=False)
        out = s.step([Segment(s.acquire(), t, list(range(len(t)))) for t in prompts])
        s.poll()
        s.close()
        return out

    among = logits(toks)
    for t, want in zip(toks[:len(LENS)], among):
        assert torch.equal(logits([t])[0], want), len(t)


@pytest.mark.parametrize("fmt", ["f16", "f32"])
def test_first_tokens_alone_and_among_others(fmt):
    """The head over a few armed rows, behind a call of any size."""
    oracle, cfg = MODELS["vodavik"]
    eng = registry.build_engine(cfg, oracle.random_weights(cfg, 5), "cuda:0", fmt)
    toks = [vu.tokens(cfg, n, 50 + i) for i, n in enumerate([40] + [25] * 100)]

    def first(prompts):
        s = eng.new_session(len(prompts), 64, 1, 4096, stop_on_end=False)
        out = s.prefill_segments([Segment(s.acquire(), t, arm=True) for t in prompts])[1]
        s.poll()
        s.close()
        return out

    among = first(toks)
    assert torch.equal(first(toks[:1])[0], among[0]) and torch.equal(first(toks[1:2])[0], among[1])
