"""Decode steps inside one cluster against the separate launches (which a session with a chosen split count takes)."""
import numpy as np
import pytest
import torch

from gpu_util import have_b200
from mdlarc_scale_b200 import _lib
from mdlarc_scale_b200.engine import Engine, initial_grid_state
from mdlarc_scale_b200.inference import generate_tokens

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]


def engine(d, dff, layers, act="f16", seed=0, chain=False):
    g = torch.Generator().manual_seed(seed)

    def r(*s, std=1.0, mean=0.0):
        return (torch.randn(s, generator=g) * std + mean).to(torch.bfloat16).float()
    w = {"token_embed.weight": r(14, d), "example_embed.weight": r(8, d, std=0.02), "ln_f.weight": r(d, std=0.05, mean=1.0),
         "lm_head.weight": r(14, d, std=d ** -0.5)}
    if chain:
        w["lm_head.weight"] = (w["token_embed.weight"].roll(1, 0) * d ** -0.5).bfloat16().float()
    for n in range(layers):
        p = f"blocks.{n}."
        w.update({p + "ln1.weight": r(d, std=0.05, mean=1.0), p + "attn.qkv_proj.weight": r(3 * d, d, std=d ** -0.5),
                  p + "attn.out_proj.weight": r(d, d, std=d ** -0.5), p + "ln2.weight": r(d, std=0.05, mean=1.0),
                  p + "ffn.fc_gate.weight": r(dff, d, std=d ** -0.5), p + "ffn.fc_gate.bias": r(dff, std=0.05),
                  p + "ffn.fc_up.weight": r(dff, d, std=d ** -0.5), p + "ffn.fc_up.bias": r(dff, std=0.05),
                  p + "ffn.fc_down.weight": r(d, dff, std=0.5 * dff ** -0.5), p + "ffn.fc_down.bias": r(d, std=0.05)})
    config = dict(d_model=d, n_heads=d // 64, n_layers=layers, d_ff=dff, vocab_size=14, max_seq_len=4096, num_examples=8, max_x=32,
                  max_y=32, max_z=8, rope_base=10000.0, norm_eps=1e-5, use_example_embedding=True)
    return Engine(w, config, "cuda:0", act_format=act)


def batch(rows, lens, seed=0):
    g = np.random.default_rng(seed)
    lens = np.resize(np.array(lens), rows)
    width = int(lens.max())
    ids, mask = g.integers(0, 12, (rows, width)), np.arange(width)[None] < lens[:, None]
    pos = np.stack([g.integers(0, m, (rows, width)) for m in (30, 30, 5)], -1)
    return ids, pos, mask, g.integers(0, 8, rows)


# one to four rows and one more; fewer and more (row, head) items than CTAs, items that do not divide them; K of fewer blocks than warps; more
# tiles and blocks than are requested ahead; prompts at the edges of the slices of 16 keys
@pytest.mark.parametrize("act", ["f16", "bf16"])
@pytest.mark.parametrize("rows", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("d,dff,layers", [(128, 64, 1), (128, 192, 3), (256, 704, 4), (256, 896, 2), (384, 256, 1), (256, 64, 2), (512, 1024, 1)])
def test_steps_match_separate_launches(d, dff, layers, rows, act):
    eng = engine(d, dff, layers, act, seed=rows)
    ids, pos, mask, ex = batch(rows, [1, 15, 16, 17, 130, 257, 90, 33], seed=d)
    new = 9
    forced = np.random.default_rng(1).integers(0, 12, (rows, new)).astype(np.int32)
    lib, counts, logits = _lib.load(), [], []
    for splits in (0, 1):
        lib.arcb_launch_count(1)
        out = generate_tokens(eng, ids, pos, mask, ex, new, stop_on_end=False, forced=forced, want_logits=True, attn_splits=splits)
        counts.append(lib.arcb_launch_count(1))
        logits.append(out.step_logits)
    # steps that fit were not launched one kernel after the other
    fits = rows <= 4 and (d, dff) != (512, 1024)
    assert counts[0] < counts[1] - 20 if fits else counts[0] >= counts[1] - 1
    # both round at the same places; sums in another order turn a rounding (2^-11, bf16 2^-8) over here and there
    scale = logits[1].square().mean().sqrt()
    assert bool(torch.isfinite(logits[0]).all())
    assert float((logits[0] - logits[1]).square().mean().sqrt() / scale) < (2 ** -9 if act == "f16" else 2 ** -6)
    eng.close()


def grid_after(state, tok):
    """Grid state after a fed token (src/inference.py:127-168)."""
    x, y = state
    if tok in (10, 12):
        return 0, 0
    if tok == 11:
        return 0, min(y + 1, 29)
    return (min(x + 1, 30), y) if tok < 10 else (x, y)


def uniform(seed, stream, index):
    m = 2 ** 64 - 1
    z = (seed + 0x9E3779B97F4A7C15 * (stream + 1) + 0xD1B54A32D192ED03 * (index + 1)) & m
    z = (z ^ z >> 30) * 0xBF58476D1CE4E5B9 & m
    z = (z ^ z >> 27) * 0x94D049BB133111EB & m
    return ((z ^ z >> 31) >> 40) / 2 ** 24


def choices(logits, state, row, index, constraints=None, temperature=0.0, top_k=None, sample_seed=0):
    """Tokens that these logits allow (several where a rounding decides a sample)."""
    adj = logits.numpy().astype(np.float32).copy()
    c = constraints or {}
    adj[list(c.get("disallow_tokens", ()))] = -np.inf
    if "palette_mask" in c:
        adj[:10][~c["palette_mask"][row]] -= np.float32(2.0)
    if "target_shape" in c and min(c["target_shape"][row]) >= 0:
        (h, w), (x, y) = c["target_shape"][row], state
        adj[slice(0, 10) if x >= w else slice(11, 12)] -= np.float32(2.0)
        if y >= h:
            adj[:10] -= np.float32(2.0)
            adj[11] -= np.float32(2.0)
    if temperature <= 0:
        return {int(adj.argmax())}
    kept = sorted(range(14), key=lambda v: (-adj[v], v))[:top_k or 14]
    p = np.array([np.exp((float(adj[v]) - float(adj.max())) / temperature) if v in kept else 0.0 for v in range(14)])
    at, ends = uniform(sample_seed, row, index), np.cumsum(p) / p.sum()
    return {int(np.argmax(ends > min(max(u, 0.0), 1 - 1e-9))) for u in (at - 1e-5, at, at + 1e-5)}


# The row of the output matrix that belongs to a token's successor points along that token's embedding: rows count up to END and
# on from 0, so they end (and at different steps).
@pytest.mark.parametrize("kw", [
    dict(), dict(stop_on_end=False), dict(freeze_finished=False),
    dict(constraints=dict(palette_mask=np.tile(np.arange(10) % 3 == 0, (4, 1)), target_shape=np.full((4, 2), 3), disallow_tokens=(10, 12))),
    dict(constraints=dict(target_shape=np.array([[2, 5], [1, 1], [-1, -1], [4, 2]]))),
    dict(temperature=1.3, top_k=5, sample_seed=11), dict(temperature=3.0, sample_seed=2 ** 63 + 5)], ids=lambda kw: "-".join(kw) or "plain")
def test_loop_ends_freezes_and_constrains(kw):
    """Every token is the one that its logits, the row's grid and the request's options give; the logits are those of separate launches
    fed the same tokens."""
    eng = engine(256, 704, 2, chain=True)
    ids, pos, mask, ex = batch(4, [40, 9, 77, 130])
    new = 40
    a = generate_tokens(eng, ids, pos, mask, ex, new, want_logits=True, **kw)
    toks, logits = a.tokens.cpu().numpy(), a.step_logits.cpu()
    last = mask.sum(1) - 1
    gx, gy, _ = initial_grid_state(ids[np.arange(4), last], pos[np.arange(4), last], np.ones(4, bool))
    frozen_rows = kw.get("stop_on_end", True) and kw.get("freeze_finished", True)
    options = {k: v for k, v in kw.items() if k not in ("stop_on_end", "freeze_finished")}
    alive = np.zeros(toks.shape, bool)
    for r in range(4):
        state, ended = (int(gx[r]), int(gy[r])), False
        for i, tok in enumerate(toks[r].tolist()):
            alive[r, i] = not (frozen_rows and ended)
            assert tok in (choices(logits[r, i], state, r, i, **options) if alive[r, i] else {13}), (r, i)
            ended |= tok == 13
            state = grid_after(state, tok)
    if not kw:
        assert (toks == 13).any(1).all() and not alive.all()       # rows have ended, and stayed
    if kw == dict(freeze_finished=False):
        assert (toks == 13).any(1).all() and ((toks[:, :-1] == 13) & (toks[:, 1:] != 13)).any()
    forced = np.full((4, new), 13, np.int32)
    forced[:, :toks.shape[1]] = toks
    b = generate_tokens(eng, ids, pos, mask, ex, new, stop_on_end=False, forced=forced, want_logits=True, attn_splits=1)
    n = toks.shape[1]
    scale = float(b.step_logits[:, :n].square().mean().sqrt())
    assert float((logits[:, :n] - b.step_logits.cpu()[:, :n])[torch.from_numpy(alive)].abs().max()) < 0.02 * scale
    eng.close()


def test_steps_in_parts_are_steps_in_one_go():
    eng = engine(256, 704, 3)
    ids, pos, mask, ex = batch(2, [50, 31])
    from mdlarc_scale_b200.engine import plan_prefill
    got = []
    for parts in ([12], [1, 1, 10], [5, 7]):
        s = eng.new_session(2, 80, 13, 128, stop_on_end=False, want_step_logits=True)
        s.prefill(plan_prefill(ids, pos, mask, np.arange(2)).to(torch.device("cuda:0")), torch.from_numpy(ex).int().cuda())
        for n in parts:
            s.decode(n)
        s.poll()
        got.append((s.out_tokens.clone(), s.step_logits.clone()))
        assert 0.0 <= s.attention_probe_ms() < 1.0
        s.close()
    for t, lg in got[1:]:
        assert torch.equal(t, got[0][0]) and torch.equal(lg, got[0][1])


def test_full_cache_drops_keys_and_reports_it():
    eng = engine(128, 192, 1)
    ids, pos, mask, ex = batch(1, [30])
    from mdlarc_scale_b200.engine import plan_prefill
    for splits in (0, 1):
        s = eng.new_session(1, 32, 200, 64, stop_on_end=False, attn_splits=splits)
        s.prefill(plan_prefill(ids, pos, mask, np.arange(1)).to(torch.device("cuda:0")), torch.from_numpy(ex).int().cuda())
        s.decode(s.t_max - 30 + 3)
        with pytest.raises(_lib.ArcbError):
            s.poll()
        s.close()


def test_probe_waits_for_its_own_steps():
    """Of steps on a stream that has later work queued, and on one that is gone."""
    eng = engine(128, 192, 1)
    ids, pos, mask, ex = batch(1, [30])
    from mdlarc_scale_b200.engine import plan_prefill
    s = eng.new_session(1, 60, 20, 64, stop_on_end=False)
    s.prefill(plan_prefill(ids, pos, mask, np.arange(1)).to(torch.device("cuda:0")), torch.from_numpy(ex).int().cuda())
    s.decode(4)
    after = torch.cuda.Event()
    torch.cuda._sleep(600_000_000)               # 0.3 s
    after.record()
    assert 0.0 < s.attention_probe_ms() < 1.0 and not after.query()
    torch.cuda.synchronize()
    handle = np.zeros(1, np.int64)
    assert torch.cuda.cudart().cudaStreamCreate(handle.ctypes.data) == torch.cuda.cudart().cudaError.success
    with torch.cuda.stream(torch.cuda.ExternalStream(int(handle[0]))):
        s.decode(4)
    assert torch.cuda.cudart().cudaStreamDestroy(int(handle[0])) == torch.cuda.cudart().cudaError.success
    assert 0.0 < s.attention_probe_ms() < 1.0
    s.poll()
    # captured by the caller: the probe is of the replay
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        s.decode(2)
    g.replay()
    assert 0.0 < s.attention_probe_ms() < 1.0
    s.poll()
    s.close()
