"""Prefill calls planned on the device against the host's plan of the same padded batch."""
import weakref

import numpy as np
import pytest
import torch

from gpu_util import have_b200
from mdlarc_scale_b200 import inference
from mdlarc_scale_b200.engine import PaddedBatch, Session, plan_prefill
from test_gpu_step_cluster import batch, engine

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]


def masks(kind, n, S, g):
    lens = g.integers(0, S + 1, n)
    lens[0], lens[-1] = S, max(1, S // 3)
    at = np.arange(S)[None, :]
    if kind == "full":
        return np.ones((n, S), bool)
    if kind == "right":
        return at < lens[:, None]
    if kind == "left":
        return at >= S - lens[:, None]
    return g.random((n, S)) < 0.7          # holes


@pytest.mark.parametrize("kind", ["full", "right", "left", "holes"])
@pytest.mark.parametrize("n,S", [(1, 1), (5, 31), (3, 256), (4, 1023), (3, 1025), (2, 2300), (300, 40)])
def test_plan_is_the_host_plan(kind, n, S):
    g = np.random.default_rng(n * 7919 + S)
    wide = np.int64 if n % 2 else np.int32
    ids = g.integers(0, 14, (n, S)).astype(wide)
    pos = np.stack([g.integers(0, 32, (n, S)), g.integers(0, 32, (n, S)), g.integers(0, 6, (n, S))], -1).astype(wide)
    mask = masks(kind, n, S, g)
    rows = np.arange(n // 3, n)
    for source in ("host", "device"):
        move = (lambda a: a) if source == "host" else (lambda a: torch.from_numpy(a).cuda())
        batch = PaddedBatch(move(ids), move(pos), None if kind == "full" and source == "device" else move(mask), "cuda:0")
        assert np.array_equal(batch.lens, mask.sum(1))
        for causal, everything, first in ((True, False, True), (True, True, False), (False, False, True), (False, True, True)):
            want = plan_prefill(ids, pos, mask, rows, is_causal=causal, all_positions=everything, with_first=first)
            got = batch.plan(rows, causal, everything, first)
            for name in ("token_ids", "pos_xyz", "seq", "kv_slot", "kv_count", "kv_row", "first_row", "first_seq", "prompt_len",
                         "grid_x", "grid_y", "grid_in_output"):
                a, b = getattr(want, name), getattr(got, name)
                assert (a is None) == (b is None) and (a is None or torch.equal(a, b.cpu())), (source, causal, everything, name)
            for name in ("n_tokens", "n_kv_rows", "n_first", "kv_row_identity"):
                assert getattr(want, name) == getattr(got, name), (source, causal, everything, name)
            # every row lies in one block, of one sequence, with that sequence's keys
            seen = np.full(want.n_tokens, -1)
            for r0, k, kv0 in zip(got.qblock_row0.tolist(), got.qblock_rows.tolist(), got.qblock_kv0.tolist()):
                assert 1 <= k <= 256 and (seen[r0:r0 + k] == -1).all() and len(set(want.seq[r0:r0 + k].tolist())) == 1
                seen[r0:r0 + k] = kv0
            base = np.cumsum(mask[rows].sum(1)) - mask[rows].sum(1)
            assert np.array_equal(seen, base[want.seq.numpy() - rows[0]])


def test_shapes_that_do_not_fit_are_refused():
    ids, pos = np.zeros((2, 5), np.int64), np.zeros((2, 5, 3), np.int64)
    for bad_pos, bad_mask in ((pos[:, :4], None), (pos[:1], None), (pos[..., :2], None), (pos, np.ones((2, 6), bool)), (pos, np.ones((1, 5), bool))):
        with pytest.raises(ValueError):
            PaddedBatch(ids, bad_pos, bad_mask, "cuda:0")


def test_rows_behind_the_batch_are_left_out():
    """Positions and masks of more sequences than there are tokens for, as the host's plan takes them."""
    g = np.random.default_rng(3)
    ids, pos, mask = g.integers(0, 14, (3, 20)), g.integers(0, 5, (5, 20, 3)), masks("right", 5, 20, g)
    want = plan_prefill(ids, pos, mask, np.arange(3), all_positions=True, with_first=False)
    for move in (lambda a: a, lambda a: torch.from_numpy(a).cuda()):
        got = PaddedBatch(move(ids), move(pos), move(mask), "cuda:0").plan(np.arange(3), all_positions=True, with_first=False)
        for name in ("token_ids", "pos_xyz", "seq", "kv_slot", "kv_count", "kv_row"):
            assert torch.equal(getattr(want, name), getattr(got, name).cpu()), name


def test_the_batch_is_gone_when_steps_begin(monkeypatch):
    """Generation holds the padded arrays on the device for the prompt alone."""
    eng = engine(128, 192, 1)
    ids, pos, mask, ex = batch(64, [300, 280])
    made, left = [], []

    class Noted(PaddedBatch):
        def __init__(self, *args):
            super().__init__(*args)
            made.append(weakref.ref(self.ids))
            made.append(weakref.ref(self.pos))

        def plan(self, *args, **kw):
            p = super().plan(*args, **kw)
            made.append(weakref.ref(p.pos_xyz))
            return p

    decode = Session.decode
    monkeypatch.setattr(inference, "PaddedBatch", Noted)
    monkeypatch.setattr(Session, "decode", lambda self, n: (left.extend(w() is not None for w in made), decode(self, n))[1])
    inference.generate_tokens(eng, ids, pos, mask, ex, 4)
    assert len(made) == 3 and left and not any(left)
    eng.close()
