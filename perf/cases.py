"""Work that programs have this framework do, as cases to time: grid models that score, continue and vote on puzzles,
and layered models (attention with mLSTM; latent attention with routed experts) that score and continue token sequences.

A case is a dict of plain values.  ``prepare`` makes what a program holds before the call (packed weights, prompts on the
host, a session where the program keeps one), ``run`` is one call, ``exact`` is the same result in 64 bits.

The weights are random, with one thing arranged: the row of the output matrix that belongs to the successor of a token
points along that token's embedding.  Next-token choices are then as clear as a trained model's (a chain of
successors), and two correct implementations pick the same tokens; with an unrelated output matrix nearly every step
has a near tie, and everything after the first one taken differently is another text.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from mdlarc_scale_b200 import forward_logits, generate, generate_tokens
from mdlarc_scale_b200.data import encode_example_np
from mdlarc_scale_b200.engine import Engine
from mdlarc_scale_b200.fanout import TaskTable, vote_records
from mdlarc_scale_b200.layered import Segment
from mdlarc_scale_b200.registry import build_engine
from mdlarc_scale_b200.sharding import generate_sharded_records

DEVICE = "cuda:0"

# width, heads, layers, feed-forward size of the grid model's sizes
GRID = {"tiny": (256, 4, 4, 704), "small": (768, 12, 4, 2048), "medium": (1024, 16, 8, 2752), "large": (1280, 20, 12, 3392)}
EXAMPLES = 64
START, NEWLINE, IO_SEP, END = 10, 11, 12, 13

# sizes of the layered benchmark
LAYERED = {
    1280: dict(heads=20, kv_heads=5, dim=64, vdim=64, ff=5120, glu_ff=3456, rot_dim=32, q_rank=768, kv_rank=256, expert_ff=448, shared_ff=1664),
    2048: dict(heads=16, kv_heads=4, dim=128, vdim=128, ff=8192, glu_ff=5440, rot_dim=64, q_rank=1024, kv_rank=512, expert_ff=704, shared_ff=2624),
    4096: dict(heads=32, kv_heads=8, dim=128, vdim=128, ff=16384, glu_ff=10944, rot_dim=64, q_rank=1536, kv_rank=512, expert_ff=1408, shared_ff=5312),
}
VOCAB, WINDOW, LAYERED_EXPERTS, LAYERED_TOP = 32000, 1024, 32, 4


def listed() -> list[dict]:
    return [
        # one small puzzle with the smallest model: what an interactive caller waits for
        dict(name="grid one puzzle", kind="grid_generate", size="tiny", rows=1, pairs=2, lo=3, hi=10, new=48),
        # one evaluation chunk of a mid-sized model: sixteen ragged prompts
        dict(name="grid chunk of 16", kind="grid_generate", size="medium", rows=16, pairs=3, lo=1, hi=20, new=96),
        # a few of the longest prompts: decoding over long caches
        dict(name="grid long caches", kind="grid_generate", size="large", rows=6, pairs=4, lo=18, hi=30, new=96),
        # throughput: the decode-bound batch of the benchmark
        dict(name="grid batch of 1024", kind="grid_generate", size="large", rows=1024, pairs=2, lo=3, hi=10, new=64),
        # likelihoods of ragged, odd-sized puzzles, padded positions included
        dict(name="grid scoring, ragged", kind="grid_score", size="small", rows=37, pairs=3, lo=1, hi=11),
        # likelihoods of full-size puzzles: the prefill-heavy configuration
        dict(name="grid scoring, 30 x 30", kind="grid_score", size="large", rows=4, pairs=5, lo=30, hi=30),
        # tasks through the augmentation fan-out, generation and the vote
        dict(name="fan-out and vote", kind="vote", size="medium", rows=2, pairs=3, lo=2, hi=16, perms=8, new=66),
        # one caller's continuation with a mixed attention / mLSTM model
        dict(name="mixed model, one caller", kind="vodavik_generate", width=1280, layers=4, act="f16", rows=1, lo=190, hi=190, new=48),
        # a batch of callers, bfloat16 operands
        dict(name="mixed model, batch", kind="vodavik_generate", width=2048, layers=8, act="bf16", rows=150, lo=100, hi=700, new=24),
        # prompts scored in 32-bit, as a reference run does
        dict(name="mixed model, 32-bit", kind="vodavik_score", width=1280, layers=4, act="f32", rows=2, lo=601, hi=999, portions=1),
        # a batch of callers of the latent-attention model
        dict(name="latent model, batch", kind="logesun_generate", width=1280, layers=6, act="f16", rows=48, lo=300, hi=1500, new=32),
        # long prompts of the latent-attention model in two portions
        dict(name="latent model, prompts", kind="logesun_score", width=2048, layers=6, act="f16", rows=8, lo=1500, hi=2048, portions=2),
    ]


def draw(rng: random.Random) -> dict:
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["grid_generate", "grid_generate", "grid_score", "vote", "vodavik_generate", "vodavik_score",
                       "logesun_generate", "logesun_score"])
    if kind.startswith("grid") or kind == "vote":
        c = dict(kind=kind, size=rng.choice(sorted(GRID)), rows=log(1, 1024), pairs=rng.randint(2, 5), lo=rng.randint(1, 10))
        c["hi"] = rng.randint(c["lo"], 30)
        if kind != "grid_score":
            c["new"] = log(16, 96)
        if kind == "vote":
            # whole rows of ten cells and a newline: other lengths end in a part of a row, which is no grid to vote for
            c["rows"], c["perms"], c["new"] = rng.randint(1, 2), rng.randint(1, 10), 11 * rng.randint(2, 9)
        budget = 40e12
    else:
        c = dict(kind=kind, width=rng.choice([1280, 1280, 2048, 2048, 4096]), layers=rng.choice([2, 4, 6]),
                 act=rng.choice(["f16", "f16", "bf16", "f32"]), rows=log(1, 200))
        c["hi"] = log(33, 2048)
        c["lo"] = rng.randint(1 + c["hi"] // 3, c["hi"])
        if kind.endswith("generate"):
            c["new"] = log(8, 48)
        else:
            c["portions"] = rng.randint(1, 2)
        if c["width"] == 4096:
            c["layers"] = 2
        budget = 40e12
        if c["act"] == "f32":
            c["width"], c["layers"], budget = 1280, rng.choice([2, 4]), 0.5e12
    while (work(c)["flops"] > budget or sum(_lengths(c)) > 250_000) and c["rows"] > 1:
        c["rows"] -= 1 + c["rows"] // 8
    while work(c)["flops"] > budget:
        c["hi"] = max(1, c["hi"] * 7 // 8)
        c["lo"] = min(c["lo"], c["hi"])
    return c


# ---------------------------------------------------------------------------
# sizes: a function of the case alone, so that every seed asks for the same amount of work
# ---------------------------------------------------------------------------
def _puzzle_shapes(case: dict) -> list[list[tuple[int, int]]]:
    """Grid shapes of every prompt: input and output of each pair, then the test input."""
    r = random.Random(7)
    return [[(r.randint(case["lo"], case["hi"]), r.randint(case["lo"], case["hi"])) for _ in range(2 * case["pairs"] + 1)]
            for _ in range(case["rows"])]


def _puzzle_length(shapes) -> int:
    return sum(h * (w + 1) + 1 + (i % 2 == 0) for i, (h, w) in enumerate(shapes))


def _lengths(case: dict) -> list[int]:
    if case["kind"].startswith("grid"):
        return [_puzzle_length(s) for s in _puzzle_shapes(case)]
    if case["kind"] == "vote":
        out = []
        for shapes in _puzzle_shapes(case):
            turned = [(w, h) for h, w in shapes]
            out += [_puzzle_length(s) for s in (shapes, turned) for _ in range(4 * case["perms"])]
        return out
    r = random.Random(11)
    return [r.randint(case["lo"], case["hi"]) for _ in range(case["rows"])]


def _portions(n: int, portions: int) -> list[int]:
    """Ends of a prompt's portions; the first is the longer one, off the tile sizes."""
    return [n] if portions == 1 or n < 3 else [max(1, n * 5 // 8), n]


def _wanted(a: int, b: int, n: int) -> list[int]:
    """Places whose logits are asked for in the portion a .. b - 1 of a prompt of n tokens: every 64th and the last."""
    return [p - a for p in range(a, b) if p % 64 == 63 or p == n - 1]


def work(case: dict) -> dict:
    lens = _lengths(case)
    new = case.get("new", 0)
    tokens = sum(lens) + len(lens) * max(0, new - 1)
    ctx = [n + max(0, new - 1) for n in lens]
    wide = 4 if case.get("act") == "f32" else 2
    if "size" in case:
        d, _, layers, ff = GRID[case["size"]]
        weights = layers * (4 * d * d + 3 * d * ff)
        flops = 2.0 * weights * tokens + sum(2.0 * d * layers * c * c for c in ctx)
        cached = layers * 2 * d * 2
        out = 14 * 4 * tokens
    else:
        cfg = _config(case)
        weights, active, pairs, cached = _layered_counts(case, cfg)
        asked = len(lens) * new if new else sum(len(_wanted(0, n, n)) for n in lens)
        head = cfg["width"] * cfg["vocab"]
        window = WINDOW if case["kind"].startswith("logesun") else 1 << 30
        seen = sum(c * c / 2 if c <= window else window * window / 2 + (c - window) * window for c in ctx)
        flops = 2.0 * active * tokens + 2.0 * head * asked + pairs * seen
        weights += head
        out = asked * cfg["vocab"] * 4
    # the weights cross once for the prompts and once for every further token (a step needs the token of the one before);
    # the cache is written once and read by every step
    steps = max(0, new - 1)
    cache = sum(n * cached + steps * (n + steps / 2) * cached for n in lens) if new else sum(lens) * cached
    return {"bytes": float(weights * wide * (1 + steps) + cache + out), "flops": float(flops)}


def tolerance(case: dict):
    """About four times what two orders of the same sums differ by."""
    if case["kind"] == "vote":
        return {"differ": 0.002}
    if case["kind"].startswith("grid"):
        return {"rel": 0.002, "max": 0.015, "differ": 0.002}
    if case["act"] == "f32":
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.0005}
    if case["kind"].startswith("logesun"):
        # a router's near tie may send a token to another expert of almost the same weight
        return {"rel": 0.005, "max": 0.1, "differ": 0.005} if case["act"] == "f16" else {"rel": 0.03, "max": 0.5, "differ": 0.01}
    return {"rel": 0.003, "max": 0.02, "differ": 0.002} if case["act"] == "f16" else {"rel": 0.02, "max": 0.15, "differ": 0.005}


# ---------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------
class _Random:
    """Seeded random tensors on the device, rounded to the 16-bit values that a checkpoint holds."""

    def __init__(self, seed: int):
        self.g = torch.Generator(device=DEVICE).manual_seed(1000003 + seed)

    def __call__(self, *shape, std=1.0, mean=0.0):
        return (torch.randn(shape, generator=self.g, device=DEVICE) * std + mean).to(torch.bfloat16).float()

    def matrix(self, rows, cols):
        return self(rows, cols, std=cols ** -0.5)


def _grid_model(size: str, seed: int):
    d, heads, layers, ff = GRID[size]
    r = _Random(seed)
    w = {"token_embed.weight": r(14, d), "example_embed.weight": r(EXAMPLES, d, std=0.02), "ln_f.weight": r(d, std=0.05, mean=1.0)}
    for n in range(layers):
        p = f"blocks.{n}."
        w.update({p + "ln1.weight": r(d, std=0.05, mean=1.0), p + "attn.qkv_proj.weight": r.matrix(3 * d, d),
                  p + "attn.out_proj.weight": r.matrix(d, d), p + "ln2.weight": r(d, std=0.05, mean=1.0),
                  p + "ffn.fc_gate.weight": r.matrix(ff, d), p + "ffn.fc_gate.bias": r(ff, std=0.05),
                  p + "ffn.fc_up.weight": r.matrix(ff, d), p + "ffn.fc_up.bias": r(ff, std=0.05),
                  p + "ffn.fc_down.weight": r.matrix(d, ff) * 0.5, p + "ffn.fc_down.bias": r(d, std=0.05)})
    head = r.matrix(14, d)
    for t, s in _grid_successors(seed).items():
        head[s] += w["token_embed.weight"][t] * d ** -0.5
    w["lm_head.weight"] = head.to(torch.bfloat16).float()
    config = dict(d_model=d, n_heads=heads, n_layers=layers, d_ff=ff, vocab_size=14, max_seq_len=16384, num_examples=EXAMPLES,
                  max_x=32, max_y=32, max_z=8, rope_base=10000.0, norm_eps=1e-5, use_example_embedding=True)
    return config, w


def _grid_successors(seed: int) -> dict[int, int]:
    """Rows of the ten colours in the seed's order: a new line, a separator or a start is followed by the first colour."""
    order = np.random.default_rng(seed + 3).permutation(10).tolist()
    return {**dict(zip(order, order[1:] + [NEWLINE])), NEWLINE: order[0], IO_SEP: order[0], START: order[0]}


def _config(case: dict) -> dict:
    s, width = LAYERED[case["width"]], case["width"]
    layers = []
    if case["kind"].startswith("vodavik"):
        # attention + feed-forward, mLSTM, attention on the first one's keys + feed-forward, mLSTM
        for n in range(case["layers"]):
            mixer = {"heads": s["heads"], "dim": s["dim"], "vdim": s["vdim"]}
            if n % 2:
                layers.append({"type": "mlstm", "mlp": None, "mixer": dict(mixer, gate_cap=15.0)})
                continue
            mixer.update(kv_heads=s["kv_heads"], scale=s["dim"] ** -0.5, q_temp={"coef": 0.1, "every": 256})
            if n % 4 == 2:
                mixer["kv_from"] = n - 2
            layers.append({"type": "attention", "mlp": {"kind": "dense", "ff": s["ff"]}, "mixer": mixer})
        return {"architecture": "Vodavik", "width": width, "vocab": VOCAB, "layers": layers, "norm": {"eps": 1e-6},
                "postln_alpha": 2.0, "logit_scale": 1.0}
    for n in range(case["layers"]):
        mixer = {"heads": s["heads"], "dim": s["dim"], "rot_dim": s["rot_dim"], "vdim": s["vdim"], "q_rank": s["q_rank"],
                 "kv_rank": s["kv_rank"], "mask": {"size": WINDOW}, "rot": {"base": 10000.0, "dims": s["rot_dim"]},
                 "scale": (s["dim"] + s["rot_dim"]) ** -0.5}
        mlp = {"kind": "dense", "ff": s["glu_ff"]}
        if n % 2:
            mlp = {"kind": "moe", "router": {"experts": LAYERED_EXPERTS, "top": LAYERED_TOP},
                   "expert": {"ff": s["expert_ff"], "limit": 7.0}, "shared": {"ff": s["shared_ff"], "limit": 7.0}}
        layers.append({"type": "latent_attention", "mixer": mixer, "mlp": mlp})
    return {"architecture": "Logesun", "width": width, "vocab": VOCAB, "layers": layers, "norm": {"eps": 1e-6},
            "loop": {"start": 0, "stop": 2, "times": 2}}


def _layer_runs(cfg: dict) -> list[tuple[int, bool]]:
    """(layer, whether the embedding is added ahead of it) in the order in which layers run."""
    loop = cfg.get("loop") or {"start": 0, "stop": 0, "times": 1}
    a, b = loop["start"], loop["stop"]
    runs = [(n, False) for n in range(a)]
    for k in range(loop["times"]):
        runs += [(n, k > 0 and n == a) for n in range(a, b)]
    return runs + [(n, False) for n in range(b, len(cfg["layers"]))]


def _layered_counts(case: dict, cfg: dict):
    """Weights, weights that a token passes, operations per pair of a query and a visible key, and cached bytes per
    position, over all layer runs."""
    w, width = LAYERED[case["width"]], case["width"]
    wide = 4 if case["act"] == "f32" else 2
    total = active = pairs = cached = 0
    for n, _ in _layer_runs(cfg):
        layer = cfg["layers"][n]
        m, f = layer["mixer"], layer["mlp"]
        if layer["type"] == "latent_attention":
            mix = width * (m["q_rank"] + m["kv_rank"] + m["rot_dim"] + m["heads"] * m["vdim"])
            mix += m["heads"] * ((m["dim"] + m["rot_dim"]) * m["q_rank"] + (m["dim"] + m["vdim"]) * m["kv_rank"])
            pairs += 2 * m["heads"] * (m["dim"] + m["rot_dim"] + m["vdim"])
            cached += wide * (m["kv_rank"] + m["rot_dim"])
        else:
            own = m.get("kv_heads", m["heads"]) if m.get("kv_from") is None else 0
            mix = width * (m["heads"] * (m["dim"] + 2 * m["vdim"]) + own * (m["dim"] + m["vdim"]))
            if layer["type"] == "attention":
                pairs += 2 * m["heads"] * (m["dim"] + m["vdim"])
                cached += wide * w["kv_heads"] * (m["dim"] + m["vdim"])
        total += mix
        active += mix
        if f is not None and f["kind"] == "moe":
            total += 3 * width * (LAYERED_EXPERTS * f["expert"]["ff"] + f["shared"]["ff"])
            active += 3 * width * (LAYERED_TOP * f["expert"]["ff"] + f["shared"]["ff"])
        elif f is not None:
            n_mats = 2 if cfg["architecture"] == "Vodavik" else 3
            total += n_mats * width * f["ff"]
            active += n_mats * width * f["ff"]
    return total, active, pairs, cached


def _layered_weights(cfg: dict, seed: int) -> dict:
    r, width = _Random(seed), cfg["width"]
    w = {"embed": r(cfg["vocab"], width)}
    routed = any((layer["mlp"] or {}).get("kind") == "moe" for layer in cfg["layers"])
    if routed:
        w["embed"][:, 0] = 12.0     # what every token has in common: the routers' offset
    gain = dict(std=0.1, mean=1.0)
    for n, layer in enumerate(cfg["layers"]):
        p, m, f = f"l{n}", layer["mixer"], layer["mlp"]
        x, heads = p + ".mix.", m["heads"]
        w[p + ".norm1"] = r(width, **gain)
        w[x + "o"] = r.matrix(width, heads * m["vdim"])
        if layer["type"] == "latent_attention":
            w.update({x + "dq": r.matrix(m["q_rank"], width), x + "dq.norm": r(m["q_rank"], **gain),
                      x + "uq": r.matrix(heads * (m["dim"] + m["rot_dim"]), m["q_rank"]),
                      x + "dkv": r.matrix(m["kv_rank"] + m["rot_dim"], width), x + "dkv.norm": r(m["kv_rank"], **gain),
                      x + "uk": r.matrix(heads * m["dim"], m["kv_rank"]), x + "uv": r.matrix(heads * m["vdim"], m["kv_rank"]),
                      x + "sink": r(heads, std=0.5), p + ".norm1b": r(width, std=0.1, mean=0.5)})
        else:
            w.update({x + "q": r.matrix(heads * m["dim"], width), x + "g": r.matrix(heads * m["vdim"], width)})
            kv = m.get("kv_heads", heads)
            if m.get("kv_from") is None:
                w.update({x + "k": r.matrix(kv * m["dim"], width), x + "v": r.matrix(kv * m["vdim"], width)})
            if layer["type"] == "mlstm":
                w.update({x + "norm": r(heads * m["vdim"], **gain), x + "i": r.matrix(heads, width), x + "i.b": r(heads, std=0.5),
                          x + "f": r.matrix(heads, width), x + "f.b": r(heads, std=0.5, mean=4.0)})
            else:
                w.update({x + "q.b": r(heads * m["dim"], std=0.1), x + "q.norm": r(m["dim"], **gain), x + "sink": r(heads, std=0.5)})
                if m.get("kv_from") is None:
                    w.update({x + "k.b": r(kv * m["dim"], std=0.1), x + "v.b": r(kv * m["vdim"], std=0.1), x + "k.norm": r(m["dim"], **gain)})
        if f is None:
            continue
        w[p + ".norm2"] = r(width, **gain)
        if cfg["architecture"] == "Vodavik":
            w.update({p + ".mlp.up": r.matrix(f["ff"], width), p + ".mlp.down": r.matrix(width, f["ff"])})
            continue
        units = [(p + ".mlp", f["ff"])] if f["kind"] == "dense" else (
            [(f"{p}.mlp.e{e}", f["expert"]["ff"]) for e in range(f["router"]["experts"])] + [(p + ".mlp.shared", f["shared"]["ff"])])
        for u, ff in units:
            w.update({u + ".gate": r.matrix(ff, width), u + ".up": r.matrix(ff, width), u + ".down": r.matrix(width, ff)})
        w[p + ".norm2b"] = r(width, std=0.05, mean=0.5 if f["kind"] == "dense" else 0.25)
        if f["kind"] == "moe":
            # Scores that fall off within the chosen ones: the last of them, which rounding may exchange for the next, hardly
            # counts.  With scores near one another a single such exchange outweighs all rounding errors of a pass.
            w[p + ".mlp.router"] = r.matrix(f["router"]["experts"], width) * 6.0
            w[p + ".mlp.router"][:, 0] = -1.7
    w["final.norm"] = r(width, **gain)
    head = torch.empty_like(w["embed"])
    head[_successors(seed)] = w["embed"] * width ** -0.5
    if routed:
        head[:, 0] = 0.0
    w["head"] = head.to(torch.bfloat16).float()
    return w


def _successors(seed: int) -> torch.Tensor:
    """The successor of every token of the layered models' vocabulary."""
    return torch.from_numpy(np.random.default_rng(seed + 5).permutation(VOCAB)).to(DEVICE)


# ---------------------------------------------------------------------------
# inputs, calls
# ---------------------------------------------------------------------------
def _grids(case: dict, seed: int) -> list[list[np.ndarray]]:
    g = np.random.default_rng(seed + 17)
    return [[np.where(g.random(s) < 0.6, 0, g.integers(1, 10, s)) for s in shapes] for shapes in _puzzle_shapes(case)]


def _prompts(case: dict, seed: int):
    """Tokens and positions of every puzzle's prompt."""
    out = []
    for grids in _grids(case, seed):
        parts = [encode_example_np(a, b) for a, b in zip(grids[0:-1:2], grids[1::2])] + [encode_example_np(grids[-1])]
        out.append((np.concatenate([t for t, _ in parts]), np.concatenate([p for _, p in parts])))
    return out


def _padded(prompts):
    width = max(len(t) for t, _ in prompts)
    ids = np.full((len(prompts), width), END, np.int64)
    pos, mask = np.zeros((len(prompts), width, 3), np.int64), np.zeros((len(prompts), width), bool)
    for i, (t, p) in enumerate(prompts):
        ids[i, :len(t)], pos[i, :len(t)], mask[i, :len(t)] = t, p, True
    return ids, pos, mask


def _sequences(case: dict, seed: int) -> list[list[int]]:
    g = np.random.default_rng(seed + 23)
    return [g.integers(0, VOCAB, n).tolist() for n in _lengths(case)]


def _examples(case: dict, seed: int) -> np.ndarray:
    return np.random.default_rng(seed + 29).integers(0, EXAMPLES, case["rows"])


def prepare(case: dict, seed: int) -> dict:
    s = {"case": case}
    if "size" in case:
        config, weights = _grid_model(case["size"], seed)
        s["engine"] = Engine(weights, config, DEVICE)
        if case["kind"] == "vote":
            s["tasks"] = [{"train": [{"input": a.tolist(), "output": b.tolist()} for a, b in zip(g[0:-1:2], g[1::2])],
                           "test": [{"input": g[-1].tolist()}]} for g in _grids(case, seed)]
            return s
        ids, pos, mask = _padded(_prompts(case, seed))
        examples = _examples(case, seed)
        if case["kind"] == "grid_score":
            ids, pos, mask, examples = (torch.from_numpy(a).to(DEVICE) for a in (ids, pos, mask, examples))
        s.update(ids=ids, pos=pos, mask=mask, examples=examples)
        return s
    cfg = _config(case)
    s["engine"] = build_engine(cfg, _layered_weights(cfg, seed), DEVICE, case["act"])
    s["prompts"] = _sequences(case, seed)
    if case["kind"].endswith("score"):
        lens = _lengths(case)
        s["session"] = s["engine"].new_session(len(lens), max(lens), 1, sum(lens), stop_on_end=False)
    return s


def run(s: dict):
    case, engine = s["case"], s["engine"]
    if case["kind"] == "grid_generate":
        t = generate_tokens(engine, s["ids"], s["pos"], s["mask"], s["examples"], case["new"], want_logits=True)
        return {"tokens": t.tokens, "first_logits": t.first_logits, "step_logits": t.step_logits}
    if case["kind"] == "grid_score":
        return {"logits": forward_logits(engine, s["ids"], s["pos"], s["examples"], s["mask"])}
    if case["kind"] == "vote":
        table = TaskTable(s["tasks"], DEVICE, num_color_perms=case["perms"])
        variants = table.variants()
        records = generate_sharded_records(table, variants, case["new"], 0, 1, engine)
        votes = vote_records(records, variants)
        return {"records": records, "votes": [np.array(g) for key in sorted(votes) for g in votes[key]]}
    if case["kind"].endswith("generate"):
        tokens, logits = generate(engine, s["prompts"], case["new"], return_logits=True)
        return {"tokens": np.array(tokens), "logits": torch.stack([logits[i] for i in range(len(tokens))])}
    session, out, begin = s["session"], [], [0] * len(s["prompts"])
    slots = [session.acquire() for _ in s["prompts"]]
    for k in range(case["portions"]):
        segments = []
        for i, (slot, toks) in enumerate(zip(slots, s["prompts"])):
            ends = _portions(len(toks), case["portions"])
            if k < len(ends):
                segments.append(Segment(slot, toks[begin[i]:ends[k]], _wanted(begin[i], ends[k], len(toks))))
                begin[i] = ends[k]
        out += [rows for rows in session.step(segments) if rows is not None]
    for slot in slots:
        session.release(slot)
    return {"logits": torch.cat(out)}


# ---------------------------------------------------------------------------
# the same in 64 bits, one sequence at a time
# ---------------------------------------------------------------------------
def _rms(x, weight, eps):
    x = x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps)
    return x if weight is None else x * weight.double()


def _centred(x, weight, eps):
    x = x - x.mean(-1, keepdim=True)
    return x * torch.rsqrt(x.square().mean(-1, keepdim=True) + eps) * weight.double()


def _linear(x, w, bias=None):
    y = x @ w.double().T
    return y if bias is None else y + bias.double()


def _attend(q, k, v, scale, keys=None, sink=None, window=None):
    """Causal attention, q [T, H, D], k [T, G, D], v [T, G, U] -> [T, H * U]; the first ``keys`` keys can be seen."""
    t, heads, _ = q.shape
    keys = t if keys is None else keys
    k, v = k[:keys], v[:keys]
    rep = heads // k.shape[1]
    d = torch.arange(t, device=q.device)[:, None] - torch.arange(keys, device=q.device)
    hidden = d < 0 if window is None else (d < 0) | (d >= window)
    out = []
    step = max(1, int(2e9 / (8.0 * t * keys)))
    for h in range(0, heads, step):
        of = torch.arange(h, min(heads, h + step), device=q.device)
        s = torch.einsum("thd,shd->hts", q[:, of], k[:, of // rep]) * scale
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink.double()[of, None, None].expand(-1, t, 1)], -1)
        s = torch.softmax(s, -1)[..., :keys]
        out.append(torch.einsum("hts,shu->thu", s, v[:, of // rep]))
    return torch.cat(out, 1).reshape(t, -1)


def _rotate(x, angle):
    """Rotates neighbouring pairs of x [T, H, 2 P] by angle [T, P]."""
    c, s = angle.cos()[:, None], angle.sin()[:, None]
    u, v = x[..., 0::2], x[..., 1::2]
    return torch.stack([u * c - v * s, v * c + u * s], -1).flatten(-2)


def _grid_logits(case, w, tokens, pos, example, keys):
    """Logits of every position of one sequence, of which the first ``keys`` are seen as keys."""
    d, heads, layers, _ = GRID[case["size"]]
    tokens, pos = torch.as_tensor(tokens, device=DEVICE), torch.as_tensor(pos, device=DEVICE).double()
    angles = []
    for axis, n in ((0, 10), (1, 10), (2, 12)):
        angles.append(pos[:, axis, None] * 10000.0 ** (-torch.arange(n, device=DEVICE, dtype=torch.float64) / n))
    angle = torch.cat(angles, -1)
    x = w["token_embed.weight"][tokens].double() + w["example_embed.weight"][example].double()
    for n in range(layers):
        p = f"blocks.{n}."
        qkv = _linear(_rms(x, w[p + "ln1.weight"], 1e-5), w[p + "attn.qkv_proj.weight"]).view(len(x), 3, heads, 64)
        o = _attend(_rotate(qkv[:, 0], angle), _rotate(qkv[:, 1], angle), qkv[:, 2], 0.125, keys)
        x = x + _linear(o, w[p + "attn.out_proj.weight"])
        h = _rms(x, w[p + "ln2.weight"], 1e-5)
        g = _linear(h, w[p + "ffn.fc_gate.weight"], w[p + "ffn.fc_gate.bias"])
        g = g * torch.sigmoid(g) * _linear(h, w[p + "ffn.fc_up.weight"], w[p + "ffn.fc_up.bias"])
        x = x + _linear(g, w[p + "ffn.fc_down.weight"], w[p + "ffn.fc_down.bias"])
    return _linear(_rms(x, w["ln_f.weight"], 1e-5), w["lm_head.weight"])


def _grid_chain(new: int, seed: int):
    """Tokens after a separator, and the positions of the cells they fill."""
    tokens, pos, t, x, y = [], [], IO_SEP, 0, 0
    after = _grid_successors(seed)
    for _ in range(new):
        t = after[t]
        tokens.append(t)
        pos.append((0 if t == NEWLINE else x, y, 3))
        x, y = (0, min(y + 1, 29)) if t == NEWLINE else (min(x + 1, 30), y)
    return np.array(tokens), np.array(pos)


def _mlstm(w, x, m, h):
    """The gated recurrence as a sum over earlier tokens."""
    t, heads = h.shape[0], m["heads"]
    q = _linear(h, w[x + "q"]).view(t, heads, -1) * m["dim"] ** -0.5
    k, v = _linear(h, w[x + "k"]).view(t, heads, -1), _linear(h, w[x + "v"]).view(t, heads, -1)
    cap = m["gate_cap"]
    i = cap * torch.tanh(_linear(h, w[x + "i"], w[x + "i.b"]) / cap)
    f = torch.nn.functional.logsigmoid(cap * torch.tanh(_linear(h, w[x + "f"], w[x + "f.b"]) / cap)).cumsum(0)
    weight = f.T[:, :, None] - f.T[:, None, :] + i.T[:, None, :]         # log weight of token s at token t
    weight = weight.masked_fill(torch.ones(t, t, device=h.device).triu(1).bool(), -math.inf)
    top = torch.maximum(weight.amax(-1), f.T)                            # the empty state's stabiliser is 0
    weight = torch.exp(weight - top[..., None]) * torch.einsum("thd,shd->hts", q, k)
    den = torch.maximum(weight.sum(-1).abs(), torch.exp(-top)) + 1e-6
    o = torch.einsum("hts,shu->thu", weight, v) / den.T[..., None]
    o = _rms(o, None, 1e-6).reshape(t, -1) * w[x + "norm"].double()
    return _linear(o * torch.sigmoid(_linear(h, w[x + "g"])), w[x + "o"])


def _mixed_logits(cfg, w, tokens, asked):
    eps, x, cache = cfg["norm"]["eps"], w["embed"][tokens].double(), {}
    t = len(x)
    for n, layer in enumerate(cfg["layers"]):
        p, m = f"l{n}", layer["mixer"]
        a = p + ".mix."
        if layer["type"] == "mlstm":
            y = _mlstm(w, a, m, x)
        else:
            if m.get("kv_from") is None:
                k = _linear(x, w[a + "k"], w[a + "k.b"]).view(t, m["kv_heads"], -1)
                cache[n] = _rms(k, w[a + "k.norm"], eps), _linear(x, w[a + "v"], w[a + "v.b"]).view(t, m["kv_heads"], -1)
            k, v = cache[m.get("kv_from", n)]
            temp = 1 + m["q_temp"]["coef"] * torch.log1p((torch.arange(t, device=x.device) + 1).div(m["q_temp"]["every"], rounding_mode="floor").double())
            q = _rms(_linear(x, w[a + "q"], w[a + "q.b"]).view(t, m["heads"], -1), w[a + "q.norm"], eps) * temp[:, None, None]
            o = _attend(q, k, v, m["scale"], sink=w[a + "sink"])
            y = _linear(o * torch.sigmoid(_linear(x, w[a + "g"])), w[a + "o"])
        x = _centred(cfg["postln_alpha"] * x + y, w[p + ".norm1"], eps)
        if layer["mlp"] is not None:
            y = _linear(torch.relu(_linear(x, w[p + ".mlp.up"])).square(), w[p + ".mlp.down"])
            x = _centred(cfg["postln_alpha"] * x + y, w[p + ".norm2"], eps)
    return _linear(_centred(x[asked], w["final.norm"], eps), w["head"]) * cfg["logit_scale"]


def _clamped(w, u, limit, h):
    g, up = _linear(h, w[u + ".gate"]).clamp(max=limit), _linear(h, w[u + ".up"]).clamp(-limit, limit)
    return _linear(g * torch.sigmoid(1.702 * g) * (up + 1), w[u + ".down"])


def _mixture(w, p, f, h):
    weight, chosen = torch.sigmoid(_linear(h, w[p + ".mlp.router"])).topk(f["router"]["top"], -1)
    y = _clamped(w, p + ".mlp.shared", f["shared"]["limit"], h)
    for e in range(f["router"]["experts"]):
        row, place = (chosen == e).nonzero(as_tuple=True)
        if len(row):
            y.index_add_(0, row, _clamped(w, f"{p}.mlp.e{e}", f["expert"]["limit"], weight[row, place, None] * h[row]))
    return y


def _latent_logits(cfg, w, tokens, asked):
    eps, embed = cfg["norm"]["eps"], w["embed"][tokens].double()
    x, t = embed, len(embed)
    for n, again in _layer_runs(cfg):
        p, m, f = f"l{n}", cfg["layers"][n]["mixer"], cfg["layers"][n]["mlp"]
        a, heads, rank = p + ".mix.", m["heads"], m["kv_rank"]
        x = x + embed if again else x
        h = _rms(x, w[p + ".norm1"], eps)
        freq = m["rot"]["base"] ** (-torch.arange(0, m["rot"]["dims"], 2, device=x.device, dtype=torch.float64) / m["rot"]["dims"])
        angle = torch.arange(t, device=x.device).double()[:, None] * freq
        y = _linear(h, w[a + "dkv"])
        c = _rms(y[:, :rank], w[a + "dkv.norm"], eps)
        kr = _rotate(y[:, None, rank:], angle).expand(-1, heads, -1)
        q = _linear(_rms(_linear(h, w[a + "dq"]), w[a + "dq.norm"], eps), w[a + "uq"]).view(t, heads, -1)
        q = torch.cat([q[..., :m["dim"]], _rotate(q[..., m["dim"]:], angle)], -1)
        k = torch.cat([_linear(c, w[a + "uk"]).view(t, heads, -1), kr], -1)
        o = _attend(q, k, _linear(c, w[a + "uv"]).view(t, heads, -1), m["scale"], sink=w[a + "sink"], window=m["mask"]["size"])
        x = x + _rms(_linear(o, w[a + "o"]), w[p + ".norm1b"], eps)
        h = _rms(x, w[p + ".norm2"], eps)
        if f["kind"] == "dense":
            g = _linear(h, w[p + ".mlp.gate"])
            y = _linear(g * torch.sigmoid(g) * _linear(h, w[p + ".mlp.up"]), w[p + ".mlp.down"])
        else:
            y = _mixture(w, p, f, h)
        x = x + _rms(y, w[p + ".norm2b"], eps)
    return _linear(_rms(x[asked], w["final.norm"], eps), w["head"])


@torch.no_grad()
def exact(case: dict, seed: int):
    lens = _lengths(case)
    if case["kind"] == "vote":
        return None     # bytes of decoded grids: nothing that 64 bits would say more exactly
    if "size" in case:
        _, w = _grid_model(case["size"], seed)
        prompts, examples = _prompts(case, seed), _examples(case, seed)
        if case["kind"] == "grid_score":
            ids, pos, _ = _padded(prompts)
            return {"logits": torch.stack([_grid_logits(case, w, ids[i], pos[i], examples[i], n) for i, n in enumerate(lens)])}
        chain, cells = _grid_chain(case["new"], seed)
        rows = []
        for (toks, pos), e in zip(prompts, examples):
            x = _grid_logits(case, w, np.concatenate([toks, chain[:-1]]), np.concatenate([pos, cells[:-1]]), e, len(toks) + len(chain) - 1)
            rows.append(x[len(toks) - 1:])
        rows = torch.stack(rows)
        return {"tokens": rows.argmax(-1).int(), "first_logits": rows[:, 0], "step_logits": rows}
    cfg = _config(case)
    w = _layered_weights(cfg, seed)
    logits = _mixed_logits if cfg["architecture"] == "Vodavik" else _latent_logits
    sequences = _sequences(case, seed)
    if case["kind"].endswith("generate"):
        after, rows = _successors(seed).tolist(), []
        for toks in sequences:
            for _ in range(case["new"] - 1):
                toks = toks + [after[toks[-1]]]
            rows.append(logits(cfg, w, torch.tensor(toks, device=DEVICE), torch.arange(len(toks) - case["new"], len(toks), device=DEVICE)))
        rows = torch.stack(rows)
        return {"tokens": rows.argmax(-1).cpu().numpy(), "logits": rows}
    out = []
    for k in range(case["portions"]):
        for toks in sequences:
            ends = _portions(len(toks), case["portions"])
            if k < len(ends):
                a = ends[k - 1] if k else 0
                asked = [a + p for p in _wanted(a, ends[k], len(toks))]
                if asked:
                    out.append(logits(cfg, w, torch.tensor(toks, device=DEVICE), torch.tensor(asked, device=DEVICE)))
    return {"logits": torch.cat(out)}
