"""Kernels of steps with few rows, through the C ABI and small models, at the edges of their tiles and of the rules that
choose them."""
import math

import numpy as np
import pytest
import torch

from gpu_util import have_b200, stream, to_act
from mdlarc_scale_b200 import _lib, registry
from mdlarc_scale_b200.engine import Engine
from mdlarc_scale_b200.inference import generate_tokens
from mdlarc_scale_b200.layered import Segment
from oracle import arc_model as om
from oracle import vodavik as vo
from vodavik_util import attention, config, mlstm, oracle_logits, rel_error, tokens

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]


@pytest.fixture(scope="module")
def lib():
    return _lib.load()


@pytest.mark.parametrize("d", [128, 640, 1280, 2048, 2176])
@pytest.mark.parametrize("rows", [1, 2048, 2049])
def test_row_kernels_on_both_sides_of_their_rules(lib, rows, d):
    """Norm and head with a CTA per row (up to 2048 rows of 2048 columns) and with a warp per row beyond."""
    g = torch.Generator(device="cuda").manual_seed(rows + d)
    x = torch.randn(rows, d, device="cuda", generator=g) * 3
    w = torch.randn(d, device="cuda", generator=g)
    out = torch.empty(rows, d, device="cuda", dtype=torch.float16)
    _lib.check(lib.arcb_op_rmsnorm(x.data_ptr(), w.data_ptr(), out.data_ptr(), rows, d, 1e-5, _lib.ACT_F16, stream()))
    n = x.double() * torch.rsqrt(x.double().square().mean(-1, keepdim=True) + 1e-5) * w.double()
    # half: 2^-11 of rounding (2^-25 where it is subnormal); fp32: a sum of d squares and four products
    assert ((out.double() - n).abs() <= n.abs() * (2 ** -11 + 1e-6 * math.sqrt(d)) + 2 ** -24).all()
    head = torch.randn(14, d, device="cuda", generator=g) * d ** -0.5
    logits = torch.empty(rows, 14, device="cuda")
    am = torch.empty(rows, dtype=torch.int32, device="cuda")
    _lib.check(lib.arcb_op_head(x.data_ptr(), None, w.data_ptr(), head.data_ptr(), logits.data_ptr(), am.data_ptr(), rows, d, 1e-5, stream()))
    ref = n @ head.double().T
    bound = (n.abs() @ head.double().abs().T) * 2 ** -24 * (d / 32 + 16)    # longest chain of additions
    assert ((logits.double() - ref).abs() <= bound).all()
    assert torch.equal(am.long(), logits.argmax(-1))


@pytest.mark.parametrize("splits", [31, 32, 33, 64])
def test_split_merge(lib, splits):
    """Two lanes' worth of splits, some of them without keys."""
    B, H, T = 2, 3, 700
    g = torch.Generator(device="cuda").manual_seed(splits)
    q = to_act(torch.randn(B, H, 64, device="cuda", generator=g), _lib.ACT_F16)
    k, v = (torch.randn(B, H, T, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    lens = torch.tensor([700, 35], dtype=torch.int32, device="cuda")
    out = torch.empty_like(q)
    scratch = torch.empty(lib.arcb_attn_scratch_bytes(B, H, splits), dtype=torch.uint8, device="cuda")
    _lib.check(lib.arcb_op_decode_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), None, lens.data_ptr(), None, B, H, T,
                                            splits, scratch.data_ptr(), _lib.ACT_F16, stream()))
    for i, n in enumerate(lens.tolist()):
        p = torch.softmax(torch.einsum("hd,htd->ht", q[i].double(), k[i, :, :n].double()) / 8, -1)
        ref = torch.einsum("ht,htd->hd", p, v[i, :, :n].double())
        assert ((out[i].double() - ref).abs() <= ref.abs() * 2 ** -11 + 1e-5).all()


@pytest.mark.parametrize("T", [256, 1100])
@pytest.mark.parametrize("splits", [1, 2, 5, 8])
def test_splits_merged_in_a_cluster(lib, splits, T):
    """Splits of a launch whose cache has 128 rows for each of them; fewer rows fall back to the merge launch.  Rows at the
    edges of a split's 16-row granules, empty splits, skipped and empty items, permuted cache rows."""
    lens_l = [n for n in (1, 15, 16, 17, 127, 129, 255, 256, 640, 1023, 1100, 0, 300) if n <= T]
    B, H = len(lens_l), 3
    g = torch.Generator(device="cuda").manual_seed(splits + T)
    q = to_act(torch.randn(B, H, 64, device="cuda", generator=g), _lib.ACT_F16)
    k, v = (torch.randn(B, H, T, 64, device="cuda", generator=g).to(torch.bfloat16) for _ in range(2))
    lens = torch.tensor(lens_l, dtype=torch.int32, device="cuda")
    seqs = torch.randperm(B, device="cuda", generator=g).to(torch.int32)
    skip = torch.zeros(B, dtype=torch.uint8, device="cuda")
    skip[2] = 1
    scratch = torch.full((max(4, lib.arcb_attn_scratch_bytes(B, H, splits)),), 255, dtype=torch.uint8, device="cuda")
    outs = []
    for _ in range(2):
        out = torch.full_like(q, float("nan"))
        _lib.check(lib.arcb_op_decode_attention(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), seqs.data_ptr(), lens.data_ptr(),
                                                skip.data_ptr(), B, H, T, splits, scratch.data_ptr(), _lib.ACT_F16, stream()))
        outs.append(out)
    assert torch.equal(outs[0], outs[1])
    for i, n in enumerate(lens_l):
        if n == 0 or i == 2:
            assert (outs[0][i] == 0).all()
            continue
        s = int(seqs[i])
        p = torch.softmax(torch.einsum("hd,htd->ht", q[i].double(), k[s, :, :n].double()) / 8, -1)
        ref = torch.einsum("ht,htd->hd", p, v[s, :, :n].double())
        assert ((outs[0][i].double() - ref).abs() <= ref.abs() * 2 ** -11 + 1e-5).all()


@pytest.mark.parametrize("rows,t_max,scratch", [(2, 12290, True), (2, 12200, True), (1, 12400, False), (6, 12290, True), (7, 12290, False)])
def test_few_sequences_over_a_long_cache(lib, rows, t_max, scratch):
    """More splits than a cluster merges where four heads x `rows` leave the machine idle in eight (5 to 24 of them, beyond 12288
    rows): a long and some short caches, against one split.  Both sum in 32 bits and round a layer's outputs to halves once:
    a rounding turned over is 2^-11 of one element."""
    cfg = om.make_config("tiny", max_seq_len=16384)
    eng = Engine(om.round_bf16(om.perturb_state(om.init_state(cfg, seed=0), seed=1)), cfg, "cuda:0")
    g = np.random.default_rng(rows)
    new = 4
    lens = np.array([t_max - new] + [40] * (rows - 1))
    width = int(lens.max())
    ids, mask = g.integers(0, 12, (rows, width)), np.arange(width)[None] < lens[:, None]
    pos = np.stack([g.integers(0, m, (rows, width)) for m in (30, 30, 5)], -1)
    forced = g.integers(0, 12, (rows, new)).astype(np.int32)
    out = [generate_tokens(eng, ids, pos, mask, None, new, stop_on_end=False, forced=forced, want_logits=True, attn_splits=s).step_logits
           for s in (0, 1, 0)]
    assert torch.equal(out[0], out[2]) and bool(torch.isfinite(out[0]).all())
    assert rel_error(out[0][:, 1:].flatten(0, 1), out[1][:, 1:].flatten(0, 1)) < 1e-3
    sizes = [eng.new_session(rows, t_max, new, 64, attn_splits=s).workspace.numel() for s in (0, 1)]
    assert (sizes[0] > sizes[1]) == scratch


@pytest.mark.parametrize("fmt", [_lib.ACT_F16, _lib.ACT_BF16])
@pytest.mark.parametrize("M", [1, 8, 9, 16, 17, 32, 33, 64, 65])
@pytest.mark.parametrize("N,K", [(128, 64), (384, 256), (1280, 704), (1024, 3392), (3072, 256), (3200, 704), (4736, 128), (4864, 704)])
def test_few_row_products(lib, M, N, K, fmt):
    """Row tiles of 8, 16, 32 and 64 and one row beyond; K of fewer blocks than warps, and of more than are in flight."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = to_act(torch.randn(M, K, device="cuda", generator=g), fmt)
    w = to_act((torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(torch.bfloat16).float(), fmt)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.double() @ w.double().T
    bound = (a.double().abs() @ w.double().abs().T) * 2 ** -24 * (K / 16 + 16)
    y = torch.full((M + 1, N), 7.0, device="cuda")
    _lib.check(lib.arcb_op_gemm(a.data_ptr(), w.data_ptr(), y.data_ptr(), M, N, K, fmt, _lib.GEMM_AUTO, stream()))
    assert ((y[:M].double() - ref).abs() <= bound).all() and (y[M] == 7).all()
    x0 = torch.randn(M + 1, N, device="cuda", generator=g)
    got = []
    for _ in range(2):
        x = x0.clone()
        _lib.check(lib.arcb_op_gemm_residual(a.data_ptr(), w.data_ptr(), bias.data_ptr(), x.data_ptr(), M, N, K, fmt, _lib.GEMM_AUTO, stream()))
        got.append(x)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0][M], x0[M])
    if M <= 16 and K >= 128:      # K is added in other parts than by a tcgen05 tile or by the CUDA cores: the kernel meant here ran
        for path in (_lib.GEMM_TC_1CTA, _lib.GEMM_SIMT):
            x = x0.clone()
            _lib.check(lib.arcb_op_gemm_residual(a.data_ptr(), w.data_ptr(), bias.data_ptr(), x.data_ptr(), M, N, K, fmt, path, stream()))
            assert not torch.equal(x, got[0])
    ref = ref + x0[:M].double() + bias.double()
    assert ((got[0][:M].double() - ref).abs() <= bound + (ref.abs() + x0[:M].double().abs() + bias.double().abs()) * 2 ** -22).all()


@pytest.mark.parametrize("fmt", [_lib.ACT_F16, _lib.ACT_BF16])
@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 127, 128, 129, 150, 241, 256, 257])
@pytest.mark.parametrize("N,K", [(128, 64), (384, 256), (1024, 2752), (3072, 1024), (8448, 320), (19200, 256)])
def test_mid_row_products(lib, M, N, K, fmt):
    """Transposed tiles of up to 256 rows, and on the other side of their rule: fewer K blocks than CTAs of a cluster, uneven
    shares of them, clusters of one to eight, more tiles than SMs."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = to_act(torch.randn(M, K, device="cuda", generator=g), fmt)
    w = to_act((torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(torch.bfloat16).float(), fmt)
    bias = torch.randn(N, device="cuda", generator=g)
    ref = a.double() @ w.double().T
    bound = (a.double().abs() @ w.double().abs().T) * 2 ** -24 * (K / 16 + 16)
    x0 = torch.randn(M + 1, N, device="cuda", generator=g)
    got = []
    for _ in range(2):
        x = x0.clone()
        _lib.check(lib.arcb_op_gemm_residual(a.data_ptr(), w.data_ptr(), bias.data_ptr(), x.data_ptr(), M, N, K, fmt, _lib.GEMM_AUTO, stream()))
        got.append(x)
    assert torch.equal(got[0], got[1]) and torch.equal(got[0][M], x0[M])
    ref = ref + x0[:M].double() + bias.double()
    assert ((got[0][:M].double() - ref).abs() <= bound + (ref.abs() + x0[:M].double().abs() + bias.double().abs()) * 2 ** -22).all()


@pytest.mark.parametrize("fmt", ["f16", "bf16"])
@pytest.mark.parametrize("slots", [33, 80, 131])
@pytest.mark.parametrize("name", ["mixed", "plain_heads", "wide_group", "unequal"])
def test_mid_row_steps(name, slots, fmt):
    """A decode step of that many sequences: heads of 64 and 128 columns with and without norms, gates, caches, vocabularies."""
    from vodavik_util import CONFIGS
    steps_match(CONFIGS[name], slots, fmt)


@pytest.mark.parametrize("fmt", ["f16", "bf16"])
@pytest.mark.parametrize("slots", [1, 8, 9, 16, 17])
def test_steps_with_wide_projections(slots, fmt):
    """Recurrent projections (no norms) of more 16-column tiles than CTAs run at once, beside attention's normed ones."""
    steps_match(config(128, 77, [mlstm(20, 64, 64), attention(30, 5, 64, 64, ff=4800)]), slots, fmt)


def steps_match(cfg, slots, fmt):
    w = vo.random_weights(cfg, 5)
    eng = registry.build_engine(cfg, w, "cuda:0", fmt)
    s = eng.new_session(slots, 16, 1, 8 * slots, stop_on_end=False)
    toks = [tokens(cfg, 2 + i % 6, 100 + i) for i in range(slots)]
    at = [s.acquire() for _ in range(slots)]
    s.step([Segment(a, t[:-1], []) for a, t in zip(at, toks)])
    got = torch.cat(s.step([Segment(a, t[-1:], [0]) for a, t in zip(at, toks)]))
    s.poll()
    want = torch.stack([oracle_logits(cfg, w, t)[-1] for t in toks])
    assert rel_error(got, want) < (1e-2 if fmt == "f16" else 6e-2)


@pytest.mark.parametrize("M,N,K", [(32, 128, 32), (33, 128, 32), (64, 384, 96), (65, 256, 64), (700, 1280, 320), (2500, 2048, 96)])
def test_cuda_core_products(lib, M, N, K):
    """32-row tiles, 64-row tiles from 33 rows on and 128-row tiles from two waves on: every sum runs over K in order, so the
    same rows give the same bits through any of them."""
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = to_act(torch.randn(M, K, device="cuda", generator=g), _lib.ACT_F16)
    w = to_act((torch.randn(N, K, device="cuda", generator=g) / math.sqrt(K)).to(torch.bfloat16).float(), _lib.ACT_F16)
    y, few = (torch.full((M + 1, N), 7.0, device="cuda") for _ in range(2))
    _lib.check(lib.arcb_op_gemm(a.data_ptr(), w.data_ptr(), y.data_ptr(), M, N, K, _lib.ACT_F16, _lib.GEMM_SIMT, stream()))
    for m in range(0, M, 32):
        rows = min(32, M - m)
        _lib.check(lib.arcb_op_gemm(a[m:].data_ptr(), w.data_ptr(), few[m:].data_ptr(), rows, N, K, _lib.ACT_F16, _lib.GEMM_SIMT, stream()))
    assert torch.equal(y, few) and (y[M] == 7).all()
    ref = a.double() @ w.double().T
    assert ((y[:M].double() - ref).abs() <= (a.double().abs() @ w.double().abs().T) * 2 ** -24 * K).all()


# widths whose norms hold a row in one to eight registers a thread, and one beyond; a vocabulary off and on quads of columns
@pytest.mark.parametrize("width,vocab", [(500, 333), (1000, 332), (2050, 96), (4100, 64)])
def test_layered_steps_of_few_rows(width, vocab):
    cfg = config(width, vocab, [attention(4, 2, 64, 64, ff=200), mlstm(2, 64, 64)])
    w = vo.random_weights(cfg, width)
    toks = tokens(cfg, 70, 3)
    want = oracle_logits(cfg, w, toks)
    for fmt, tol in (("f32", 3e-5), ("f16", 1e-2), ("bf16", 6e-2)):
        eng = registry.build_engine(cfg, w, "cuda:0", fmt)
        for first in (1, 9, 40, 66):
            s = eng.new_session(3, 70, 1, 70, stop_on_end=False)
            slot = s.acquire()
            rows = [s.step([Segment(slot, toks[:first], list(range(first)))])[0]]
            rows += [s.step([Segment(slot, [t], [0])])[0] for t in toks[first:]]
            s.poll()
            s.close()
            assert rel_error(torch.cat(rows), want) < tol
