"""Rules that choose kernels and splits of decode steps (csrc/step_rules.cuh), compiled for the host: what was measured on 148 SMs
stays, other SM counts move the lines with them, and every shape fits an SM."""
import ctypes as C
import random
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mdlarc_scale_b200" / "csrc"
SOURCE = r"""
#include "step_rules.cuh"
extern "C" {
int splits(long long work, int t_max, int sms) { return attn_splits(work, t_max, sms); }
int scratch(long long work, int requested, int sms) { return attn_scratch_splits(work, requested, sms); }
int cta_per_item(long long n, int sms) { return attn_cta_per_item(n, sms); }
int wide(int M, int N, int sms) { return rows_wide_columns(M, N, sms); }
int transposes(int M, int N, int K, int sms) { return mid_transposes(M, N, K, sms); }
void shape(int M, int N, int K, int sms, int at_once_ctas, int* out) {
  const GmShape s = gm_shape(M, N, K, sms, [&](int n) { return at_once_ctas / n; });
  out[0] = s.rows; out[1] = s.splits; out[2] = s.stages; out[3] = s.smem();
}
int ask(int* slot, int works, int answer, int* asked) {
  return asked_once(*slot, [&](int& n) { ++*asked; n = answer; return works != 0; });
}
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), str(d / "rules.cpp"), "-o", str(d / "rules.so")], check=True)
    lib = C.CDLL(str(d / "rules.so"))
    lib.splits.argtypes = [C.c_longlong, C.c_int, C.c_int]
    lib.scratch.argtypes = [C.c_longlong, C.c_int, C.c_int]
    lib.cta_per_item.argtypes = [C.c_longlong, C.c_int]
    return lib


def shape(rules, M, N, K, sms, at_once=None):
    out = (C.c_int * 4)()
    rules.shape(M, N, K, sms, sms if at_once is None else at_once, out)
    return list(out)


# what the choices were measured with
MEASURED = {
    "splits": [((2048, 400), 1), ((6 * 20, 5200), 4), ((4, 190), 1), ((20, 10240), 8), ((20, 12288), 8), ((20, 12289), 20), ((16, 32768), 25),
               ((24, 16384), 17), ((25, 16384), 8), ((5, 20000), 64), ((4, 32768), 8), ((16 * 16, 1200), 2)],
    "wide": [((1, 4608), 0), ((1, 4736), 0), ((1, 4864), 1), ((16, 1280), 0), ((16, 3072), 0), ((16, 3200), 1), ((17, 32000), 0)],
    "transposes": [((32, 1280, 1280), 0), ((33, 1280, 1280), 1), ((24, 1280, 3456), 1), ((16, 32000, 1280), 1), ((16, 18944, 1280), 0),
                   ((256, 1280, 1280), 1), ((257, 1280, 1280), 0)],
}


@pytest.mark.parametrize("rule", sorted(MEASURED))
def test_lines_on_148_sms(rules, rule):
    for args, want in MEASURED[rule]:
        assert getattr(rules, rule)(*args, 148) == want, args
    assert not rules.cta_per_item(295, 148) and rules.cta_per_item(296, 148)


def test_lines_move_with_the_sm_count(rules):
    r = random.Random(0)
    for _ in range(3000):
        work, t_max = r.randint(1, 3000), r.randint(1, 20000)
        assert rules.splits(work, t_max, 74) == rules.splits(2 * work, t_max, 148)
    assert rules.cta_per_item(148, 74) and not rules.cta_per_item(147, 74)
    assert rules.wide(1, 2432, 74) and not rules.wide(1, 2368, 74) and rules.wide(16, 1664, 74) and not rules.wide(16, 1536, 74)
    assert rules.transposes(16, 75 * 128, 1280, 74) and not rules.transposes(16, 74 * 128, 1280, 74)
    # 24 tiles of 16 K blocks: clusters of six fill 148 SMs, fewer CTAs a cluster fit 74
    assert shape(rules, 40, 3072, 1024, 148)[1] == 6 and shape(rules, 40, 3072, 1024, 74)[1] in (1, 2, 3)


# (column tiles, K blocks) -> CTAs of a cluster: the products that test_gpu_divided_steps.py means by its clusters
DIVIDED = {(1, 1): [(6, 4), (11, 4)],
           (5, 8): [(18, 12), (12, 12), (12, 20), (21, 20), (8, 20), (15, 20), (10, 16), (6, 20), (10, 20)],
           (2, 4): [(30, 20), (53, 20), (28, 20), (41, 20), (36, 20), (47, 20), (30, 16), (48, 20)]}


@pytest.mark.parametrize("least,most", sorted(DIVIDED))
def test_clusters_of_step_products(rules, least, most):
    for tiles, blocks in DIVIDED[least, most]:
        for M in (33, 48, 80, 129, 130, 256):
            assert least <= shape(rules, M, 128 * tiles, 64 * blocks, 148, 132)[1] <= most, (tiles, blocks, M)


@pytest.mark.parametrize("sms", [1, 66, 148, 160])
def test_scratch_holds_every_choice(rules, sms):
    """Splits that no cluster merges find scratch, whatever the cache, and have a CTA iteration of rows each."""
    for work in range(1, 400):
        room = rules.scratch(work, 0, sms)
        for t_max in (1, 255, 256, 4096, 12288, 12289, 16384, 65536, 2 ** 31 - 1):
            s = rules.splits(work, t_max, sms)
            assert 1 <= s <= 64 and (s <= 8 or (s <= room and t_max >= 128 * s and rules.cta_per_item(work * s, sms)))
        assert rules.scratch(work, 5, sms) == 5 and rules.scratch(work, 99, sms) == 64


@pytest.mark.parametrize("sms", [1, 66, 132, 148, 160])
def test_shapes_fit(rules, sms):
    r = random.Random(sms)
    for _ in range(4000):
        M, N, K = r.randint(1, 256), 128 * r.randint(1, 300), 64 * r.randint(1, 260)
        at_once = r.choice([0, sms // 2, sms])
        rows, splits, stages, smem = shape(rules, M, N, K, sms, at_once)
        assert rows % 16 == 0 and M <= rows < M + 16 and stages >= 1 and 1 <= splits <= min(8, K // 64)
        assert smem <= 222 * 1024 + 1024 and smem <= 227 * 1024
        if splits > 1:
            assert N // 128 * splits <= sms and N // 128 <= at_once // splits
        # tensor memory: 128 columns up to 128 rows, 256 beyond, of 512; an SM has 228 KB of shared memory, a CTA takes 1 KB more than its own
        ctas = 228 * 1024 // (smem + 1024)
        assert ctas * (128 if rows <= 128 else 256) <= 512


def test_a_failed_query_is_asked_again(rules):
    """Clusters that run at once on a device: an error is no answer, and an answer (none at all included) is kept."""
    for answer in (0, 22):
        slot, asked = C.c_int(0), C.c_int(0)
        ask = lambda works, n: rules.ask(C.byref(slot), works, n, C.byref(asked))  # noqa: E731
        assert [ask(0, 9), ask(0, 9), ask(1, answer), ask(1, 5), ask(0, 5)] == [0, 0, answer, answer, answer]
        assert asked.value == 3
