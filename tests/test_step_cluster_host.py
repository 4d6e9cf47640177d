"""The rule that puts decode steps into one cluster (csrc/step_rules.cuh), compiled for the host."""
import ctypes as C
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "mdlarc_scale_b200" / "csrc"
SOURCE = r"""
#include "step_rules.cuh"
extern "C" int fits(int rows, int d, int dff, int layers, int t, int cl) { return step_cluster_fits(rows, d, dff, layers, t, cl); }
extern "C" void smem(int rows, int d, int dff, int cl, int* out) {
  const StepClusterSmem s = step_cluster_smem(rows, d, dff, d / 64, cl);
  const int v[] = {s.xn, s.hs, s.q, s.rec, s.red, s.tokens, s.head, s.even, s.odd, s.total};
  for (int i = 0; i < 10; ++i) out[i] = v[i];
}
"""


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    d = tmp_path_factory.mktemp("rules")
    (d / "rules.cpp").write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-I", str(CSRC), str(d / "rules.cpp"), "-o", str(d / "rules.so")], check=True)
    return C.CDLL(str(d / "rules.so"))


@pytest.mark.parametrize("args,want", [
    ((1, 256, 704, 4, 216, 16), 1), ((4, 256, 704, 4, 400, 16), 1), ((5, 256, 704, 4, 216, 16), 0), ((0, 256, 704, 4, 216, 16), 0),
    ((1, 256, 704, 4, 2300, 16), 1), ((1, 256, 704, 4, 4096, 16), 0), ((1, 768, 2048, 4, 216, 16), 0), ((1, 512, 1024, 1, 64, 16), 0),
    ((1, 192, 704, 1, 64, 16), 0), ((1, 256, 700, 1, 64, 16), 0), ((1, 256, 704, 4, 216, 8), 0), ((1, 128, 192, 2, 64, 8), 1)])
def test_lines(rules, args, want):
    assert rules.fits(*args) == want


def test_what_fits_lies_apart_in_shared_memory(rules):
    seen = 0
    for d in range(128, 513, 128):
        for dff in range(64, 2049, 64):
            for rows in range(1, 5):
                for cl in (8, 16):
                    if not rules.fits(rows, d, dff, 1, 64, cl):
                        continue
                    seen += 1
                    out = (C.c_int * 10)()
                    rules.smem(rows, d, dff, cl, out)
                    xn, hs, q, rec, red, tokens, head, even, odd, total = out
                    up = lambda a, b: -(-a // b)
                    qkv, gu, narrow = up(3 * d // 16, cl), 2 * up(dff // 16, cl), up(d // 16, cl)
                    parts = lambda k: 8 if k >= 512 else 4 if k >= 256 else 2 if k >= 128 else 1
                    assert xn >= 2 * 8 * d * 4 and hs - xn >= 8 * (2 * d + 64) and q - hs >= 8 * (2 * dff + 64) and rec - q >= 16 * d
                    items = rows * (d // 64)
                    assert red - rec >= max(items * max(1, cl // items), 1) * 68 * 4
                    assert tokens - red >= 160 * 4 * max(max(qkv, gu) * parts(d), narrow * max(parts(d), parts(dff)))
                    assert head - tokens >= (14 + rows) * d * 4 and even - head >= 15 * d * 4
                    assert odd - even >= max(qkv, gu) * 32 * d and total - odd >= narrow * 32 * max(d, dff) and total <= 220 * 1024
                    assert all(v % 16 == 0 for v in out) and even % 128 == 0 and odd % 128 == 0
    assert seen > 100


@pytest.mark.parametrize("args,want", [
    ((1, 128, 512, 1, 30000), 1), ((1, 256, 704, 1, 12000), 1), ((4, 256, 704, 1, 1200), 1), ((4, 256, 704, 4, 580), 1), ((2, 384, 448, 4, 300), 1),
    ((4, 384, 256, 1, 300), 1), ((4, 384, 256, 1, 1200), 0), ((3, 384, 64, 1, 2400), 0), ((4, 384, 448, 4, 300), 0), ((1, 384, 448, 1, 9000), 0)])
def test_caches_and_rows_that_launches_read_sooner(rules, args, want):
    """Both sides were measured; what the cluster is slower at goes to the launches."""
    assert rules.fits(*args, 16) == want


def test_widths_that_shared_memory_holds(rules):
    widest = {d: max((dff for dff in range(64, 4097, 64) if rules.fits(1, d, dff, 1, 64, 16)), default=0) for d in range(128, 1025, 128)}
    assert widest == {128: 1536, 256: 1024, 384: 448, **{d: 0 for d in range(512, 1025, 128)}}
