"""32-bit products as sums of bf16 pieces on the matrix unit, against 64 bits and against 32-bit multiply-adds."""
import pytest
import torch

from gpu_util import have_b200, stream
from mdlarc_scale_b200 import _lib

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not have_b200(), reason="needs a B200")]


def product(a, w, path=_lib.GEMM_AUTO):
    y = torch.full((a.shape[0], w.shape[0]), float("nan"), device="cuda")
    _lib.check(_lib.load().arcb_op_gemm(a.data_ptr(), w.data_ptr(), y.data_ptr(), a.shape[0], w.shape[0], a.shape[1], _lib.ACT_F32, path, stream()))
    return y


def operands(M, N, K, kind):
    g = torch.Generator(device="cuda").manual_seed(M * 31 + N * 7 + K)
    a, w = torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g) * K ** -0.5
    if kind == "wide":          # factors of either size
        a, w = a * torch.randn(M, K, device="cuda", generator=g).exp(), w * torch.randn(N, K, device="cuda", generator=g).exp()
    if kind == "16-bit weights":
        w = w.bfloat16().float()
    if kind == "mixed weights":  # blocks with and without finer pieces, one after the other and within one
        w[:, ::2] = w[:, ::2].bfloat16().float()
        w[:, : K // 2] = w[:, : K // 2].bfloat16().float()
    return a, w


@pytest.mark.parametrize("kind", ["plain", "wide", "16-bit weights", "mixed weights"])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (127, 128, 128), (128, 256, 192), (129, 128, 1344), (300, 384, 640), (70, 640, 5120)])
def test_against_64_bits(M, N, K, kind):
    a, w = operands(M, N, K, kind)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    got, plain = product(a, w).double(), product(a, w, _lib.GEMM_SIMT).double()
    # dropped pieces 2^-23; ten additions of the matrix unit and two of the drain, a unit in the last place (2^-23) each; then one
    # rounding (2^-24) a chunk of 128
    assert ((got - ref).abs() <= size * 2.0 ** -23 * (1 + 12 + K / 256)).all()
    if K >= 1280:               # where sums are long, no further off than multiply-adds one after the other
        assert (got - ref).norm() <= (plain - ref).norm()
    # a row's sums do not depend on the rows beside it
    assert torch.equal(product(a[M // 2:], w), got[M // 2:].float())


@pytest.mark.parametrize("where", ["a", "w"])
@pytest.mark.parametrize("value", [float("inf"), float("-inf"), float("nan"), 3.4e38])
def test_values_without_pieces(value, where):
    a, w = operands(130, 256, 192, "plain")
    (a if where == "a" else w)[5, 70] = value
    got, plain = product(a, w), product(a, w, _lib.GEMM_SIMT)
    assert torch.equal(got.isnan(), plain.isnan()) and torch.equal(got.isinf(), plain.isinf())
    hit = torch.zeros_like(got, dtype=torch.bool)
    if where == "a":
        hit[5] = True
    else:
        hit[:, 5] = True
    assert torch.equal(got[hit].nan_to_num(), plain[hit].nan_to_num())
    ref = a.double() @ w.double().T
    assert ((got - ref).abs()[~hit] <= (a.double().abs() @ w.double().abs().T)[~hit] * 2.0 ** -19).all()


@pytest.mark.parametrize("value", [float("inf"), float("nan"), 3.4e38])
@pytest.mark.parametrize("M,N,K", [(128, 128, 64), (200, 256, 192), (70, 128, 1280)])
def test_rows_beside_such_values_keep_their_bits(M, N, K, value):
    a, w = operands(M, N, K, "plain")
    clean = product(a, w)
    for row, col in ((0, None), (M - 1, None), (M // 2, N - 1), (None, 0), (None, 77)):
        b, v = a.clone(), w.clone()
        if row is not None:
            b[row, K - 1] = value
        if col is not None:
            v[col, 0] = value
        keep = torch.ones_like(clean, dtype=torch.bool)
        if row is not None:
            keep[row] = False
        if col is not None:
            keep[:, col] = False
        got, plain = product(b, v), product(b, v, _lib.GEMM_SIMT)
        assert torch.equal(got[keep], clean[keep])
        assert torch.equal(got[~keep].nan_to_num(), plain[~keep].nan_to_num())
        assert torch.equal(got.isnan(), plain.isnan()) and torch.equal(got.isinf(), plain.isinf())
    b = torch.full_like(a, value)                # all of them
    assert torch.equal(product(b, w).nan_to_num(), product(b, w, _lib.GEMM_SIMT).nan_to_num())


@pytest.mark.parametrize("kind", ["plain", "wide", "16-bit weights", "mixed weights"])
@pytest.mark.parametrize("K", [64, 128, 192, 320, 640, 1280, 2560])
def test_no_further_off_than_multiply_adds(K, kind):
    """Of 131072 sums: the norm of all errors, at every length."""
    a, w = operands(256, 512, K, kind)
    ref = a.double() @ w.double().T
    got, plain = ((product(a, w, path).double() - ref).norm() for path in (_lib.GEMM_AUTO, _lib.GEMM_SIMT))
    assert got <= plain
