"""The kernels of the 32-bit run alone: the float32 product against float64, at the edges of their tiles,
and against themselves under other cuts of the same rows (a sum's order hangs on the operation's sizes only)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
EPS = 2.0 ** -24        # half a unit in the last place of float32


def _product(a, w, rows):
    from bare_cuda_4gib_b200.kernels import lib as K
    out = torch.full((rows, w.shape[0]), float("nan"), device=DEV)
    K.matmul_plain(a, w, out, rows)
    return out


@pytest.mark.parametrize("n,k", [(1, 4), (63, 36), (130, 300), (2560, 2048), (5000, 260), (300, 5632)])
def test_matmul_f32(n, k):
    torch.manual_seed(n + k)
    a, w = torch.randn(600, k, device=DEV), torch.randn(n, k, device=DEV)
    want, size = a.double() @ w.double().t(), a.double().abs() @ w.double().abs().t()
    whole = _product(a, w, 600)
    # chains of k / 16 + 32 packed FMAs at most, then the pair and the eight segments: each rounds once, relative to at most
    # the sum of the sizes
    assert ((whole.double() - want).abs() <= (k / 16 + 32 + 9) * EPS * size).all()
    for rows in (1, 2, 3, 4, 5, 8, 9, 16, 17, 24, 25, 33, 64, 65, 100, 257):
        assert torch.equal(_product(a, w, rows), whole[:rows]), rows


def test_matmul_f32_strided_rows_and_bad_values():
    torch.manual_seed(3)
    wide = torch.randn(40, 2 * 64, device=DEV)
    a, w = wide[:, 64:], torch.randn(70, 64, device=DEV)
    wide[7, 70] = float("inf")
    wide[9, 65] = float("nan")
    got, clean = _product(a, w, 40), _product(a.contiguous(), w, 40)
    assert torch.equal(got.nan_to_num(7.0, 8.0, 9.0), clean.nan_to_num(7.0, 8.0, 9.0))
    bad = ~torch.isfinite(got).all(-1)
    assert bad.nonzero().flatten().tolist() == [7, 9]        # a row's values stay in that row
