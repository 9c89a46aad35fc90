"""The 32-bit path's contraction by pieces on the tensor cores and its attention over prompt tiles.  Needs a GPU."""
import pytest
import torch

from test_kernels_gpu import DEV, _attention_case

pytestmark = pytest.mark.gpu


def _gemm(x, w, epilogue=None, out=None):
    from dlgo_b200.csrc import kernels as k
    got = k.gemm_simt(x, w, k.EPI_STORE_F32 if epilogue is None else epilogue, out, static_weight=True)
    k.check_device_errors()
    return got


@pytest.mark.parametrize("N,K_", [(16400, 64), (2052, 516), (2049, 512), (530, 2052), (257, 4160), (129, 8192)])
@pytest.mark.parametrize("M", [17, 64, 65, 128, 129, 260])
def test_products_by_pieces(M, N, K_):
    """Rows and outputs at the edges of tiles, K that leaves chunks or spans short or empty (every weight has 2^20 values and
    more, from where pieces are used).  In units of 2^-24 of the products' absolute sum: a chunk's two instructions cut off
    at most 2 each, a running sum of K / 256 chunks and eight spans round by 1 each, the pieces left out and the cuts of
    the small sums (2^-7 as large, 3 K / 128 instructions) are below 2 + K / 2700."""
    from dlgo_b200.csrc import kernels as k
    torch.manual_seed(M + N)
    x = torch.randn(M, K_, device=DEV)
    w = torch.randn(N, K_, device=DEV)
    ref = x.double() @ w.double().t()
    bound = (x.double().abs() @ w.double().abs().t()) * (K_ / 200 + 16) * 2.0 ** -24
    got = _gemm(x, w)
    assert ((got.double() - ref).abs() <= bound).all()
    acc = torch.randn(M, N + 3, device=DEV)
    before = acc.clone()
    _gemm(x, w, k.EPI_ADD_F32, acc[:, :N])
    assert torch.equal(acc[:, :N], before[:, :N] + got) and torch.equal(acc[:, N:], before[:, N:])
    # among more than 16 rows, a row does not depend on those beside it, on the tile's width, nor on how x lies in memory
    for at, n in ((M - 17, 17), (M // 2, M - M // 2), (0, min(M, 64))):
        if n > 16:
            assert torch.equal(_gemm(x[at:at + n].contiguous(), w), got[at:at + n])
    wide = torch.randn(M, K_ + 5, device=DEV)
    wide[:, 3:3 + K_] = x
    assert torch.equal(_gemm(wide[:, 3:3 + K_], w), got)


@pytest.mark.parametrize("M", [40, 200])
@pytest.mark.parametrize("K_", [2048, 8192])
def test_products_by_pieces_are_no_further_off_than_those_of_the_fp32_pipes(M, K_):
    """A weight that does not lie on 16 bytes is contracted on the fp32 pipes."""
    torch.manual_seed(K_)
    x, w = torch.randn(M, K_, device=DEV), torch.randn(1024, K_, device=DEV) * 0.02
    aside = torch.empty(1024 * K_ + 1, device=DEV)[1:].view(1024, K_).copy_(w)
    ref = x.double() @ w.double().t()
    split, pipes = ((_gemm(x, a).double() - ref).norm() for a in (w, aside))
    assert 0 < split <= pipes


@pytest.mark.parametrize("M", [40, 70])
def test_products_by_pieces_with_infinities_and_no_numbers(M):
    x, w = torch.randn(M, 2048, device=DEV), torch.randn(1024, 2048, device=DEV)
    x[0, 5], x[1, 9], w[11, 700], w[12, 1], w[13] = float("inf"), float("nan"), -float("inf"), 3.4e38, 0.0
    x[:, 1] = 1e-3
    ref = (x.double() @ w.double().t()).float()
    got = _gemm(x, w)
    finite = torch.isfinite(ref)
    assert torch.equal(torch.isnan(got), torch.isnan(ref)) and torch.equal(torch.isfinite(got), finite)
    assert torch.equal(got[torch.isinf(ref)], ref[torch.isinf(ref)])
    torch.testing.assert_close(got[finite], ref[finite], atol=2e-3, rtol=1e-5)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("hq,hkv,hd", [(4, 2, 16), (6, 1, 32), (8, 2, 64), (3, 3, 64), (6, 2, 128), (33, 1, 128)])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_of_prompt_tiles(dtype, hq, hkv, hd, window):
    """Tiles of few and of all rows, one page and several, from the first position and from the middle of a page, with and
    without a window (whose pages behind it were given back); the tolerances of the general kernel's tests."""
    out, ref = _attention_case(dtype, hq, hkv, hd, [(0, 1), (0, 64), (63, 2), (130, 75)], window=window, dead_pages=True)
    torch.testing.assert_close(out, ref, **(dict(atol=2e-5, rtol=1e-5) if dtype == "float32" else dict(atol=2e-2, rtol=2e-2)))
