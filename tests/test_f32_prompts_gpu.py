"""Attention over prompt tiles on the fp32 pipes.  Needs a GPU."""
import pytest
import torch

from test_kernels_gpu import _attention_case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("hq,hkv,hd", [(4, 2, 16), (4, 1, 16), (6, 1, 32), (2, 2, 32), (8, 2, 64), (3, 3, 64), (6, 2, 128),
                                       (2, 2, 128), (33, 1, 128)])
@pytest.mark.parametrize("window", [0, 70])
def test_attention_of_prompt_tiles(dtype, hq, hkv, hd, window):
    """Both heights of a tile at every head size, tiles of few and of all rows, one page and several, from the first position and from the middle of a page, with and
    without a window (whose pages behind it were given back); the tolerances of the general kernel's tests."""
    out, ref = _attention_case(dtype, hq, hkv, hd, [(0, 1), (0, 64), (63, 2), (130, 75)], window=window, dead_pages=True)
    torch.testing.assert_close(out, ref, **(dict(atol=2e-5, rtol=1e-5) if dtype == "float32" else dict(atol=2e-2, rtol=2e-2)))
