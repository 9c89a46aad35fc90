"""What the device sampler copies to the GPU in one piece: requests, draw indices and windows of recent tokens."""
import numpy as np
import pytest
import torch

from dlgo_b200.sampling.sampler import _int32_rows


@pytest.mark.parametrize("kind", [list, tuple, np.array])
@pytest.mark.parametrize("lengths", [[], [0], [64], [3, 65, 64, 200, 0]])
def test_rows_keep_their_last_tokens_and_are_padded(kind, lengths):
    width = 64
    rows = [list(range(100 * i, 100 * i + n)) for i, n in enumerate(lengths)]
    got = _int32_rows((kind([5, 6]), kind([2 ** 31 - 1, 0])), [kind(r) for r in rows], width, torch.device("cpu"))
    want = [5, 6, 2 ** 31 - 1, 0] + [t for r in rows for t in (r[-width:] + [-1] * width)[:width]]
    assert got.dtype == torch.int32 and got.tolist() == want
