"""What the device sampler copies to the GPU in one piece: requests, draw indices and windows of recent tokens."""
from collections import deque

import numpy as np
import pytest
import torch

from dlgo_b200.sampling.sampler import DeviceSampler, SamplerConfig, _int32_rows


@pytest.mark.parametrize("kind", [list, tuple, np.array])
@pytest.mark.parametrize("lengths", [[], [0], [64], [3, 65, 64, 200, 0]])
def test_rows_keep_their_last_tokens_and_are_padded(kind, lengths):
    width = 64
    rows = [list(range(100 * i, 100 * i + n)) for i, n in enumerate(lengths)]
    got = _int32_rows((kind([5, 6]), kind([2 ** 31 - 1, 0])), [kind(r) for r in rows], width, torch.device("cpu"))
    want = [5, 6, 2 ** 31 - 1, 0] + [t for r in rows for t in (r[-width:] + [-1] * width)[:width]]
    assert got.dtype == torch.int32 and got.tolist() == want


@pytest.mark.parametrize("kind", [deque, iter, torch.tensor, lambda r: [float(t) for t in r], lambda r: range(r[0], r[0] + len(r))])
@pytest.mark.parametrize("n", [3, 64, 65, 200])
def test_whatever_a_list_can_be_made_of_is_a_row(kind, n):
    row = list(range(7, 7 + n))
    got = _int32_rows((kind([5, 6]),), [kind(row), row], 64, torch.device("cpu"))
    one = (row[-64:] + [-1] * 64)[:64]
    assert got.dtype == torch.int32 and got.tolist() == [5, 6] + one + one


@pytest.mark.parametrize("many", [2 ** 31, -2 ** 31 - 1])
def test_numbers_beyond_32_bits_are_refused_as_a_tensor_refuses_them(many):
    with pytest.raises(RuntimeError):
        _int32_rows(([many], [0]), [], 64, torch.device("cpu"))


def test_the_sampler_takes_iterators_and_deques_and_refuses_no_rows(monkeypatch):
    from dlgo_b200.sampling import sampler as S
    seen = []
    monkeypatch.setattr(S, "draw_on_device", lambda logits, cfg, req, draws, rec, seed: seen.append((req, draws, rec)))
    logits, cfg = torch.zeros(2, 300), SamplerConfig()
    rows = [list(range(100)), [3, 4]]
    for how in (lambda r: r, deque, iter):
        DeviceSampler().sample(logits, cfg, how([8, 9]), how([1, 2]), how([how(r) for r in rows]))
        req, draws, rec = seen.pop()
        assert req.tolist() == [8, 9] and draws.tolist() == [1, 2]
        assert rec.tolist() == [rows[0][-64:], rows[1] + [-1] * 62]
    with pytest.raises(IndexError):
        DeviceSampler().sample(logits, cfg, [8, 9], [1, 2], [])
    with pytest.raises(ValueError):
        DeviceSampler().sample(logits, cfg, [8, 9], [1], rows)


def test_numbers_that_are_read_natively():
    """Lists of whole numbers of 32 bits are, edges and all; anything else is left to the general way, untouched."""
    from dlgo_b200.csrc import kernels as K
    low, high = -2 ** 31, 2 ** 31 - 1
    assert K.pack_rows([[1, True], [low]], [[], [high], list(range(7))], 3).tolist() == [1, 1, low, -1, -1, -1, high, -1, -1, 4, 5, 6]
    assert K.pack_rows([[np.int64(5)]], [], 3).tolist() == [5] and K.pack_rows([[]], [], 3).tolist() == []
    for odd in ([[1.0]], [[high + 1]], [[low - 1]], [["1"]], [[None]], [(1, 2)]):
        assert K.pack_rows(odd, [], 3) is None and K.pack_rows([[1]], odd, 3) is None
    row = iter([1, 2])
    assert K.pack_rows([[1]], [row], 3) is None and list(row) == [1, 2]


@pytest.mark.parametrize("error", ["build", "load"])
def test_lists_are_flattened_where_the_native_reader_cannot_be_had(monkeypatch, tmp_path, error):
    from dlgo_b200.csrc import build, kernels as K
    calls = []

    def ensure_built(names, verbose=True):
        calls.append(names)
        if error == "build":
            raise build.KernelBuildError("no compiler")
        return {n: str(tmp_path / n) for n in names}

    monkeypatch.setattr(K, "_pack_rows", None)
    monkeypatch.setattr(build, "ensure_built", ensure_built)
    for _ in range(2):
        got = _int32_rows(([5, 6], [7, 8]), [[1, 2], [3, 4, 5, 6]], 3, torch.device("cpu"))
        assert got.tolist() == [5, 6, 7, 8, 1, 2, -1, 4, 5, 6]
    assert len(calls) == 1          # (asked for once, not for every draw)


def test_a_list_of_another_class_is_read_as_it_iterates():
    class Newest(list):
        def __iter__(self):
            return reversed(self)

    got = _int32_rows(([1], [2]), [[3, 4], Newest([5, 6])], 3, torch.device("cpu"))
    assert got.tolist() == [1, 2, 3, 4, -1, 6, 5, -1]
