"""Which form of decode attention a step takes and what it allocates for it (host code: nothing is launched)."""
from types import SimpleNamespace as NS

import pytest
import torch

from dlgo_b200.csrc import kernels as K
from dlgo_b200.parts import attention
from dlgo_b200.parts.attention import GQAAttention


@pytest.fixture
def plan(monkeypatch):
    """``plan(heads, kv_heads, head_dim, sequences, reach, dtype)``: (slices, {what it allocated: how many})."""
    monkeypatch.setattr(attention, "_sm_count", lambda device: 148)
    monkeypatch.setattr(K, "attention_decode_takes", lambda act, hd, page: True)
    monkeypatch.setattr(K, "attention_decode_mma_takes", lambda act, hd, page, n: act == torch.bfloat16 and hd in (64, 128))
    monkeypatch.setattr(K, "attention_decode_shares_scratch", lambda hq, hkv, hd: 7)

    def of(hq, hkv, hd, T, reach, dtype=torch.bfloat16):
        mixer = GQAAttention(64, hq, hkv, hd, 1.0)
        asked = {}
        ctx = NS(n_tokens=T, decode=True, captured=True, capacity=reach, scratch=lambda name, n: asked.setdefault(name, n),
                 zeros=lambda name, n: asked.setdefault(name, n))
        cache = NS(page_size=64, keys=torch.empty(0, dtype=dtype))
        _, _, n_splits, scratch, counters, _ = mixer._decode_plan(ctx, cache, dtype)
        assert (scratch, counters) == tuple(asked.get(n) for n in ("attention", "attention_tickets" if n_splits == 0 else "attention_counters"))
        return n_splits, asked
    return of


@pytest.mark.parametrize("T", [1, 2, 8])
def test_a_step_in_even_shares_allocates_nothing_else(plan, T):
    assert plan(32, 8, 64, T, 16384) == (0, {"attention": 7, "attention_tickets": 8 * T})
    assert plan(20, 1, 128, 2, 16384) == (0, {"attention": 7, "attention_tickets": 2 * 3})


def test_slices_allocate_as_they_did(plan):
    assert plan(32, 8, 64, 4, 4096) == (8, {})
    assert plan(32, 8, 64, 64, 4096) == (1, {})
    assert plan(32, 8, 64, 2, 16384, torch.float32) == (37, {"attention": K.attention_scratch_floats(2, 32, 64, 37), "attention_counters": 16})


@pytest.mark.parametrize("T", [1, 4, 8])
@pytest.mark.parametrize("reach", [40, 64, 128, 190])
def test_few_pages_do_not_make_even_shares(plan, T, reach):
    """Heads of 128: shares where few slices FIT, not where a short sequence has no more pages."""
    assert plan(24, 8, 128, T, reach) == (min(-(-reach // 64), 296 // (8 * T)), {})
    assert plan(24, 8, 128, 10, 4096)[0] == 0 and plan(24, 8, 128, 37, 4096)[0] == 0 and plan(24, 8, 128, 9, 4096)[0] == 4
