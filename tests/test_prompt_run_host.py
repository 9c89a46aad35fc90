"""Which form of each product the native loop of a prompt step is told to run (host code: nothing is launched)."""
import importlib
from types import SimpleNamespace as NS

import pytest
import torch

from dlgo_b200.csrc import kernels as K
from dlgo_b200.parts import attention, tensor_core

D, HQ, HKV, HD, F = 256, 4, 2, 64, 1024
MANY, FEW, STREAM = 0, 1, 2          # forms


@pytest.fixture
def step_of(monkeypatch):
    """``step_of(tokens)``: the step description that a run of one layer hands to the native loop."""
    from dlgo_b200.engine import prompt_run
    monkeypatch.setattr(tensor_core, "sm_count", lambda device=None: 148)
    monkeypatch.setattr(tensor_core, "_workspaces", {})
    monkeypatch.setattr(tensor_core, "_counters", {})
    monkeypatch.setattr(K, "prompt_entry_points", lambda: None)
    seen = []
    monkeypatch.setattr(K, "prompt_layers", lambda entry, shape, layers, step: seen.append(step))
    linear = {n: NS(_tc=tensor_core.TensorCorePlan(torch.empty(rows, cols, dtype=torch.bfloat16), swiglu=n == "w_gate_up"))
              for n, rows, cols in (("wqkv", (HQ + 2 * HKV) * HD, D), ("wo", D, HQ * HD), ("w_gate_up", 2 * F, D), ("w_down", D, F))}
    mixer = NS(wqkv=linear["wqkv"], wo=linear["wo"], fuses_prompt_rope=lambda *a: True)
    model = NS(blocks={0: NS(mixer=mixer, ffn=NS(w_gate_up=linear["w_gate_up"], w_down=linear["w_down"]))}, order=[NS(layer=0)],
               positions={"rope": NS(cos=torch.empty(1), sin=torch.empty(1))})
    view = NS(page_table=torch.empty(1, 4, dtype=torch.int32), page_size=64, keys=torch.empty(1, dtype=torch.bfloat16))
    cache = NS(view=lambda i: view)

    def build(tokens):
        run = prompt_run.PromptRun(0, 1, (D, HQ, HKV, HD, F, 1.0, 0, "rope", HD, False, "full"))
        run._descriptors = lambda *a: (None, None)
        some = torch.empty(1, dtype=torch.int32)
        ctx = NS(decode=False, n_tokens=tokens, tiles=lambda *a, **k: (some, 1, 1), token_pos=some, token_seq=some, seq_slot=some,
                 scratch=lambda name, n, dt: torch.empty(n, dtype=dt), zeros=lambda name, n, dt: torch.zeros(n, dtype=dt))
        monkeypatch.setattr(K, "attention_prefill_tc_takes", lambda *a: True)
        if not run.takes(ctx, cache):
            return None
        run.run(model, torch.empty(tokens, D), ctx, cache)
        return seen.pop()

    return build


def test_streamed_products_end_where_their_kernel_does(step_of, monkeypatch):
    from dlgo_b200.engine import prompt_run
    monkeypatch.setenv("DLGO_PROMPT_STREAM_MAX", "256")
    importlib.reload(prompt_run)
    try:
        assert list(step_of(K.GEMM_TC_STREAM_MAX).form) == [STREAM, STREAM, MANY, STREAM]
        assert list(step_of(K.GEMM_TC_STREAM_MAX + 1).form) == [MANY] * 4
    finally:
        monkeypatch.delenv("DLGO_PROMPT_STREAM_MAX")
        importlib.reload(prompt_run)
    assert list(step_of(64).form) == [FEW] * 4 and list(step_of(65).form) == [STREAM, STREAM, MANY, STREAM]


@pytest.mark.parametrize("tokens", [2, 64, 65, 128, 129])
def test_the_switch_of_the_projections_fp32_sum_holds_for_prompts(step_of, monkeypatch, tokens):
    assert bool(step_of(tokens).qkv_sum) == (tokens <= 128)
    monkeypatch.setattr(attention, "_QKV_SUM", 0)
    step = step_of(tokens)
    if tokens <= 64:
        assert step is None             # part by part
    else:
        assert step.form[0] == MANY and not step.qkv_sum and step.fuse_rope == 1
        assert list(step.form)[1:] == ([STREAM, MANY, STREAM] if tokens <= 128 else [MANY] * 3)
