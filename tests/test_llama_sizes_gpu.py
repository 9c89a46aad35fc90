"""The engine at the layer sizes of Llama 3.2 1B (hidden 2048, 32/8 heads of 64, feed-forward 8192,
vocabulary 128256, llama3 rope scaling factor 32, tied head) with FOUR layers instead of sixteen so
that the plain implementation stays within a minute on the CPU.  These sizes take the kernels the
tiny models never reach: the tensor-core prompt attention (head size 64), 128 x 256 GEMM tiles over
many tiles, K-slices, a vocabulary that is no multiple of any tile.  The same at the layer sizes of
Llama 3.2 3B and Llama 3.1 8B (heads of 128, three and four query heads per kv head, an untied head).
Needs a GPU."""
import pytest
import torch

import plain_llama as P
import traces as T

pytestmark = pytest.mark.gpu

CFG = dict(architectures=["LlamaForCausalLM"], hidden_size=2048, num_hidden_layers=4, intermediate_size=8192,
           num_attention_heads=32, num_key_value_heads=8, head_dim=64, vocab_size=128256, rope_theta=500000.0,
           rope_scaling=dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0,
                             original_max_position_embeddings=8192),
           rms_norm_eps=1e-5, max_position_embeddings=131072, tie_word_embeddings=True)
# Llama 3.1 8B layer sizes (hidden 4096, 32/8 heads of 128, feed-forward 14336, untied head, rope factor 8),
# two layers and a 32000 vocabulary to keep the plain implementation quick: head size 128 everywhere
CFG_8B = dict(architectures=["LlamaForCausalLM"], hidden_size=4096, num_hidden_layers=2, intermediate_size=14336,
              num_attention_heads=32, num_key_value_heads=8, head_dim=128, vocab_size=32000, rope_theta=500000.0,
              rope_scaling=dict(rope_type="llama3", factor=8.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                original_max_position_embeddings=8192),
              rms_norm_eps=1e-5, max_position_embeddings=131072, tie_word_embeddings=False)
# Llama 3.2 3B layer sizes (hidden 3072, 24/8 heads of 128: three query heads per kv head, feed-forward 8192, tied),
# two layers and a 32000 vocabulary
CFG_3B = dict(architectures=["LlamaForCausalLM"], hidden_size=3072, num_hidden_layers=2, intermediate_size=8192,
              num_attention_heads=24, num_key_value_heads=8, head_dim=128, vocab_size=32000, rope_theta=500000.0,
              rope_scaling=dict(rope_type="llama3", factor=32.0, low_freq_factor=1.0, high_freq_factor=4.0,
                                original_max_position_embeddings=8192),
              rms_norm_eps=1e-5, max_position_embeddings=131072, tie_word_embeddings=True)
ROWS = [0, 1, 63, 64, 127, 128, 141] + list(range(142, 150))       # places compared (the last 8 are decoded)


def build(tmp_path_factory, CFG, seed):
    from dlgo_b200.config import config_from_dict
    from dlgo_b200.weights import write_random_model
    d = str(tmp_path_factory.mktemp("llama_sizes"))
    write_random_model(config_from_dict(CFG), seed, d, device="cuda")
    g = torch.Generator().manual_seed(3)
    reqs = {"long": torch.randint(0, CFG["vocab_size"], (150,), generator=g).tolist(),
            "short": torch.randint(0, CFG["vocab_size"], (21,), generator=g).tolist()}
    cfg, w = P.read_model(d)
    freqs = P.rope_frequencies(cfg["head_dim"], cfg["rope_theta"], cfg["rope_scaling"])
    refs = {}
    for rid, toks in reqs.items():
        x = P.embedding(w["model.embed_tokens.weight"], toks)
        for i in range(cfg["num_hidden_layers"]):
            x = P.layer(x, w, f"model.layers.{i}.", cfg, freqs)
        rows = [r for r in ROWS if r < len(toks)] if rid == "long" else list(range(len(toks)))
        xn = P.rmsnorm(x[rows], w["model.norm.weight"], cfg["rms_norm_eps"])
        head = w["model.embed_tokens.weight"] if cfg["tie_word_embeddings"] else w["lm_head.weight"]
        refs[rid] = (rows, P.linear(xn, head))
    del w
    return d, reqs, refs


@pytest.fixture(scope="module")
def big(tmp_path_factory):
    return build(tmp_path_factory, CFG, 2)


@pytest.fixture(scope="module")
def big8(tmp_path_factory):
    return build(tmp_path_factory, CFG_8B, 5)


@pytest.fixture(scope="module")
def big3(tmp_path_factory):
    return build(tmp_path_factory, CFG_3B, 4)


def run(engine, reqs, refs, dtype, what):
    long_rows = refs["long"][0]
    n = len(reqs["long"])
    # whole: both requests in one step; then the long one again with its last 8 tokens one by one
    steps = [{"step": 0, "entries": [{"id": "long", "tokens": reqs["long"], "want": long_rows},
                                      {"id": "short", "tokens": reqs["short"], "want": list(range(len(reqs["short"])))}],
              "end": ["long", "short"]},
             {"step": 1, "entries": [{"id": "l2", "tokens": reqs["long"][:n - 8], "want": [r for r in long_rows if r < n - 8]}],
              "end": []}]
    for j in range(n - 8, n):
        steps.append({"step": len(steps), "entries": [{"id": "l2", "tokens": [reqs["long"][j]], "want": [0]}],
                      "end": ["l2"] if j == n - 1 else []})
    outs = T.run_in_process(engine, steps)
    tol = 1e-4 if dtype == "float32" else 3e-2
    ref_long, ref_short = refs["long"][1], refs["short"][1]
    scale = float(ref_long.abs().max())

    def close(got, ref, name):
        assert torch.isfinite(got).all(), name
        err = float((got - ref).abs().max())
        assert err <= tol * scale, f"{what} {name} ({dtype}): max abs diff {err:.3e} > {tol * scale:.3e}"

    close(outs[0][:len(long_rows)], ref_long, "whole, long")
    close(outs[0][len(long_rows):], ref_short, "whole, short beside it")
    k = len([r for r in long_rows if r < n - 8])
    close(outs[1], ref_long[:k], "prefix")
    tail = torch.cat([outs[s] for s in range(2, 10)])
    close(tail, ref_long[k:], "last 8 one by one")
    # the long request once more, fed in three pieces (several tokens on top of a cache that is not empty)
    cuts = [(0, 60), (60, 130), (130, n)]
    steps = [{"step": i, "entries": [{"id": "l3", "tokens": reqs["long"][a:b],
                                      "want": [r - a for r in long_rows if a <= r < b]}],
              "end": ["l3"] if b == n else []} for i, (a, b) in enumerate(cuts)]
    outs = T.run_in_process(engine, steps)
    close(torch.cat([outs[i] for i in range(3) if i in outs]), ref_long, "in three pieces")
    from dlgo_b200.csrc import kernels
    kernels.check_device_errors()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_llama_1b_sizes_against_the_plain_implementation(big, dtype):
    from dlgo_b200.engine.engine import Engine
    d, reqs, refs = big
    eng = Engine(d, dtype=dtype, max_tokens=512, max_seq_len=256)
    eng.cache.poison()
    run(eng, reqs, refs, dtype, "graphs")
    if dtype == "bfloat16":
        eng2 = Engine(d, dtype=dtype, max_tokens=512, max_seq_len=256, cuda_graphs=False)
        eng2.cache.poison()
        run(eng2, reqs, refs, dtype, "no graphs")


def test_prompt_steps_run_through_the_native_layer_loop_and_match_the_parts(big, monkeypatch):
    """A bfloat16 prompt step of more than 64 tokens hands its run of like layers to one native call, which
    launches what the parts launch one by one, with the same arguments: with the epilogue that adds a tile into
    the residual in one piece (no K-slices, whose order is not fixed) the logits are the same bit for bit.  A
    prompt on top of a cache that is not empty goes the same way."""
    from dlgo_b200.csrc import kernels
    from dlgo_b200.engine import prompt_run
    from dlgo_b200.engine.engine import Engine
    d, reqs, refs = big
    g = torch.Generator().manual_seed(11)
    prompts = [torch.randint(0, CFG["vocab_size"], (n,), generator=g).tolist() for n in (300, 77, 129)]
    more = [torch.randint(0, CFG["vocab_size"], (n,), generator=g).tolist() for n in (90, 70, 101)]
    calls = []
    real = kernels.prompt_layers
    monkeypatch.setattr(kernels, "prompt_layers", lambda e, sh, layers, step: (calls.append((len(layers), step.tokens)),
                                                                                 real(e, sh, layers, step))[1])

    def logits(eng):
        slots = [eng.take_slot() for _ in prompts]
        a = eng.step(slots, prompts, [[len(p) - 1, 0, len(p) // 2] for p in prompts]).float().cpu()
        b = eng.step(slots, more, [[len(p) - 1] for p in more]).float().cpu()
        for s in slots:
            eng.free_slot(s)
        return torch.cat([a, b])

    eng = Engine(d, dtype="bfloat16", max_tokens=2048, max_seq_len=512)
    runs = eng.model.prompt_runs
    assert len(runs) == 1 and runs[0].n == CFG["num_hidden_layers"]
    for direct in ("1", None):
        if direct:
            monkeypatch.setenv("DLGO_TC_DIRECT_EPILOGUE", direct)     # read at every call
        else:
            monkeypatch.delenv("DLGO_TC_DIRECT_EPILOGUE")
        del calls[:]
        monkeypatch.setattr(eng.model, "prompt_runs", runs)
        got = logits(eng)
        assert calls == [(CFG["num_hidden_layers"], 506), (CFG["num_hidden_layers"], 261)]
        monkeypatch.setattr(eng.model, "prompt_runs", {})
        want = logits(eng)
        assert len(calls) == 2
        if direct:
            assert torch.equal(got, want)
        else:
            # K-slices add themselves into the residual in no fixed order: bfloat16 rounding apart
            assert float((got - want).abs().max()) <= 3e-2 * float(want.abs().max())
    kernels.check_device_errors()
    # float32 has no native loop: the parts run
    eng32 = Engine(d, dtype="float32", max_tokens=512, max_seq_len=256)
    assert eng32.model.prompt_runs == {} and prompt_run.ENABLED


@pytest.mark.parametrize("lens", [[2], [5, 9], [17], [30, 3, 31], [65], [50, 27], [128]])
def test_short_prompt_steps_through_the_native_layer_loop_match_the_parts(big, lens, monkeypatch):
    """Up to 64 tokens, up to 128: other products than longer prompts (the weight is the tensor core's M operand and its
    K-slices meet in fp32), onto an empty cache and onto one that is not."""
    from dlgo_b200.csrc import kernels
    from dlgo_b200.engine.engine import Engine
    d, _, _ = big
    g = torch.Generator().manual_seed(sum(lens))
    prompts, more = ([torch.randint(0, CFG["vocab_size"], (n,), generator=g).tolist() for n in lens] for _ in range(2))
    calls = []
    real = kernels.prompt_layers
    monkeypatch.setattr(kernels, "prompt_layers", lambda e, sh, layers, step: (calls.append(step.tokens),
                                                                                 real(e, sh, layers, step))[1])

    def logits(eng):
        slots = [eng.take_slot() for _ in prompts]
        out = [eng.step(slots, p, [[len(q) - 1, 0] for q in p]).float().cpu() for p in (prompts, more)]
        for s in slots:
            eng.free_slot(s)
        return torch.cat(out)

    eng = Engine(d, dtype="bfloat16", max_tokens=1024, max_seq_len=512)
    got = logits(eng)
    assert calls == [sum(lens)] * 2
    monkeypatch.setattr(eng.model, "prompt_runs", {})
    want = logits(eng)
    assert len(calls) == 2
    assert float((got - want).abs().max()) <= 3e-2 * float(want.abs().max())     # (sums in no fixed order: bfloat16 rounding)
    kernels.check_device_errors()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_llama_8b_layer_sizes_against_the_plain_implementation(big8, dtype):
    from dlgo_b200.engine.engine import Engine
    d, reqs, refs = big8
    eng = Engine(d, dtype=dtype, max_tokens=512, max_seq_len=256)
    eng.cache.poison()
    run(eng, reqs, refs, dtype, "8B sizes")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_llama_3b_layer_sizes_against_the_plain_implementation(big3, dtype):
    from dlgo_b200.engine.engine import Engine
    d, reqs, refs = big3
    eng = Engine(d, dtype=dtype, max_tokens=512, max_seq_len=256)
    eng.cache.poison()
    run(eng, reqs, refs, dtype, "3B sizes")


# ---------------------------------------------------------------------------------------------------
# The schedule that decoding at real sizes takes: several sequences of unequal lengths, some longer than
# 512 tokens (so that decode attention works in slices), prompts in one step and then one token each
# through the captured graph; contractions cut into K-slices that add themselves into the residual, the
# q/k/v sum that the rotation reads and clears.  Two layers keep the plain implementation quick.
CFG_2L = dict(CFG, num_hidden_layers=2)
BATCH_LENS = [530, 37, 700, 8, 129, 612, 64, 250]     # prompt lengths; 8 more tokens are decoded
N_DECODE = 8


@pytest.fixture(scope="module")
def batch8(tmp_path_factory):
    from dlgo_b200.config import config_from_dict
    from dlgo_b200.weights import write_random_model
    d = str(tmp_path_factory.mktemp("llama_batch8"))
    write_random_model(config_from_dict(CFG_2L), 2, d, device="cuda")
    g = torch.Generator().manual_seed(11)
    reqs = {f"r{i}": torch.randint(0, CFG_2L["vocab_size"], (n + N_DECODE,), generator=g).tolist()
            for i, n in enumerate(BATCH_LENS)}
    cfg, w = P.read_model(d)
    freqs = P.rope_frequencies(cfg["head_dim"], cfg["rope_theta"], cfg["rope_scaling"])
    refs = {}
    for (rid, toks), n in zip(reqs.items(), BATCH_LENS):
        x = P.embedding(w["model.embed_tokens.weight"], toks)
        for i in range(cfg["num_hidden_layers"]):
            x = P.layer(x, w, f"model.layers.{i}.", cfg, freqs)
        xn = P.rmsnorm(x[n - 1:], w["model.norm.weight"], cfg["rms_norm_eps"])
        refs[rid] = P.linear(xn, w["model.embed_tokens.weight"])       # rows n-1 .. n+7: the prompt's end, 8 decoded
    del w
    return d, reqs, refs


def batch_steps(reqs):
    ids = list(reqs)
    steps = [{"step": 0, "entries": [{"id": r, "tokens": reqs[r][:n], "want": [n - 1]} for r, n in zip(ids, BATCH_LENS)],
              "end": []}]
    for j in range(N_DECODE):
        steps.append({"step": j + 1, "entries": [{"id": r, "tokens": [reqs[r][n + j]], "want": [0]}
                                                  for r, n in zip(ids, BATCH_LENS)],
                      "end": ids if j == N_DECODE - 1 else []})
    return steps


@pytest.fixture
def persistent_decode(monkeypatch):
    """Engines built inside the test run their decode steps' layers as one persistent kernel."""
    from dlgo_b200.engine import fused_decode
    monkeypatch.setattr(fused_decode, "ENABLED", True)


def test_the_persistent_decode_kernel_against_the_plain_implementation(batch8, persistent_decode):
    test_a_batch_of_eight_unequal_sequences_decodes_through_the_graph(batch8, "bfloat16", fused=True)


def test_the_persistent_decode_kernel_at_8b_and_3b_layer_sizes(big8, big3, persistent_decode):
    from dlgo_b200.engine.engine import Engine
    for d, reqs, refs in (big8, big3):
        eng = Engine(d, dtype="bfloat16", max_tokens=512, max_seq_len=256)
        assert eng.model.fused_runs
        eng.cache.poison()
        run(eng, reqs, refs, "bfloat16", "persistent kernel")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_batch_of_eight_unequal_sequences_decodes_through_the_graph(batch8, dtype, fused=False):
    from dlgo_b200.csrc import kernels
    from dlgo_b200.engine.engine import Engine
    d, reqs, refs = batch8
    eng = Engine(d, dtype=dtype, max_tokens=8 * 1024, max_seq_len=1024)      # grids sized for 16 pages a sequence
    eng.cache.poison()
    outs = T.run_in_process(eng, batch_steps(reqs))
    assert (8, 1024) in eng._graphs, "the decode steps should have replayed the graph of batch 8"
    assert bool(eng.model.fused_runs) == fused
    if fused:
        # both layers as one persistent kernel: embedding, that kernel, final norm, head
        assert eng._graphs[(8, 1024)].kernels_per_replay <= 6, eng._graphs[(8, 1024)].kernels_per_replay
    tol = 1e-4 if dtype == "float32" else 3e-2
    for i, rid in enumerate(reqs):
        ref = refs[rid]
        scale = float(ref.abs().max())
        for s in range(N_DECODE + 1):
            got = outs[s][i]
            assert torch.isfinite(got).all(), (rid, s)
            err = float((got - ref[s]).abs().max())
            assert err <= tol * scale, f"{rid} ({BATCH_LENS[i]} tokens), step {s} ({dtype}): {err:.3e} > {tol * scale:.3e}"
    kernels.check_device_errors()


def test_ordered_sums_make_bfloat16_decoding_repeatable_bit_for_bit(batch8, monkeypatch):
    # DLGO_ORDERED_SUMS=1: K-slices are kept apart and added in slice order by the next norm instead of adding
    # themselves into the residual in whatever order they finish.  Two runs of the same batch then give the
    # same bits (another batch size cuts K into other slices: close, not bit-equal).
    from dlgo_b200.engine.engine import Engine
    from dlgo_b200.parts import tensor_core
    monkeypatch.setattr(tensor_core, "ORDERED_SUMS", True)
    d, reqs, refs = batch8
    eng = Engine(d, dtype="bfloat16", max_tokens=8 * 1024, max_seq_len=1024)
    first = T.run_in_process(eng, batch_steps(reqs))
    again = T.run_in_process(eng, batch_steps(reqs))
    for s in range(N_DECODE + 1):
        assert torch.equal(first[s], again[s]), f"step {s}: two runs differ"
    for i, rid in enumerate(reqs):
        scale = float(refs[rid].abs().max())
        for s in range(N_DECODE + 1):
            assert float((first[s][i] - refs[rid][s]).abs().max()) <= 3e-2 * scale, (rid, s)
    # request r2 alone (batch 1: other K-slicing, other graph) decodes to the same bits as inside the batch of 8
    rid, n = "r2", BATCH_LENS[2]
    slot = eng.take_slot()
    eng.step([slot], [reqs[rid][:n]])
    for j in range(N_DECODE):
        lg = eng.step([slot], [[reqs[rid][n + j]]]).float().cpu()
        err = float((lg[0] - first[j + 1][2]).abs().max())
        assert err <= 3e-2 * float(refs[rid].abs().max())      # (other slice counts: close, not bit-equal)
    eng.free_slot(slot)


def test_default_cache_sizing_and_a_very_long_capacity(batch8):
    # no max_tokens: the cache is sized from the context (131072 positions here).  Captured steps are sized for
    # the reach they are asked for: these short sequences replay the graph for 4,096 positions; the same step
    # through the graph for the whole context (2048 pages a sequence: decode attention takes even shares of all
    # keys instead of slices) gives the same logits
    from dlgo_b200.engine import graphs
    from dlgo_b200.engine.engine import Engine
    d, reqs, refs = batch8
    eng = Engine(d, dtype="bfloat16")
    assert eng.max_seq_len == 131072 and eng.cache.n_pages >= 2048
    ids = list(reqs)[:3]
    lens = BATCH_LENS[:3]
    slots = [eng.take_slot() for _ in ids]
    lg = [eng.step(slots, [reqs[r][:n] for r, n in zip(ids, lens)]).float().cpu()]
    for j in range(3):
        lg.append(eng.step(slots, [[reqs[r][n + j]] for r, n in zip(ids, lens)]).float().cpu().clone())
    assert list(eng._graphs) == [(3, 4096)]
    # the last of these steps once more, through the graph that reaches the whole context (it writes the same
    # keys and values to the same places)
    far = graphs.decode_with_graph(eng, slots, [reqs[r][n + 2] for r, n in zip(ids, lens)], [n + 2 for n in lens],
                                   reach=eng.max_seq_len).float().cpu()
    assert list(eng._graphs) == [(3, 4096), (3, 131072)]
    for s in slots:
        eng.free_slot(s)
    for i, rid in enumerate(ids):
        scale = float(refs[rid].abs().max())
        for s in range(4):
            assert float((lg[s][i] - refs[rid][s]).abs().max()) <= 3e-2 * scale, (rid, s)
        assert float((far[i] - refs[rid][3]).abs().max()) <= 3e-2 * scale, rid
    # this engine's cache took half of the device's free memory: hand it back now, so that later tests do not
    # find the allocator releasing cached blocks in the middle of a graph capture
    del eng
    import gc
    gc.collect()
    torch.cuda.empty_cache()


def test_native_runs_at_real_sizes_agree_with_single_steps(batch8):
    # greedy and sampled runs of several steps in one native call (what generate() uses) against the same
    # engine stepped one by one.  In bfloat16 the K-slices add themselves into the residual in no fixed
    # order, so two runs may differ in the last bits: a different token is accepted only where the two
    # candidates' logits are nearly tied.
    from dlgo_b200.csrc import kernels
    from dlgo_b200.engine.engine import Engine
    d, reqs, _ = batch8
    eng = Engine(d, dtype="bfloat16", max_tokens=8 * 1024, max_seq_len=1024)
    ids = list(reqs)
    prompts = [reqs[r][:n] for r, n in zip(ids, BATCH_LENS)]

    def start():
        slots = [eng.take_slot() for _ in ids]
        first = kernels.argmax(eng.step(slots, prompts)).cpu().tolist()
        return slots, first

    slots, first = start()
    run = eng.greedy_run(slots, first, 6)
    assert run is not None and len(run) == 6
    for s in slots:
        eng.free_slot(s)
    slots, again = start()
    assert again == first
    feed = list(first)
    alive = [True] * len(ids)
    for step in range(6):
        lg = eng.step(slots, [[t] for t in feed]).float().cpu()
        for i in range(len(ids)):
            if not alive[i]:
                continue
            got, want = run[step][i], int(lg[i].argmax())
            if got != want:
                gap = float(lg[i, want] - lg[i, got])
                assert gap <= 2e-2 * float(lg[i].abs().max()), (ids[i], step, got, want, gap)
                alive[i] = False            # from here on the two runs see different tokens
        feed = [run[step][i] if alive[i] else int(lg[i].argmax()) for i in range(len(ids))]
        if not all(alive):
            break
    for s in slots:
        eng.free_slot(s)
    assert sum(alive) >= 6, "most sequences should choose the same tokens in both runs"
    kernels.check_device_errors()


def test_sampled_generation_at_real_sizes(batch8):
    # generate() with a temperature through the Python entry point: the same requests alone and in a batch
    # draw the same tokens (a draw depends on seed, request and draw index only), up to the rare draw that
    # falls on a boundary moved by the last bits of the logits
    import dlgo_b200
    d, reqs, _ = batch8
    llm = dlgo_b200.load_llm(d, dtype="bfloat16", max_tokens=8 * 1024, max_seq_len=1024, max_batch=8)
    prompts = [reqs[r][:n] for r, n in zip(reqs, BATCH_LENS)]
    # (random weights give nearly flat distributions over 128,256 tokens, where the last bit of a logit
    # moves the draw; a low temperature makes the draw depend on the logits' leading digits)
    opts = dict(max_tokens=6, temperature=0.02, top_k=0, top_p=1.0, repetition_penalty=1.0, seed=5, ignore_eos=True)
    together = llm.generate(prompts, **opts)
    assert all(len(t) == 6 for t in together)
    # request i keeps its index in a smaller batch (requests 0..i): the batch size and its graph differ
    same = 0
    for i in (0, 2, 5):
        smaller = llm.generate(prompts[:i + 1], **opts)[i]
        same += smaller == together[i]
    assert same >= 2, (together,)
