"""Layers that are alike: one goes through Python, the others' calls are made again from what it did."""
import pytest
import torch

pytestmark = pytest.mark.gpu

CONFIG = {"model_type": "qwen3", "architectures": ["Qwen3ForCausalLM"], "num_hidden_layers": 5, "hidden_size": 256,
          "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 64, "intermediate_size": 512, "vocab_size": 300,
          "rope_theta": 10000.0, "rms_norm_eps": 1e-6, "tie_word_embeddings": True, "max_position_embeddings": 4096,
          "eos_token_id": None}


def _engine(dtype, config=CONFIG, **kw):
    from llm_infer_rust_b200 import Engine
    return Engine(None, random_weights_config=config, random_weights_seed=3, dtype=dtype, max_running_req=24, max_seq_len=600,
                  max_total_tokens=4000, cuda_graph_bs=0, log_level="warn", **kw)


def _steps(engine):
    """Prompts in portions, prompts beside decoding rows, many decoding rows, few: the logits of every step."""
    from llm_infer_rust_b200 import StepEntry
    gen = torch.Generator().manual_seed(1)
    ids = lambda n: torch.randint(0, 300, (n,), generator=gen).tolist()
    out = []
    for r in range(20):
        engine.open_request(r + 1)
    out.append(engine.step([StepEntry(1, ids(300), [0, 150, 299])]).clone())
    out.append(engine.step([StepEntry(1, ids(90), [89]), StepEntry(2, ids(17), [16])]).clone())
    out.append(engine.step([StepEntry(r + 1, ids(20 + r), [5]) for r in range(2, 20)]).clone())
    out.append(engine.step([StepEntry(r + 1, ids(1), [0]) for r in range(20)]).clone())
    out.append(engine.step([StepEntry(3, ids(40), [39])] + [StepEntry(r + 1, ids(1), [0]) for r in range(4, 20)]).clone())
    out.append(engine.step([StepEntry(1, ids(1), [0]), StepEntry(2, ids(2), [1])]).clone())
    for r in range(20):
        engine.close_request(r + 1)
    return out


@pytest.mark.parametrize("dtype", ["bfloat16", "float32"])
def test_repeated_layers_give_the_same_bits(dtype):
    from llm_infer_rust_b200.kernels import ops
    engine = _engine(dtype)
    again = []
    inner = ops.LayerCalls.again
    ops.LayerCalls.again = lambda self, values: again.append(inner(self, values)) or again[-1]
    try:
        before = ops.launch_count()
        got = _steps(engine)
        launches = ops.launch_count() - before
        assert all(again) and len(again) >= 3 * 4               # layers 2 to 4 of the steps of many tokens
        engine.model.repeats_layers, n = False, len(again)
        before = ops.launch_count()
        want = _steps(engine)
        assert len(again) == n and ops.launch_count() - before == launches
    finally:
        ops.LayerCalls.again = inner
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    engine.check_kernel_errors()


def test_a_layer_whose_weights_are_of_another_kind_goes_through_python():
    """A norm's weight kept in float32: the calls of the layers before would read it as bfloat16."""
    engine = _engine("bfloat16")
    want = _steps(engine)
    norm = engine.model.blocks[3].input_norm
    kept = norm.params["weight"]
    norm.params["weight"] = kept.float()
    got = _steps(engine)
    engine.model.repeats_layers = False
    plain = _steps(engine)
    assert all(torch.equal(a, b) for a, b in zip(got, plain)) and all(torch.equal(a, b) for a, b in zip(got, want))


def test_a_layer_that_was_changed_goes_through_python():
    """A wrapper round one layer sees every step of many tokens, a scale and a window set on another layer's attention count."""
    engine = _engine("bfloat16")
    seen, block = [], engine.model.blocks[3]
    inner = block.forward
    block.forward = lambda h, residual, ctx, cache: seen.append(h.shape[0]) or inner(h, residual, ctx, cache)
    before = _steps(engine)
    assert seen == [300, 107, sum(range(22, 40)), 20, 56, 3]
    engine.model.blocks[2].mixer.scale *= 2.0
    engine.model.blocks[4].mixer.window = 50
    got = _steps(engine)
    engine.model.repeats_layers = False
    want = _steps(engine)
    assert all(torch.equal(a, b) for a, b in zip(got, want)) and not any(torch.equal(a, b) for a, b in zip(got, before))


def test_repeated_layers_inside_a_captured_prompt():
    """A shape that comes a second time is captured: what is kept are launches, and the graph gives what the step gave."""
    from llm_infer_rust_b200 import StepEntry
    engine = _engine("bfloat16", prefill_cuda_graph_max_tokens=512)
    gen = torch.Generator().manual_seed(1)
    prompt = torch.randint(0, 300, (200,), generator=gen).tolist()
    out = []
    for _ in range(4):
        engine.open_request(1)
        out.append(engine.step([StepEntry(1, prompt, [199])]).clone())
        engine.close_request(1)
    assert len(engine._shape_graphs) == 1 and all(torch.equal(o, out[0]) for o in out)


def test_kept_layers_hold_little():
    """The peak of a step of many tokens is what it is without kept calls."""
    from llm_infer_rust_b200 import StepEntry
    config = dict(CONFIG, num_attention_heads=16, num_key_value_heads=8, head_dim=128)
    engine = _engine("bfloat16", config)
    peaks = []
    for engine.model.repeats_layers in (False, True):
        for r in range(1, 6):
            engine.open_request(r)
        torch.cuda.synchronize()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        engine.step([StepEntry(r, list(range(2, 290)) * 2, [575]) for r in range(1, 6)])
        peaks.append(torch.cuda.max_memory_allocated() - before)
        for r in range(1, 6):
            engine.close_request(r)
    assert peaks[1] <= peaks[0] + (1 << 20)
