"""Which layers' calls may be made again with another layer's memory (parts/block.py, parts/model.py), decided without a GPU."""
from types import SimpleNamespace

import pytest
import torch

from llm_infer_rust_b200.config.spec import PartSpec
from llm_infer_rust_b200.kernels import ops
from llm_infer_rust_b200.parts.attention import GQAttention
from llm_infer_rust_b200.parts.base import BuildEnv
from llm_infer_rust_b200.parts.block import PreNormDeferredAdd
from llm_infer_rust_b200.parts.feed_forward import SwiGLU
from llm_infer_rust_b200.parts.norm import RMSNorm

ENV = BuildEnv(torch.float32, torch.device("cpu"), {})
CACHE = SimpleNamespace(k=torch.zeros(3, 2, 16, 32), v=torch.zeros(3, 2, 16, 32))


def _bound(part):
    for name, decl in part.param_decls().items():
        part.bind(name, torch.zeros(decl.shape))
    return part


def _attention(**spec):
    return _bound(GQAttention(PartSpec("gq_attention", dict(dict(hidden_size=64, num_heads=4, num_kv_heads=2, head_dim=32, qk_norm_eps=1e-6), **spec)), ENV))


def _feed_forward():
    return _bound(SwiGLU(PartSpec("swiglu", dict(hidden_size=64, intermediate_size=96)), ENV))


@pytest.mark.parametrize("takes", ["qkv_proj", "o_proj", "gate_up_proj", "down_proj", None])
def test_a_product_on_the_few_row_kernels_is_not_made_again(monkeypatch, takes):
    """Those take their operands' addresses in a block of parameters.  Whichever of a part's products goes there, and also when only
    the plain form of it does, behind a fused form that is refused, the layer goes through Python."""
    mixer, feed = _attention(), _feed_forward()
    on_few = {**mixer.params, **feed.params}.get(takes)
    monkeypatch.setattr(ops, "few_row_takes", lambda rows, weight, dtype, mode=ops.EPI_PLAIN_BF16, head_dim=0, norm=True:
                        weight is on_few and mode == ops.EPI_PLAIN_BF16 and not norm)
    assert (mixer.repeat_slots(9, CACHE) is None) == (takes in ("qkv_proj", "o_proj"))
    assert (feed.repeat_slots(torch.zeros(9, 64)) is None) == (takes in ("gate_up_proj", "down_proj"))


def _block():
    block = PreNormDeferredAdd.__new__(PreNormDeferredAdd)
    block.input_norm, block.post_mixer_norm = (_bound(RMSNorm(PartSpec("rms_norm", dict(width=64, eps=1e-6)), ENV)) for _ in range(2))
    block.mixer, block.feed_forward = _attention(), _feed_forward()
    return block


@pytest.mark.parametrize("where", ["block", "input_norm", "post_mixer_norm", "mixer", "feed_forward"])
def test_a_layer_whose_forward_was_replaced_says_so(where):
    """A wrapper put on one object, as one does to look at what a layer gives: its calls are not made past it."""
    block, h = _block(), torch.zeros(9, 64)
    assert block.repeat_slots(h, CACHE) is not None
    part = block if where == "block" else getattr(block, where)
    name = "forward_add" if where.endswith("norm") else "forward"
    setattr(part, name, getattr(part, name))
    assert block.repeat_slots(h, CACHE) is None


@pytest.mark.parametrize("where,name,value", [("input_norm", "eps", 1e-3), ("post_mixer_norm", "eps", 1e-3), ("mixer", "scale", 0.5),
                                              ("mixer", "window", 5), ("mixer", "qk_eps", 1e-3), ("mixer", "nkv", 1),
                                              ("mixer", "rope", SimpleNamespace())])
def test_a_layer_with_other_numbers_is_not_like_the_others(where, name, value):
    block, other, h = _block(), _block(), torch.zeros(9, 64)
    assert block.repeat_slots(h, CACHE)[0] == other.repeat_slots(h, CACHE)[0]
    setattr(getattr(block, where), name, value)
    assert block.repeat_slots(h, CACHE)[0] != other.repeat_slots(h, CACHE)[0]


def test_a_step_whose_intermediates_are_many_is_not_kept():
    """A kept layer's QKV, q and heads' outputs stay beside what the feed-forward makes: 24 MiB of them at most."""
    mixer, bytes_a_token = _attention(), (3 * 4 + 2 * 2) * 32 * 4
    assert mixer.repeat_slots((24 << 20) // bytes_a_token, CACHE) is not None
    assert mixer.repeat_slots((24 << 20) // bytes_a_token + 1, CACHE) is None
