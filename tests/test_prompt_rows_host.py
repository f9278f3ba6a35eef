"""Which models take prompt passes of more than 64 rows, decided from the graph and the configuration alone."""
from types import SimpleNamespace

import pytest
import torch

from cacheir_b200 import ModelConfig, build_decoder_artifact
from cacheir_b200.runtime import _Engine


def _engine(edit=lambda graph: None, **changes):
    config = dict(architecture="LlamaForCausalLM", hidden_size=512, intermediate_size=768, num_layers=2, num_attention_heads=4, num_key_value_heads=2,
                  vocab_size=640, max_position_embeddings=512, rope_theta=10000.0, dtype="float16")
    artifact = build_decoder_artifact(ModelConfig(**{**config, **changes}), quant="int8", modes=("decode",))
    edit(artifact.graph("decode"))
    engine = SimpleNamespace(graph=artifact.graph("decode"), config=artifact.config, dtype=torch.float16, quant="int8", page_size=16,
                             tp=SimpleNamespace(enabled=False))
    engine.weight_rows = lambda name: _Engine.weight_rows(engine, name)
    engine._operands_recent = lambda nodes: _Engine._operands_recent(engine, nodes)
    return engine


def test_models_that_take_them():
    assert _Engine._prompt_rows(_engine(), "same") == 2048
    assert _Engine._prompt_rows(_engine(vocab_size=400000), "same") == 256
    assert _Engine._prompt_rows(_engine(), "int8") == 0
    assert _Engine._prompt_rows(_engine(hidden_size=576, num_attention_heads=9, num_key_value_heads=3), "same") == 0


def _nodes(graph, op):
    return [node for node in graph.nodes if node.op == op]


def _late_residual(graph):      # the embedding joins again behind the last layer: the plan's buffer of it has been taken since
    add = _nodes(graph, "add")[-1]
    add.inputs[0] = "hidden_0"


def _late_gate(graph):          # the second layer's down projection reads the first layer's gated values
    _nodes(graph, "quantized_matmul")[3].inputs[0] = _nodes(graph, "quantized_fused_swiglu")[0].outputs[0]


@pytest.mark.parametrize("edit", [_late_residual, _late_gate])
def test_graphs_that_read_an_older_value_than_the_plan_keeps(edit):
    """Prompt plans share a few buffers between all layers; graphs that reach further back keep passes of 64 rows, whose plan holds all values."""
    assert _Engine._prompt_rows(_engine(edit), "same") == 0


def test_widths_that_meet():
    """A gated width, or the vocabulary, of the residual's width."""
    assert _Engine._prompt_rows(_engine(intermediate_size=512), "same") == 2048
    assert _Engine._prompt_rows(_engine(vocab_size=512), "same") == 2048
    assert _Engine._prompt_rows(_engine(vocab_size=768, intermediate_size=768), "same") == 2048


def _wider_values(graph):       # value heads of another width than the key heads
    graph.weights[_nodes(graph, "quantized_fused_rmsnorm_qkv_rope")[1].inputs[4]].shape = (512, 512)


def _other_keys(graph):         # an attention over another layer's keys: its own are not appended by any projection
    first, second = _nodes(graph, "paged_attention_decode")
    second.inputs[1] = first.inputs[1]


def _other_heads(graph):
    _nodes(graph, "paged_attention_decode")[0].attrs["num_heads"] = 8


def _second_reader(graph):      # two attentions over one projection: only one of them has its keys appended
    first, second = _nodes(graph, "paged_attention_decode")
    second.inputs[:] = first.inputs


@pytest.mark.parametrize("edit", [_wider_values, _other_keys, _other_heads, _second_reader])
def test_graphs_whose_attention_a_prompt_pass_cannot_serve(edit):
    """They keep passes of 64 rows, whose plan appends and attends separately."""
    assert _Engine._prompt_rows(_engine(edit), "same") == 0
