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
    return engine


def test_models_that_take_them():
    assert _Engine._prompt_rows(_engine(), "same") == 2048
    assert _Engine._prompt_rows(_engine(vocab_size=400000), "same") == 256
    assert _Engine._prompt_rows(_engine(), "int8") == 0
    assert _Engine._prompt_rows(_engine(hidden_size=576, num_attention_heads=9, num_key_value_heads=3), "same") == 0


def _nodes(graph, op):
    return [node for node in graph.nodes if node.op == op]


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
