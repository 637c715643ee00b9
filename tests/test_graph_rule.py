"""Which models and engine settings decode inside CUDA graphs: only those whose attention runs on kernels from end to end."""
import pytest
import torch

from fastllm_b200.engine import EngineConfig, ModelRunner
from fastllm_b200.models import from_hf_dict, random_init


@pytest.mark.parametrize("head_dim,max_batch,safe", [(64, 4, True), (64, 1024, True), (64, 1025, False), (128, 1025, True), (60, 4, False), (256, 4, True), (264, 4, False)])
def test_rule_by_head_width(head_dim, max_batch, safe):
    cfg = from_hf_dict(dict(model_type="llama", vocab_size=512, hidden_size=256, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2,
                            intermediate_size=512, max_position_embeddings=1024, head_dim=head_dim))
    runner = ModelRunner(random_init(cfg, "cpu", torch.bfloat16), EngineConfig(max_batch=max_batch, max_context=256), num_pages=8)
    assert runner._graph_safe() == safe
