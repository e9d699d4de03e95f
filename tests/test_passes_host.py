"""What decides whether a pass is issued as one host call (passes.py), as far as no GPU is needed: models that it does not cover, changes
of a model that a table must notice."""

import pytest
import torch
from torch.nn.utils import prune

from gpt_triton_b200 import passes
from gpt_triton_b200.gpt import FusedGPT, GPTConfig


def _gpt():
    return FusedGPT(GPTConfig(vocab_size=64, block_size=16, n_layer=2, n_head=2, n_embd=32)).eval()


def _blocks(model):
    return [tuple(b.children()) for b in model.blocks]


@pytest.mark.parametrize("slot,name", [(0, "c_attn_weight"), (0, "layer_norm_bias"), (1, "ffn2_bias")])
def test_a_gpt_weight_that_is_no_parameter_is_not_covered(slot, name):
    model = _gpt()
    prune.random_unstructured(model.blocks[1][slot], name, amount=0.5)
    assert passes._gpt_table(model, _blocks(model), folded=False) is None
