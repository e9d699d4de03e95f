"""float32 blocks whose intermediate rows leave their producers as the fp16 operands they are: the same bits as the operator
sequence that stores them in float32 and converts them on the way in (kernels.py:229-234 of the reference rounds them there).
q | k | v stay float32 between their product and the attention."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("M,K_,N", [(1, 8, 8), (64, 768, 2304), (65, 200, 104), (512, 64, 3072), (513, 72, 264), (640, 768, 768), (1300, 128, 512)])
@pytest.mark.parametrize("gelu", [False, True])
@pytest.mark.parametrize("with_bias", [False, True])
def test_products_give_the_bits_of_the_float32_operators(M, K_, N, gelu, with_bias):
    from gpt_triton_b200 import kernels as K

    g = torch.Generator().manual_seed(M + N)
    x = torch.randn((M, K_), generator=g).to(DEV)
    w = K.pack_weight((torch.randn((K_, N), generator=g) * 0.2).to(DEV))
    b = torch.randn(N, generator=g).to(DEV) if with_bias else None
    r = torch.randn((M, N), generator=g).to(DEV)
    assert K.takes_operand_rows(x, w, b) == (M > 128)
    assert torch.equal(K.operand_ffn(x.half(), w, b, add_gelu=gelu), K.fused_ffn(x, w, bias=b, add_gelu=gelu).half())
    assert torch.equal(K.operand_ffn_residual(x.half(), w, b, r), K.fused_ffn(x, w, bias=b, residual=r))
    assert K.device_status() == 0


@pytest.mark.parametrize("hidden,heads,B,L", [(64, 4, 2, 70), (64, 4, 2, 64), (128, 2, 3, 65), (256, 2, 5, 33), (768, 12, 2, 300), (60, 2, 8, 20)])
@pytest.mark.parametrize("session", [False, True])
def test_blocks_match_the_operator_sequence(hidden, heads, B, L, session):
    """Bit for bit, the prompt of a session (whose keys and values join a cache) too."""
    from gpt_triton_b200 import kernels as K
    from gpt_triton_b200.gpt import FusedAttention, FusedMLP

    if hidden == 60:
        heads = 15  # (head size 4 is no attention size: only the feed-forward runs, by the old route, as 60 % 8 != 0)
    torch.manual_seed(hidden)
    x = torch.randn((B, L, hidden), device=DEV)
    mlp = FusedMLP(hidden).to(DEV).eval()
    ln = lambda m: K.fused_layer_norm(x, m.layer_norm_weight.data, m.layer_norm_bias.data)
    y = K.fused_ffn(ln(mlp), mlp._operand(mlp.ffn1_weight), bias=mlp.ffn1_bias.data, add_gelu=True)
    assert torch.equal(mlp(x), K.fused_ffn(y, mlp._operand(mlp.ffn2_weight), bias=mlp.ffn2_bias.data, residual=x))
    if hidden == 60:
        return
    att = FusedAttention(hidden, heads).to(DEV).eval()
    qkv = K.fused_ffn(ln(att), att._operand(att.c_attn_weight), bias=att.c_attn_bias.data)
    y = K.flash_attention_v1(*K.split_qkv(qkv, heads), merged_heads=True)
    ref = K.fused_ffn(y, att._operand(att.c_proj_weight), bias=att.c_proj_bias.data, residual=x)
    cache = torch.zeros((B, L + 3, 2 * hidden), device=DEV) if session else None
    assert torch.equal(att(x, kv_cache=cache), ref)
    if session:
        assert torch.equal(cache[:, :L], qkv.view(B, L, -1)[:, :, hidden:]) and not cache[:, L:].any()
    assert K.device_status() == 0


@pytest.mark.parametrize("hidden,heads,L", [(128, 2, 100), (768, 12, 128), (96, 3, 129)])
def test_float32_rows_do_not_depend_on_the_batch(hidden, heads, L):
    """The same sequence alone, in a batch and as the prompt of a session (128 rows and fewer take the operators one by one)."""
    from gpt_triton_b200 import kernels as K
    from gpt_triton_b200.gpt import FusedAttention

    torch.manual_seed(L)
    x = torch.randn((3, L, hidden), device=DEV)
    att = FusedAttention(hidden, heads).to(DEV).eval()
    alone = torch.cat([att(x[i:i + 1].contiguous()) for i in range(3)])
    assert torch.equal(att(x), alone)
    assert torch.equal(att(x, kv_cache=torch.zeros((3, L, 2 * hidden), device=DEV)), alone)
    assert K.device_status() == 0


@pytest.mark.parametrize("B,L", [(2, 65), (1, 200), (3, 128)])
def test_attention_block_against_the_oracle(B, L):
    """Head size 64 and more than 128 rows, within the 1e-4 that the float32 operators keep to: the fp16 roundings of P need
    exponentials that are exact in float32."""
    from gpt_triton_b200.gpt import FusedAttention
    from oracle import gpt2_oracle as orc

    hidden, heads = 256, 4
    g = torch.Generator().manual_seed(L)
    att = FusedAttention(hidden, heads).eval()
    with torch.no_grad():
        for name, p in att.named_parameters():
            p.copy_(torch.randn(p.shape, generator=g) * (hidden ** -0.5 if p.dim() == 2 else 0.1) + (name == "layer_norm_weight"))
    x = torch.randn((B, L, hidden), generator=g)
    ref = orc.attention_block({k: v.data for k, v in att.named_parameters()}, "", x, heads)
    got = att.to(DEV)(x.to(DEV)).cpu()
    assert (got - ref).abs().max().item() < 1e-4 * max(1.0, ref.abs().max().item())
