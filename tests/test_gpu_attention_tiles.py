"""Causal attention on the tensor cores by head size, length and number of tiles: the kernel for many tiles (up to 64 columns), the one
for few, the one for 128 columns, and what stays with the generic kernel."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _qkv(B, H, L, D, dtype, seed=0):
    g = torch.Generator().manual_seed(seed)
    return [torch.randn((B, H, L, D), generator=g).to(dtype).to(DEV) for _ in range(3)]


def _check(q, k, v, z, rows=None):
    """Against float64: P rounded to fp16 (2^-11 of itself, denominators not; below 2^-14 absolutely, by 2^-25 per key), ex2.approx and
    the fp32 sums (1e-6), the result to its type."""
    L, D = q.shape[2], q.shape[3]
    s = q.double() @ k.double().transpose(2, 3) / math.sqrt(D)
    s.masked_fill_(torch.ones(L, L, dtype=torch.bool, device=DEV).triu(1), -math.inf)
    p = torch.softmax(s, -1)
    ref = p @ v.double()
    weight = (s.amax(-1).exp() / s.exp().sum(-1))[..., None]  # of the largest score: what a rounding of exp(s - max) counts
    unit = 2.0 ** -11 if z.dtype == torch.float16 else 2.0 ** -8
    bound = (2.0 ** -11 + 2e-6) * (p @ v.double().abs()) + 2.0 ** -25 * weight * v.double().abs().cumsum(2) + unit * ref.abs() + 1e-6
    assert ((z.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [16, 32, 64, 128])
@pytest.mark.parametrize("B,H,L", [(1, 1, 1), (2, 3, 63), (1, 2, 64), (2, 2, 65), (3, 2, 128), (2, 5, 129), (1, 3, 300), (40, 16, 193), (1, 2, 1100), (9, 25, 257)])
def test_against_64_bits(dtype, D, B, H, L):
    from gpt_triton_b200 import kernels as K

    q, k, v = _qkv(B, H, L, D, dtype, seed=L + D)
    _check(q, k, v, K.flash_attention_v1(q, k, v))
    assert K.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64, 128])
def test_views_of_a_fused_projection(dtype, D):
    from gpt_triton_b200 import kernels as K

    B, H, L = 40, 8, 200
    x = torch.randn((B, L, 3 * H * D), generator=torch.Generator().manual_seed(D)).to(dtype).to(DEV)
    q, k, v = K.split_qkv(x, H)
    merged = K.flash_attention_v1(q, k, v, merged_heads=True)
    z = K.flash_attention_v1(*(t.contiguous() for t in (q, k, v)))
    assert torch.equal(merged.view(B, L, H, D).transpose(1, 2), z)
    _check(q, k, v, z)
    assert K.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,L", [(16, 200), (32, 129), (64, 300), (64, 128), (64, 1100), (128, 300)])
def test_a_head_does_not_depend_on_the_others(dtype, D, L):
    """Few heads and many take different kernels at 64 columns: the same bits."""
    from gpt_triton_b200 import kernels as K

    q, k, v = _qkv(60, 12, L, D, dtype)
    whole = K.flash_attention_v1(q, k, v)
    for b, h in ((0, 0), (59, 11), (31, 5)):
        one = [t[b:b + 1, h:h + 1].contiguous() for t in (q, k, v)]
        assert torch.equal(K.flash_attention_v1(*one)[0, 0], whole[b, h])
    assert K.device_status() == 0


def test_growing_scores():
    """Every block raises the running maximum far: the output is rescaled in each of them."""
    from gpt_triton_b200 import kernels as K

    B, H, L, D = 40, 12, 700, 64
    q, k, v = _qkv(B, H, L, D, torch.float16)
    q = q.abs() * 0.5
    k = k.abs() * (torch.arange(L, device=DEV) / 100.0)[None, None, :, None].half()
    _check(q, k, v, K.flash_attention_v1(q, k, v))
    assert K.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,L", [(16, 100), (16, 129), (16, 300), (16, 1100), (32, 128)])
def test_small_heads_stay_with_the_generic_kernel(dtype, D, L):
    """The bits of the one kernel that takes rows at any address."""
    from gpt_triton_b200 import kernels as K

    q, k, v = _qkv(2, 3, L, D, dtype)
    anywhere = [torch.empty(t.numel() + 1, dtype=dtype, device=DEV)[1:].view(t.shape).copy_(t) for t in (q, k, v)]
    assert torch.equal(K.flash_attention_v1(q, k, v), K.flash_attention_v1(*anywhere))
    assert K.device_status() == 0
