"""Attention of float32 rows that are fetched ahead (head sizes up to 64, 16-byte rows): the bits of the general kernel, which takes the
same rows one element off, on each side of the lines between its variants."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("out_dtype", [torch.float32, torch.float16])
@pytest.mark.parametrize("D", [16, 32, 64])
@pytest.mark.parametrize("B,H,L", [(1, 1, 1), (2, 3, 17), (1, 2, 64), (2, 2, 65), (1, 3, 129), (1, 2, 513), (40, 15, 64), (16, 12, 300), (3, 37, 512), (6, 12, 600), (9, 25, 193)])
def test_the_bits_of_the_general_kernel(out_dtype, D, B, H, L):
    from gpt_triton_b200 import kernels as K

    g = torch.Generator().manual_seed(L + D)
    x = (torch.randn((B, L, 3 * H * D), generator=g) * 2).to(DEV)
    x[0, L // 2, : D] = float("inf")  # a query and, behind it, a key without a score, and a value beyond fp16
    x[-1, L // 3, H * D : H * D + 4] = float("nan")
    x[-1, L // 4, -1] = 1e6
    odd = torch.empty((B, L, 3 * H * D + 1), device=DEV)
    odd[..., 1:] = x
    rows = lambda t: [t[..., i * H * D : (i + 1) * H * D].view(B, L, H, D).transpose(1, 2) for i in range(3)]
    assert rows(odd[..., 1:])[0].data_ptr() % 16 == 4
    for merged in (True, False):
        a = K.flash_attention_v1(*rows(x), merged_heads=merged, out_dtype=out_dtype)
        b = K.flash_attention_v1(*rows(odd[..., 1:]), merged_heads=merged, out_dtype=out_dtype)
        assert torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(0.0), b.nan_to_num(0.0))
    finite = [t.nan_to_num(0.0, 1.0, -1.0).clamp(-8, 8) for t in rows(x)]
    wide = [torch.empty((B, H, L, D + 4), device=DEV)[..., :D].copy_(t) for t in finite]  # (another row stride)
    y = K.flash_attention_v1(*finite, out_dtype=out_dtype)
    assert torch.equal(K.flash_attention_v1(*wide, out_dtype=out_dtype), y)
    # the first rows, with neither the rows behind them nor the other sequences
    assert torch.equal(K.flash_attention_v1(*(t[:1, :, : (L + 1) // 2] for t in finite), out_dtype=out_dtype), y[:1, :, : (L + 1) // 2])
    assert K.device_status() == 0
