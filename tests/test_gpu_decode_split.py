"""One-query attention over the cache with 8, 4, 2 and 1 warps per (batch, head), a block of keys and
values in registers ahead or not: which one runs depends on the number of (batch, head)
pairs and on the cache's length; keys at the edges of a 64-key block and of a group of blocks.  Against the last row of the
oracle's flash_attention_v1 (kernels.py:417-474 of the reference)."""

import pytest
import torch

from oracle import gpt2_oracle as orc

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("B,NH,L", [(1, 1, 1), (2, 3, 64), (2, 3, 65), (1, 12, 512), (1, 12, 513), (2, 5, 601),  # eight warps
                                    (19, 8, 256), (19, 8, 257), (24, 12, 70),                                    # four
                                    (25, 12, 128), (25, 12, 129), (49, 12, 66),                                  # two
                                    (50, 12, 1), (50, 12, 64), (50, 12, 252),                                    # one
                                    (50, 12, 257), (50, 12, 600),                                                # four, values behind the softmax
                                    (99, 12, 127), (100, 12, 130),                                               # two
                                    (223, 12, 129), (296, 12, 40),                                               # one
                                    (297, 12, 65)])                                                              # two
def test_matches_the_last_row_of_full_attention(dtype, D, B, NH, L):
    from gpt_triton_b200 import kernels as K

    H, cap = NH * D, L + 4
    g = torch.Generator().manual_seed(B * L + D)
    q, k, v = (torch.randn((B, NH, L, D), generator=g).to(dtype) for _ in range(3))
    ref = orc.flash_attention_v1(q, k, v)[:, :, -1, :].reshape(B, H).float()
    merged = lambda t: t.transpose(1, 2).reshape(B, L, H)
    cache = torch.full((B, cap, 2 * H), float("nan"), dtype=dtype)  # what lies behind the position must not be read
    cache[:, :L - 1, :H], cache[:, :L - 1, H:] = merged(k)[:, :L - 1], merged(v)[:, :L - 1]
    new = torch.cat([merged(t)[:, -1] for t in (q, k, v)], dim=1).contiguous()
    cache_d = cache.to(DEV)
    out = K.attention_decode(new.to(DEV), cache_d, torch.tensor([L - 1, 0], dtype=torch.int32, device=DEV), NH).cpu().float()
    assert K.device_status() == 0
    # half a unit in the last place of outputs below 4 on either side; P is rounded to fp16 on both, a flip of one weight moves an
    # output by at most 2^-11 of it
    assert (out - ref).abs().max().item() < {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]
    got = cache_d.cpu()
    assert torch.equal(got[:, L - 1], new[:, H:])
    assert torch.equal(got[:, :L - 1], cache[:, :L - 1]) and torch.isnan(got[:, L:].float()).all()
