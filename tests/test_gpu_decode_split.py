"""One-query attention over the cache with 8, 4, 2 and 1 warps per (batch, head), a block of keys and
values in registers ahead or not: which one runs depends on how many (batch, head) pairs the GPU has room for
at once and on the cache's length (below: at head size 64); keys at the edges of a 64-key block and of a group of blocks.  Against the last row of the
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
                                    (297, 12, 65)])                                                              # one, no room for all at once
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


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D", [32, 64, 128])
@pytest.mark.parametrize("pairs", [12, 148, 149, 296, 297, 592, 593, 1036, 1037, 1184, 1185, 2368, 2369, 3552, 3553, 4737])
def test_one_block_of_keys_in_a_long_cache(dtype, D, pairs):
    """Up to 64 keys are one block, whose result does not depend on how many warps the cache's length asks for: the bits of a cache that
    is just long enough (pairs: at the edges of what finds room at once)."""
    from gpt_triton_b200 import kernels as K

    g = torch.Generator(device=DEV).manual_seed(pairs + D)
    B, NH = (pairs // 4, 4) if pairs % 4 == 0 else (pairs, 1)
    H = NH * D
    keys = torch.randn((B, 64, 2 * H), generator=g, device=DEV).to(dtype)
    for n in (1, 16, 17, 64):
        new = torch.randn((B, 3 * H), generator=g, device=DEV).to(dtype)
        pos = torch.tensor([n - 1, 0], dtype=torch.int32, device=DEV)
        outs = []
        for room in (0, 30, 100, 300):
            cache = torch.full((B, n + room, 2 * H), float("nan"), device=DEV, dtype=dtype)
            cache[:, :n - 1] = keys[:, :n - 1]
            outs.append(K.attention_decode(new, cache, pos, NH))
            assert torch.equal(cache[:, n - 1], new[:, H:]) and torch.equal(cache[:, :n - 1], keys[:, :n - 1])
        assert all(torch.equal(o, outs[0]) for o in outs) and not torch.isnan(outs[0].float()).any()
    assert K.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D", [32, 64])
@pytest.mark.parametrize("B,n", [(400, 120), (400, 150), (400, 321)])
def test_more_pairs_than_find_room(dtype, D, B, n):
    """12 heads; tolerances as above."""
    from gpt_triton_b200 import kernels as K

    g = torch.Generator(device=DEV).manual_seed(n + D)
    H = 12 * D
    cache = torch.randn((B, n, 2 * H), generator=g, device=DEV).to(dtype)
    new = torch.randn((B, 3 * H), generator=g, device=DEV).to(dtype)
    out = K.attention_decode(new, cache, torch.tensor([n - 1, 0], dtype=torch.int32, device=DEV), 12)
    assert K.device_status() == 0 and torch.equal(cache[:, -1], new[:, H:])
    operand = lambda t: t.half().float()
    k, v = (operand(t).view(B, n, 12, D) for t in cache.split(H, dim=-1))
    p = torch.einsum("bhd,bnhd->bhn", operand(new[:, :H]).view(B, 12, D), k).div(D ** 0.5).softmax(-1)
    ref = torch.einsum("bhn,bnhd->bhd", p, v).reshape(B, H)
    assert (out.float() - ref).abs().max().item() < {torch.float16: 2e-3, torch.bfloat16: 1.6e-2}[dtype]
