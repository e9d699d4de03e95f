"""One-query attention of many sequences with keys and values staged in shared memory, and the calls on the other side of its lines:
fewer pairs than 6 per SM (10 at head size 32), a cache of one block, pairs that fill a wave and a bit."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("dtype", [torch.float16, torch.bfloat16])
@pytest.mark.parametrize("D,B,NH", [(64, 887, 1), (64, 222, 4), (64, 148, 12), (64, 1777, 1), (64, 333, 8), (64, 256, 12), (32, 1479, 1), (32, 148, 10), (32, 142, 25), (32, 256, 25)])
@pytest.mark.parametrize("n,spare", [(1, 70), (63, 2), (64, 1), (65, 0), (128, 5), (129, 0), (331, 3)])
def test_against_64_bits(dtype, D, B, NH, n, spare):
    from gpt_triton_b200 import kernels as K

    H, cap = NH * D, n + spare
    g = torch.Generator(device=DEV).manual_seed(n + D + B)
    rows = torch.randn((B, n, 3 * H), generator=g, device=DEV).to(dtype)
    cache = torch.full((B, cap, 2 * H), float("nan"), device=DEV, dtype=dtype)  # what lies behind the position must not be read
    cache[:, : n - 1] = rows[:, : n - 1, H:]
    new = rows[:, -1].contiguous()
    out = K.attention_decode(new, cache, torch.tensor([n - 1, 0], dtype=torch.int32, device=DEV), NH).view(B, NH, D)
    assert torch.equal(cache[:, n - 1], new[:, H:]) and torch.isnan(cache[:, n:].float()).all()
    assert torch.equal(cache[:, : n - 1], rows[:, : n - 1, H:])
    q, k, v = (t.view(B, n, NH, D).transpose(1, 2).double() for t in rows.split(H, dim=2))
    s = (q[:, :, -1:] @ k.transpose(2, 3)) / math.sqrt(D)
    p = torch.softmax(s, -1)
    ref = (p @ v)[:, :, 0]
    # P is rounded to fp16 (2^-11 of itself; 2^-25 per key of the largest weight below 2^-14), the sums and ex2.approx are fp32 (2e-6 at
    # scores of at most 2^4), the result takes its type
    unit = 2.0 ** -11 if dtype == torch.float16 else 2.0 ** -8
    bound = (2.0 ** -11 + 2e-5) * (p @ v.abs())[:, :, 0] + 2.0 ** -25 * p.amax(-1) * v.abs().sum(2) + unit * ref.abs() + 1e-6
    assert ((out.double() - ref).abs() <= bound).all()
    assert K.device_status() == 0
