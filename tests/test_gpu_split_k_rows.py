"""Products of at most 16 rows around deferred norms that are cut along K (linear_few_kernel): depths of one to eight ranges per
cluster with ragged last steps, columns at the edges of its 64-column slices, both of its row counts (8 and 16)."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randn(*shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale


@pytest.mark.parametrize("rows", [1, 8, 9, 16])
@pytest.mark.parametrize("K_,N", [(512, 64), (520, 72), (2056, 1032), (4096, 2048), (8184, 136), (2048, 9536)])
def test_against_64_bits(rows, K_, N):
    """Bounds as in test_gpu_few_rows.py: an fp32 sum of K exact products against the sum of their magnitudes, bf16 results by 2^-8."""
    from gpt_triton_b200 import kernels as K

    a, w = _randn(rows, K_, seed=1).bfloat16(), _randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16()
    sumsq = _randn((K_ + 63) // 64, rows, seed=3).abs() + 0.1
    normed, op = K.NormedRows(a.to(DEV), sumsq.to(DEV), K_, 1e-3), K.operand_rows(w.to(DEV))[0]
    scale = (sumsq.double().sum(0) / K_ + 1e-3).rsqrt()
    z = a.double() @ w.double().T * scale[:, None]
    bound = 2e-6 * (a.double().abs() @ w.double().abs().T * scale[:, None]) + 1e-6
    assert ((K.linear(normed, op, out_dtype=torch.float32).double().cpu() - z).abs() <= bound).all()
    bias = _randn(N, seed=4)
    zb = z + bias.double()
    got = K.linear(normed, op, bias=bias.to(DEV), act="silu", act_split=N // 2 + 1, act_after="sigmoid").double().cpu()
    s = torch.sigmoid(zb)
    ref = torch.cat([(zb * s)[:, :N // 2 + 1], s[:, N // 2 + 1:]], dim=1)
    assert ((got - ref).abs() <= 2 * bound + ref.abs() * 2.0 ** -8 + 1e-5).all()
    x0, gain = _randn(rows, N, seed=5), 1 + 0.1 * _randn(N, seed=6)
    x = x0.to(DEV)
    nxt = K.linear_residual(normed, op, x, gain.to(DEV), 1e-3)
    want = x0.double() + z
    assert ((x.double().cpu() - want).abs() <= bound + want.abs() * 2.0 ** -22).all()
    assert torch.equal(nxt.data.cpu(), (x.cpu() * gain).bfloat16())
    for i in range(nxt.sumsq.shape[0]):
        part = x.double().cpu()[:, i * 64:(i + 1) * 64].pow(2).sum(1)
        assert ((nxt.sumsq[i].double().cpu() - part).abs() <= 1e-5 * part + 1e-9).all()
    assert K.linear_residual(normed, op, x) is None
    F = N // 2
    out = K.gated_linear(normed, K.operand_rows(K.interleave_gated(w[:F], w[F:2 * F]).to(DEV))[0], K.interleave_gated(bias[:F], bias[F:2 * F]).to(DEV), F, limit=1.5,
                         alpha=1.7).double().cpu()
    zg, zu = zb[:, :F].clamp(max=1.5), zb[:, F:2 * F].clamp(-1.5, 1.5)
    ref = zg * torch.sigmoid(1.7 * zg) * (zu + 1)
    assert ((out - ref).abs() <= 4 * (bound[:, :F] + bound[:, F:2 * F]) + ref.abs() * 2.0 ** -8 + 1e-5).all()
    assert K.device_status() == 0


@pytest.mark.parametrize("K_,N", [(512, 64), (1016, 1024), (1024, 1024), (1024, 3088), (1024, 4096), (1536, 3200), (2048, 8192), (2048, 8320), (2048, 9408), (4096, 1032)])
def test_up_to_16_rows_a_row_does_not_depend_on_the_others(K_, N):
    """Whichever kernel takes the product: on both sides of the lines between the two.  (Beyond 16 rows sums are in another order.)"""
    from gpt_triton_b200 import kernels as K

    a, w = _randn(16, K_, seed=1).bfloat16().to(DEV), _randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16()
    op, pairs = K.operand_rows(w.to(DEV))[0], K.operand_rows(K.interleave_gated(w[:N // 2], w[N // 2:]).to(DEV))[0]
    sumsq, x0, gain, bias = _randn(3, 16, seed=3).abs().to(DEV), _randn(16, N, seed=4).to(DEV), _randn(N, seed=5).to(DEV), _randn(pairs.shape[0], seed=6).to(DEV)

    def results(rows):
        normed = K.NormedRows(a[:rows].contiguous(), sumsq[:, :rows].contiguous(), K_, 1e-3)
        x = x0[:rows].clone()
        following = K.linear_residual(normed, op, x, gain, 1e-3)
        return [K.linear(normed, op, out_dtype=torch.float32), K.linear(normed, op, act="silu"), x, following.data, following.sumsq.t(),
                K.gated_linear(normed, pairs, bias, N // 2, limit=1.5, alpha=1.7)]

    whole = results(16)
    for rows in (1, 3, 8, 9, 15):
        assert all(torch.equal(few, all_[:rows]) for few, all_ in zip(results(rows), whole))
