"""Products on tiles of 64 rows (gemm_few_kernel): rows at the edges of its tiles of A (16, 32, 64 rows) and of one and several row
tiles (above 64 rows the larger of the shapes below go to the next kernel, and those of 300 rows and 264 columns stay),
columns at the edges of its 16, 32 and 64-column tiles, depths below and above one k-block and one pass through the ring."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
ROWS = [1, 15, 16, 17, 33, 64, 65, 128, 300]


def _randn(*shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("K_,N", [(8, 16), (72, 40), (200, 1032), (3072, 768), (128, 3848), (1216, 7696)])
def test_same_bits_as_the_kernel_for_many_rows(rows, K_, N):
    from gpt_triton_b200 import kernels as K

    x = _randn(640, K_, seed=K_).half().to(DEV)
    w = K.pack_weight(_randn(K_, N, seed=N, scale=0.05).half().to(DEV))
    b, r = _randn(N, seed=1).half().to(DEV), _randn(640, N, seed=2).half().to(DEV)
    few = lambda t: t[:rows].contiguous()
    for kw in ({}, {"add_gelu": True}):
        assert torch.equal(K.fused_ffn(few(x), w, bias=b, **kw), K.fused_ffn(x, w, bias=b, **kw)[:rows])
    z, s = K.fused_ffn(few(x), w, bias=b, residual=few(r), return_row_stats=True)
    zw, sw = K.fused_ffn(x, w, bias=b, residual=r, return_row_stats=True)
    assert torch.equal(z, zw[:rows])
    assert (s.mean - sw.mean[:rows]).abs().max() < 1e-5 and (s.rstd / sw.rstd[:rows] - 1).abs().max() < 1e-5
    if N <= 1032:
        g, be = (1 + 0.1 * _randn(N, seed=3)).half().to(DEV), _randn(N, seed=4, scale=0.1).half().to(DEV)
        fw = K.fold_layer_norm(_randn(N, 264, seed=5, scale=0.05).half().to(DEV), g, be, _randn(264, seed=6).half().to(DEV))
        stats = K.RowStats(sw.data[:rows].contiguous(), N, sw.ext[:rows].contiguous())
        assert torch.equal(K.fused_ffn(z, fw, ln_stats=stats, add_gelu=True), K.fused_ffn(zw, fw, ln_stats=sw, add_gelu=True)[:rows])
    assert K.device_status() == 0


@pytest.mark.parametrize("rows", ROWS)
@pytest.mark.parametrize("K_,N", [(8, 24), (136, 72), (2048, 264), (520, 3904), (64, 7752)])
def test_products_around_deferred_norms(rows, K_, N):
    """Against float64: an fp32 sum of K exact products is off by at most K * 2^-24 of the sum of their magnitudes (random signs:
    far less), a bf16 result by 2^-8 of itself."""
    from gpt_triton_b200 import kernels as K

    a = _randn(rows, K_, seed=1).bfloat16()
    w = _randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16()
    sumsq = _randn((K_ + 63) // 64, rows, seed=3).abs() + 0.1
    normed = K.NormedRows(a.to(DEV), sumsq.to(DEV), K_, 1e-3)
    op = K.operand_rows(w.to(DEV))[0]
    scale = (sumsq.double().sum(0) / K_ + 1e-3).rsqrt()
    z = a.double() @ w.double().T * scale[:, None]
    bound = 2e-6 * (a.double().abs() @ w.double().abs().T * scale[:, None]) + 1e-6
    assert ((K.linear(normed, op, out_dtype=torch.float32).double().cpu() - z).abs() <= bound).all()
    bias = _randn(N, seed=4)
    got = K.linear(normed, op, bias=bias.to(DEV), act="silu", act_split=N // 2, act_after="sigmoid").double().cpu()
    zb = z + bias.double()
    ref = torch.cat([zb[:, :N // 2] * torch.sigmoid(zb[:, :N // 2]), torch.sigmoid(zb[:, N // 2:])], dim=1)
    assert ((got - ref).abs() <= 2 * bound + ref.abs() * 2.0 ** -8 + 1e-5).all()
    x0, gain = _randn(rows, N, seed=5), 1 + 0.1 * _randn(N, seed=6)
    x = x0.to(DEV)
    nxt = K.linear_residual(normed, op, x, gain.to(DEV), 1e-3)
    want = x0.double() + z
    assert ((x.double().cpu() - want).abs() <= bound + want.abs() * 2.0 ** -22).all()
    xs = x.double().cpu()
    for i in range(nxt.sumsq.shape[0]):
        part = xs[:, i * 64:(i + 1) * 64] if rows <= 512 else xs[:, i * 128:(i + 1) * 128]
        assert ((nxt.sumsq[i].double().cpu() - part.pow(2).sum(1)).abs() <= 1e-5 * part.pow(2).sum(1) + 1e-9).all()
    assert torch.equal(nxt.data.cpu(), (x.cpu() * gain).bfloat16())
    F = N // 2
    g, u = w[:F], w[F:2 * F]
    out = K.gated_linear(normed, K.operand_rows(K.interleave_gated(g, u).to(DEV))[0], K.interleave_gated(bias[:F], bias[F:2 * F]).to(DEV), F, limit=1.5,
                         alpha=1.7).double().cpu()
    zg, zu = zb[:, :F].clamp(max=1.5), zb[:, F:2 * F].clamp(-1.5, 1.5)
    ref = zg * torch.sigmoid(1.7 * zg) * (zu + 1)
    assert ((out - ref).abs() <= 4 * (bound[:, :F] + bound[:, F:2 * F]) + ref.abs() * 2.0 ** -8 + 1e-5).all()
    assert K.device_status() == 0


@pytest.mark.parametrize("rows", [1, 17, 64, 65])
@pytest.mark.parametrize("N", [4480, 4608, 8192])
def test_residual_stream_at_the_edge_of_what_fits(rows, N):
    """Tiles of 16 columns in clusters as long as all of them find room at once (4480 columns), tiles of 64 beyond; bounds as above."""
    from gpt_triton_b200 import kernels as K

    K_ = 136
    a, w = _randn(rows, K_, seed=1).bfloat16(), _randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16()
    x0, gain = _randn(rows, N, seed=5), 1 + 0.1 * _randn(N, seed=6)
    x = x0.to(DEV)
    nxt = K.linear_residual(a.to(DEV), K.operand_rows(w.to(DEV))[0], x, gain.to(DEV), 1e-3)
    want = x0.double() + a.double() @ w.double().T
    bound = 2e-6 * (a.double().abs() @ w.double().abs().T) + 1e-6
    assert ((x.double().cpu() - want).abs() <= bound + want.abs() * 2.0 ** -22).all()
    assert torch.equal(nxt.data.cpu(), (x.cpu() * gain).bfloat16())
    part = x.double().cpu().view(rows, N // 64, 64).pow(2).sum(-1).T
    assert ((nxt.sumsq.double().cpu() - part).abs() <= 1e-5 * part + 1e-9).all()
    assert K.device_status() == 0
