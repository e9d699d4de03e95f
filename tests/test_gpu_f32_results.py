"""fp32 results that leave the wide product kernel through staging boxes (32 rows x 32 columns): edges of boxes, slices and tiles.
Against the same kernel's stores from registers (taken by a row pitch that no tensor map allows): the same bits; and, for the residual
stream, against float64."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _randn(*shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale


@pytest.mark.parametrize("rows", [1, 33, 129, 257, 700])
@pytest.mark.parametrize("K_,N", [(72, 36), (64, 132), (768, 264), (200, 1028)])
def test_same_bits_as_stores_from_registers(rows, K_, N):
    from gpt_triton_b200 import kernels as K

    x, w = _randn(rows, K_, seed=1).to(DEV), K.pack_weight(_randn(K_, N, seed=2, scale=0.1).to(DEV))
    b, r = _randn(N, seed=3).to(DEV), _randn(rows, N, seed=4).to(DEV)
    for kw in ({}, {"bias": b}, {"bias": b, "add_gelu": True}, {"bias": b, "residual": r}, {"bias": b, "residual": r, "add_gelu": True}):
        odd = torch.full((rows, N + 1), 7.0, device=DEV)
        staged = torch.full((rows, N + 4), 7.0, device=DEV)
        K.fused_ffn(x, w, out=odd[:, :N], **kw)
        K.fused_ffn(x, w, out=staged[:, :N], **kw)
        assert torch.equal(odd[:, :N], staged[:, :N])
        assert (odd[:, N:] == 7).all() and (staged[:, N:] == 7).all()
    assert K.device_status() == 0


@pytest.mark.parametrize("rows", [513, 769])
@pytest.mark.parametrize("K_,N", [(64, 24), (136, 132), (1024, 264), (64, 1030)])  # (1030: rows that no tensor map allows)
def test_residual_stream_and_row_sums(rows, K_, N):
    """An fp32 sum of K exact products is off by at most K * 2^-24 of the sum of their magnitudes (random signs: far less)."""
    from gpt_triton_b200 import kernels as K

    a, w = _randn(rows, K_, seed=1).bfloat16(), _randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16()
    sumsq = _randn((K_ + 127) // 128, rows, seed=3).abs() + 0.1
    normed = K.NormedRows(a.to(DEV), sumsq.to(DEV), K_, 1e-3)
    scale = (sumsq.double().sum(0) / K_ + 1e-3).rsqrt()[:, None]
    z, bound = a.double() @ w.double().T * scale, 2e-6 * (a.double().abs() @ w.double().abs().T * scale) + 1e-6
    x0, gain = _randn(rows, N, seed=5), 1 + 0.1 * _randn(N, seed=6)
    x = x0.to(DEV)
    nxt = K.linear_residual(normed, K.operand_rows(w.to(DEV))[0], x, gain.to(DEV), 1e-3)
    want = x0.double() + z
    assert ((x.double().cpu() - want).abs() <= bound + want.abs() * 2.0 ** -22).all()
    assert torch.equal(nxt.data.cpu(), (x.cpu() * gain).bfloat16())
    for i in range(nxt.sumsq.shape[0]):
        part = x.double().cpu()[:, i * 128:(i + 1) * 128].pow(2).sum(1)
        assert ((nxt.sumsq[i].double().cpu() - part).abs() <= 1e-5 * part + 1e-9).all()
    y = _randn(rows, N, seed=7).to(DEV)
    assert K.linear_residual(normed, K.operand_rows(w.to(DEV))[0], y) is None
    logits = K.linear(normed, K.operand_rows(w.to(DEV))[0], out_dtype=torch.float32)
    assert ((logits.double().cpu() - z).abs() <= bound).all()
    assert K.device_status() == 0


# Several tiles of 256 x 256 per CTA pair (20000 rows: 79 row tiles), so that the boxes' barriers are used again from tile to tile;
# 1056 columns leave one box in the last tile's slice, 1124 a whole tile and an odd number of boxes, 1252 a slice without columns.
@pytest.mark.parametrize("N", [1056, 1124, 1252])
def test_many_tiles_with_a_residual(N):
    from gpt_triton_b200 import kernels as K

    g = torch.Generator(device=DEV).manual_seed(N)
    rows, K_ = 20000, 64
    x, w = torch.randn((rows, K_), device=DEV, generator=g), K.pack_weight(torch.randn((K_, N), device=DEV, generator=g) * 0.1)
    b, r = torch.randn(N, device=DEV, generator=g), torch.randn((rows, N), device=DEV, generator=g)
    for kw in ({"bias": b, "residual": r}, {"bias": b, "residual": r, "add_gelu": True}, {"bias": b}):
        odd = torch.full((rows, N + 1), 7.0, device=DEV)
        K.fused_ffn(x, w, out=odd[:, :N], **kw)
        assert torch.equal(K.fused_ffn(x, w, **kw), odd[:, :N])
    assert K.device_status() == 0


@pytest.mark.parametrize("N", [1056, 1124, 1252])
@pytest.mark.parametrize("with_gain", [False, True])
def test_residual_stream_over_many_tiles(N, with_gain):
    """Bounds as in test_residual_stream_and_row_sums."""
    from gpt_triton_b200 import kernels as K

    g = torch.Generator(device=DEV).manual_seed(N)
    rows, K_ = 20000, 64
    a, w = torch.randn((rows, K_), device=DEV, generator=g).bfloat16(), (torch.randn((N, K_), device=DEV, generator=g) / 8).bfloat16()
    sumsq = torch.rand((1, rows), device=DEV, generator=g) * K_ + 1
    scale = (sumsq[0].double() / K_ + 1e-3).rsqrt()[:, None]
    z, bound = a.double() @ w.double().T * scale, 2e-6 * (a.double().abs() @ w.double().abs().T * scale) + 1e-6
    x0, gain = torch.randn((rows, N), device=DEV, generator=g), 1 + 0.1 * torch.randn(N, device=DEV, generator=g)
    x = x0.clone()
    nxt = K.linear_residual(K.NormedRows(a, sumsq, K_, 1e-3), K.operand_rows(w)[0], x, gain if with_gain else None, 1e-3)
    want = x0.double() + z
    assert ((x.double() - want).abs() <= bound + want.abs() * 2.0 ** -22).all()
    if with_gain:
        assert torch.equal(nxt.data, (x * gain).bfloat16())
        for i in range(nxt.sumsq.shape[0]):
            part = x.double()[:, i * 128:(i + 1) * 128].pow(2).sum(1)
            assert ((nxt.sumsq[i].double() - part).abs() <= 1e-5 * part + 1e-9).all()
    assert K.device_status() == 0
