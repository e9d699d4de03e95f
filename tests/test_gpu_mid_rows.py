"""Products of a few hundred to a few thousand rows, on both sides of the line between small and wide tiles (narrow_is_faster): the same
bits as among many rows, and the sums of squares per 128 columns beyond 512 rows whichever kernel leaves them."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
MANY = 6500  # rows that take the wide kernel at all widths below


def _randn(*shape, seed, scale=1.0):
    return torch.randn(shape, generator=torch.Generator().manual_seed(seed)) * scale


@pytest.mark.parametrize("rows", [200, 512, 513, 1100, 1537, 3072])
@pytest.mark.parametrize("K_,N", [(768, 768), (136, 776), (200, 3072), (64, 10888)])
def test_same_bits_as_among_many_rows(rows, K_, N):
    from gpt_triton_b200 import kernels as K

    x, wf = _randn(MANY, K_, seed=K_).half().to(DEV), _randn(K_, N, seed=N, scale=0.05).to(DEV)
    w, b, r = K.pack_weight(wf.half()), _randn(N, seed=1).half().to(DEV), _randn(MANY, N, seed=2).half().to(DEV)
    few = lambda t: t[:rows].contiguous()
    for kw in ({}, {"add_gelu": True}):
        assert torch.equal(K.fused_ffn(few(x), w, bias=b, **kw), K.fused_ffn(x, w, bias=b, **kw)[:rows])
    z, s = K.fused_ffn(few(x), w, bias=b, residual=few(r), return_row_stats=True)
    zw, sw = K.fused_ffn(x, w, bias=b, residual=r, return_row_stats=True)
    assert torch.equal(z, zw[:rows])
    if rows > 512:
        assert torch.equal(s.data, sw.data[:rows]) and torch.equal(s.ext, sw.ext[:rows])
    assert (s.mean - sw.mean[:rows]).abs().max() < 1e-5 and (s.rstd / sw.rstd[:rows] - 1).abs().max() < 1e-5
    g, be = (1 + 0.1 * _randn(K_, seed=3)).half().to(DEV), _randn(K_, seed=4, scale=0.1).half().to(DEV)
    fw = K.fold_layer_norm(wf.half(), g, be, b)
    st = K.row_stats(x)
    mine = K.RowStats(st.data[:rows].contiguous(), K_, st.ext[:rows].contiguous())
    assert torch.equal(K.fused_ffn(few(x), fw, ln_stats=mine, add_gelu=True), K.fused_ffn(x, fw, ln_stats=st, add_gelu=True)[:rows])
    w32, b32, r32 = K.pack_weight(wf), b.float(), r.float()
    assert torch.equal(K.operand_ffn_residual(few(x), w32, b32, few(r32)), K.operand_ffn_residual(x, w32, b32, r32)[:rows])
    assert torch.equal(K.operand_ffn(few(x), w32, b32, add_gelu=True), K.operand_ffn(x, w32, b32, add_gelu=True)[:rows])
    xf, odd = few(x).float(), torch.empty((rows, N + 1), device=DEV)[:, :N]  # (an unaligned float32 result: element by element)
    assert torch.equal(K.fused_ffn(xf, w32, bias=b32, residual=few(r32), add_gelu=True, out=odd), K.fused_ffn(x.float(), w32, bias=b32, residual=r32, add_gelu=True)[:rows])
    assert K.device_status() == 0


@pytest.mark.parametrize("rows", [513, 1100, 2048])
@pytest.mark.parametrize("K_,N", [(136, 776), (1024, 1024), (72, 832)])
def test_the_residual_stream_has_the_same_bits_as_among_many_rows(rows, K_, N):
    from gpt_triton_b200 import kernels as K

    a, op = _randn(MANY, K_, seed=1).bfloat16().to(DEV), K.operand_rows(_randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16().to(DEV))[0]
    x0, gain = _randn(MANY, N, seed=5).to(DEV), (1 + 0.1 * _randn(N, seed=6)).to(DEV)
    x, few = x0.clone(), x0[:rows].clone()
    many, mine = K.linear_residual(a, op, x, gain, 1e-3), K.linear_residual(a[:rows].contiguous(), op, few, gain, 1e-3)
    assert torch.equal(few, x[:rows]) and torch.equal(mine.data, many.data[:rows]) and torch.equal(mine.sumsq, many.sumsq[:, :rows])
    assert K.device_status() == 0


@pytest.mark.parametrize("rows", [300, 512, 513, 1100, 2048, 2500])
@pytest.mark.parametrize("K_,N", [(136, 776), (1024, 1024), (72, 832), (264, 64), (64, 10880)])
def test_products_around_deferred_norms(rows, K_, N):
    """Bounds as in test_gpu_few_rows.py."""
    from gpt_triton_b200 import kernels as K

    a, w = _randn(rows, K_, seed=1).bfloat16(), _randn(N, K_, seed=2, scale=K_ ** -0.5).bfloat16()
    sumsq = _randn((K_ + 127) // 128, rows, seed=3).abs() + 0.1
    normed, op = K.NormedRows(a.to(DEV), sumsq.to(DEV), K_, 1e-3), K.operand_rows(w.to(DEV))[0]
    scale = (sumsq.double().sum(0) / K_ + 1e-3).rsqrt().to(DEV)[:, None]
    ad, wd = a.double().to(DEV), w.double().to(DEV)
    z = ad @ wd.T * scale
    bound = 2e-6 * (ad.abs() @ wd.abs().T * scale) + 1e-6
    assert ((K.linear(normed, op, out_dtype=torch.float32).double() - z).abs() <= bound).all()
    got = K.linear(normed, op, act="silu").double()
    ref = z * torch.sigmoid(z)
    assert ((got - ref).abs() <= 2 * bound + ref.abs() * 2.0 ** -8 + 1e-5).all()
    x0, gain = _randn(rows, N, seed=5).to(DEV), (1 + 0.1 * _randn(N, seed=6)).to(DEV)
    x = x0.clone()
    nxt = K.linear_residual(normed, op, x, gain, 1e-3)
    want = x0.double() + z
    assert ((x.double() - want).abs() <= bound + want.abs() * 2.0 ** -22).all()
    assert torch.equal(nxt.data, (x * gain).bfloat16())
    cols = 64 if rows <= 512 else 128
    assert nxt.sumsq.shape == ((N + cols - 1) // cols, rows)
    for i in range(nxt.sumsq.shape[0]):
        part = x.double()[:, i * cols:(i + 1) * cols].pow(2).sum(1)
        assert ((nxt.sumsq[i].double() - part).abs() <= 1e-5 * part + 1e-9).all()
    y = x0.clone()
    assert K.linear_residual(normed, op, y) is None and torch.equal(y, x)
    bias, F = _randn(N, seed=4), N // 2
    out = K.gated_linear(normed, K.operand_rows(K.interleave_gated(w[:F], w[F:2 * F]).to(DEV))[0], K.interleave_gated(bias[:F], bias[F:2 * F]).to(DEV), F, limit=1.5,
                         alpha=1.7).double()
    zb = z + bias.double().to(DEV)
    zg, zu = zb[:, :F].clamp(max=1.5), zb[:, F:2 * F].clamp(-1.5, 1.5)
    ref = zg * torch.sigmoid(1.7 * zg) * (zu + 1)
    assert ((out - ref).abs() <= 4 * (bound[:, :F] + bound[:, F:2 * F]) + ref.abs() * 2.0 ** -8 + 1e-5).all()
    assert K.device_status() == 0


@pytest.mark.parametrize("N", [64, 72])
def test_more_row_tiles_than_a_grid_has_rows(N):
    """65536 tiles of 128 rows: few columns, so that the rounds alone would allow small tiles at any number of rows."""
    from gpt_triton_b200 import kernels as K

    M, K_ = 65535 * 128 + 1, 16
    a = torch.randn((M, K_), device=DEV, dtype=torch.float16)
    w = torch.randn((N, K_), device=DEV, dtype=torch.float16) * 0.25
    rows = torch.tensor([0, 127, 128, M // 2, M - 129, M - 2, M - 1], device=DEV)
    want = a[rows].double() @ w.double().T
    bound = 2e-6 * (a[rows].double().abs() @ w.double().abs().T) + 1e-6  # an fp32 sum of 16 exact products
    got = K.fused_ffn(a, K.pack_weight(w, weight_is_nk=True))[rows].double()
    assert ((got - want).abs() <= bound + want.abs() * 2.0 ** -11).all()
    got = K.linear(a.bfloat16(), w.bfloat16(), out_dtype=torch.float32)[rows].double()
    ab, wb = a[rows].bfloat16().double(), w.bfloat16().double()
    assert ((got - ab @ wb.T).abs() <= 2e-6 * (ab.abs() @ wb.abs().T) + 1e-6).all()
    assert K.device_status() == 0
