"""Products, LayerNorms and attention that start under the kernel in front of them: chains through reused buffers give the bits of
the same calls made one at a time, in a stream, in a captured graph, and behind a join of two streams."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("batch,length", [(1, 513), (4, 1280), (7, 732), (16, 1000)])  # up to, at and beyond the few- and mid-row lines
@pytest.mark.parametrize("captured", [False, True])
def test_chains_through_reused_buffers(batch, length, captured):
    from gpt_triton_b200 import kernels as K

    H, heads, rows = 768, 12, batch * length
    rand = lambda *s, seed, scale=1.0: (torch.randn(s, generator=torch.Generator().manual_seed(seed)) * scale).half().to(DEV)
    w1, b1 = K.pack_weight(rand(H, 3 * H, seed=1, scale=0.03)), rand(3 * H, seed=2)
    w2, b2 = K.pack_weight(rand(H, H, seed=3, scale=0.03)), rand(H, seed=4)
    gain, shift, x0 = 1 + 0.1 * rand(H, seed=5), rand(H, seed=6, scale=0.1), rand(rows, H, seed=7)
    x, qkv, y = torch.empty_like(x0), rand(rows, 3 * H, seed=8), rand(rows, H, seed=9)

    def chain(side=None, pause=lambda: None):
        x.copy_(x0)
        for _ in range(3):  # every step writes what the step in front of it has just read
            K.fused_ffn(x, w1, bias=b1, out=qkv)
            pause()
            q, k, v = K.split_qkv(qkv.view(batch, length, 3 * H), heads)
            o = K.flash_attention_v1(q, k, v, merged_heads=True).view(rows, H)
            pause()
            if side is not None:  # the other half of the rows on a second stream; a product stands behind the join
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    K.fused_ffn(o[rows // 2 :], w2, bias=b2, residual=x[rows // 2 :], out=y[rows // 2 :])
                K.fused_ffn(o[: rows // 2], w2, bias=b2, residual=x[: rows // 2], out=y[: rows // 2])
                torch.cuda.current_stream().wait_stream(side)
            else:
                K.fused_ffn(o, w2, bias=b2, residual=x, out=y)
            pause()
            K.fused_ffn(y, w2, bias=b2, out=x)
            pause()
            n = K.fused_layer_norm(x, gain, shift)
            pause()
            K.fused_ffn(n, w2, bias=b2, residual=y, add_gelu=True, out=x)
            pause()
        return x

    expected = chain(pause=torch.cuda.synchronize).clone()
    assert torch.isfinite(expected).all()
    for side in (None, torch.cuda.Stream()):
        if captured:
            x.zero_()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                chain(side)
            for _ in range(3):
                graph.replay()
        else:
            for _ in range(3):
                chain(side)
        torch.cuda.synchronize()
        assert torch.equal(x, expected)
    assert K.device_status() == 0
