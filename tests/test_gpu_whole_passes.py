"""A pass issued as one host call (passes.py) against the operators one by one: the same bits, the same launches."""

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _launches(fn):
    from gpt_triton_b200 import _lib

    n0 = _lib.load().b200_launch_count()
    out = fn()
    return out, _lib.load().b200_launch_count() - n0


def _both(model, fn):
    """fn() as whole passes and operator by operator; results must be equal, launches too."""
    a, na = _launches(fn)
    model.whole_passes = False
    b, nb = _launches(fn)
    model.whole_passes = True
    a, b = (x if isinstance(x, (list, tuple)) else [x] for x in (a, b))
    assert len(a) == len(b) and all(torch.equal(x, y) for x, y in zip(a, b)) and na == nb > 0


def _gpt(dtype, hidden=128, heads=4, layers=3):
    from gpt_triton_b200.gpt import FusedGPT, GPTConfig

    torch.manual_seed(hidden + layers)
    model = FusedGPT(GPTConfig(vocab_size=300, block_size=96, n_layer=layers, n_head=heads, n_embd=hidden)).to(DEV)
    for p in model.parameters():
        p.data.copy_(torch.randn_like(p) * 0.05 + (1.0 if p.dim() == 1 and p.shape[0] == hidden else 0.0))
    return model.to(dtype).eval()


@pytest.mark.parametrize("dtype,fold", [(torch.float16, True), (torch.bfloat16, True), (torch.bfloat16, False), (torch.float32, False)])
@pytest.mark.parametrize("B,L", [(1, 1), (3, 43), (2, 64), (4, 96)])  # on both sides of 128 rows
def test_gpt(dtype, fold, B, L):
    from gpt_triton_b200 import kernels as K
    from gpt_triton_b200 import passes
    from gpt_triton_b200.generation import GenerationSession
    from gpt_triton_b200.gpt import FusedAttention, FusedMLP

    model = _gpt(dtype)
    model.fold_layer_norm = fold
    ids = torch.randint(0, 300, (B, L), device=DEV)
    model.logits(ids)
    assert passes.gpt_body(model, ids, None, None, FusedAttention, FusedMLP) is not None  # (covered)
    _both(model, lambda: model(ids))

    def request():
        s = GenerationSession(model, B, capacity=96, use_cuda_graph=False)
        rows = [s.extend(ids[:, :L - 1].contiguous())] if L > 1 else []
        return rows + [s.extend(ids[:, L - 1:].contiguous()), *[c[:, :L].contiguous() for c in s.cache]]

    _both(model, request)
    assert K.device_status() == 0


def test_gpt_notices_changes():
    model = _gpt(torch.float16)
    ids = torch.randint(0, 300, (2, 40), device=DEV)
    first = model(ids)
    with torch.no_grad():
        model.blocks[1][1].ffn1_weight.mul_(1.5)
    model(ids)
    _both(model, lambda: model(ids))
    assert not torch.equal(model(ids), first)
    model.blocks[0][0].c_proj_weight.data.mul_(0.5)  # (no counter notices)
    model.blocks[0][0].refresh_operands()
    model(ids)
    _both(model, lambda: model(ids))
    model.blocks[2] = torch.nn.Sequential(*reversed(list(model.blocks[2].children())))  # a shape that is not covered
    with pytest.raises(TypeError, match="kv_cache"):  # (the operators' own: a feed-forward takes no cache)
        model(ids)


def _decoder(kind, width=64, passes=2):
    from gpt_triton_b200.fogilix import Fogilix
    from gpt_triton_b200.nufasun import Nufasun

    mlp = {"kind": "dense", "ff": 96}
    if kind == "fogilix":
        latent = {"heads": 4, "dim": 16, "vdim": 24, "kv_rank": 32, "mask": {"size": 20}, "scale": 0.25}
        lightning = {"heads": 4, "dim": 16, "vdim": 16, "decay": [0.9, 0.95, 0.99, 1.0]}
        layers = [{"type": "lightning", "mixer": lightning, "mlp": mlp}, {"type": "latent_attention", "mixer": latent}, {"type": "lightning", "mixer": lightning},
                  {"type": "latent_attention", "mixer": {**latent, "kv_from": 1, "heads": 2, "mask": {"size": 33}}, "mlp": mlp}]
        cfg, cls = {"vocab": 211, "width": width, "layers": layers, "norm": {"eps": 1e-5}, "logit_scale": 1.0}, Fogilix
        model = cls(__import__("gpt_triton_b200.fogilix", fromlist=["x"]).FogilixConfig.from_dict(cfg))
    else:
        mlp = {"kind": "dense", "ff": 104, "limit": 2.0}
        delta = {"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 16, "conv": 4}
        pair = {"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 24, "mask": {"size": 21}, "diff": 0.4, "softcap": 20.0, "scale": 0.25, "rot": {"base": 1e4, "dims": 8}}
        layers = [{"type": "delta", "mixer": delta, "mlp": mlp}, {"type": "attention", "mixer": pair, "mlp": mlp}, {"type": "delta", "mixer": delta},
                  {"type": "attention", "mixer": pair}]
        cfg = {"vocab": 211, "width": width, "layers": layers, "norm": {"eps": 1e-5}, "embedding": {"scale": 2.0}, "logit_softcap": 15.0,
               "loop": {"start": 1, "stop": 3, "times": passes}}
        model = Nufasun(__import__("gpt_triton_b200.nufasun", fromlist=["x"]).NufasunConfig.from_dict(cfg))
    torch.manual_seed(1)
    for p in model.parameters():
        p.data.copy_(torch.randn_like(p) * (0.3 if p.dim() < 2 else p.shape[-1] ** -0.5))
    return model.to(DEV).to(torch.bfloat16).eval()


@pytest.mark.parametrize("kind", ["fogilix", "nufasun"])
@pytest.mark.parametrize("B,n", [(1, 5), (2, 70), (3, 300)])
def test_decoders(kind, B, n):
    from gpt_triton_b200 import kernels as K
    from gpt_triton_b200.generation import GenerationSession
    from gpt_triton_b200.mixers import PromptContext

    model = _decoder(kind)
    ids = torch.randint(0, 211, (B, n + 3), device=DEV)
    model.logits(ids)
    assert model._whole_pass(ids.reshape(-1), PromptContext(B, n + 3, 0, None), False) is not None  # (covered)
    _both(model, lambda: model.logits(ids))

    def request():
        s = GenerationSession(model, B, capacity=n + 3, use_cuda_graph=False)
        out = [s.extend(ids[:, :n // 2].contiguous()), s.extend(ids[:, n // 2:n].contiguous()), s.extend(ids[:, n:n + 1].contiguous()), s.extend(ids[:, n + 1:n + 2].contiguous())]
        out = [t for r in out for t in ((r.data, r.sumsq) if isinstance(r, K.NormedRows) else (r,))]
        return out + [model.head_logits(s.extend(ids[:, n + 2:].contiguous()))]

    _both(model, request)
    assert K.device_status() == 0


def test_a_decoder_notices_changes():
    model = _decoder("fogilix")
    ids = torch.randint(0, 211, (2, 50), device=DEV)
    first = model.logits(ids)
    model.layers[1].mix.window = 5
    model.logits(ids)
    _both(model, lambda: model.logits(ids))
    with torch.no_grad():
        model.layers[0].mix.q.mul_(2.0)
    model.logits(ids)
    _both(model, lambda: model.logits(ids))
    assert not torch.equal(model.logits(ids), first)


def test_a_pruned_gpt_runs_its_operators():
    from torch.nn.utils import prune

    from gpt_triton_b200 import passes
    from gpt_triton_b200.gpt import FusedAttention, FusedMLP

    model = _gpt(torch.float16)
    ids = torch.randint(0, 300, (2, 40), device=DEV)
    for _ in range(3):
        first = model(ids)
    prune.l1_unstructured(model.blocks[1][1], "ffn2_bias", amount=0.5)
    for _ in range(3):
        assert not torch.equal(model(ids), first)
    assert passes.gpt_body(model, ids, None, None, FusedAttention, FusedMLP) is None


@pytest.mark.parametrize("kind,where", [("fogilix", "layers.0.mlp.down"), ("fogilix", "layers.1.mix.o"), ("nufasun", "layers.0.mix.o"),
                                        ("nufasun", "layers.1.mlp.down_b"), ("nufasun", "layers.1.norm1b")])
def test_a_decoder_notices_pruning(kind, where):
    """A pruned weight is no parameter any more; pruned again it is another tensor under the same name."""
    from torch.nn.utils import prune

    model = _decoder(kind)
    ids = torch.randint(0, 211, (2, 50), device=DEV)
    owner, _, name = where.rpartition(".")
    last = model.logits(ids)
    for _ in range(2):
        for _ in range(3):
            model.logits(ids)
        prune.random_unstructured(model.get_submodule(owner), name, amount=0.5)
        model.logits(ids)  # (packs the new weights)
        for _ in range(3):
            _both(model, lambda: model.logits(ids))
        assert not torch.equal(model.logits(ids), last)
        last = model.logits(ids)


@pytest.mark.parametrize("kind", ["fogilix", "nufasun"])
def test_a_decoder_with_a_wider_feed_forward(kind):
    """Weights twice as wide (Nufasun's width is a constant of the module too, which the products check)."""
    model = _decoder(kind)
    ids = torch.randint(0, 211, (2, 50), device=DEV)
    first = [model.logits(ids) for _ in range(3)][-1]
    mlp = model.layers[0].mlp
    if kind == "nufasun":
        mlp.ff *= 2
    for name, p in list(mlp._parameters.items()):
        if name != "down_b":
            setattr(mlp, name, torch.nn.Parameter(torch.cat([p.data, 0.5 * p.data], 1 if name == "down" else 0)))
    model.logits(ids)  # (packs the new weights)
    for _ in range(3):
        _both(model, lambda: model.logits(ids))
    assert not torch.equal(model.logits(ids), first)


@pytest.mark.parametrize("make", [lambda: _gpt(torch.bfloat16), lambda: _decoder("fogilix"), lambda: _decoder("nufasun")])
def test_a_copy_is_a_model_of_its_own(make):
    import copy

    model = make()
    ids = torch.randint(0, 200, (2, 50), device=DEV)
    first = [model.logits(ids) for _ in range(3)][-1]
    other = copy.deepcopy(model)
    for _ in range(3):
        assert torch.equal(other.logits(ids), first)
    with torch.no_grad():
        for p in other.parameters():
            p.mul_(1.25)
    other.logits(ids)  # (packs the new weights)
    for _ in range(3):
        _both(other, lambda: other.logits(ids))
        assert torch.equal(model.logits(ids), first) and not torch.equal(other.logits(ids), first)


def test_functions_set_on_a_model_run():
    """Set on a block, on a sublayer or in the place of an operator, after whole passes have run."""
    from gpt_triton_b200 import kernels as K

    ids = torch.randint(0, 200, (2, 50), device=DEV)
    calls = []

    def counted(fn):
        def call(*args, **kwargs):
            calls.append(fn)
            return fn(*args, **kwargs)
        return call

    gpt, fogilix, nufasun = _gpt(torch.float16), _decoder("fogilix"), _decoder("nufasun")
    for model, owner, name, per_pass in ((gpt, gpt.blocks[1][1], "forward_folded", 1), (gpt, K, "flash_attention_v1", 3), (fogilix, fogilix.layers[0].mlp, "prompt", 1),
                                         (fogilix, K, "linear_residual", 6), (nufasun, nufasun.layers[3].mix, "_mix", 1), (nufasun, K, "gated_delta", 3)):
        first = [model.logits(ids) for _ in range(3)][-1]
        before = getattr(owner, name)
        setattr(owner, name, counted(before))
        try:
            calls.clear()
            for n in range(1, 4):
                assert torch.equal(model.logits(ids), first) and len(calls) == n * per_pass
        finally:
            if owner is K:
                K.__dict__[name] = before
            else:
                delattr(owner, name)


@pytest.mark.parametrize("dtype,fold,L", [(torch.float16, True, 96), (torch.bfloat16, False, 96), (torch.float32, False, 96), (torch.float32, False, 1)])
def test_a_gpt_pass_holds_no_more_than_its_operators(dtype, fold, L):
    """(The workspace is one block: a little more for sections rounded up to 256 bytes and its own rounding, of up to 2 MB.)"""
    model = _gpt(dtype, layers=2)
    model.fold_layer_norm = fold
    ids = torch.randint(0, 300, (128 if L == 1 else 400, L), device=DEV)
    peaks = []
    for model.whole_passes in (True, False):
        for _ in range(2):
            model(ids)
        torch.cuda.empty_cache()
        torch.cuda.reset_peak_memory_stats()
        before = torch.cuda.memory_allocated()
        model(ids)
        peaks.append(torch.cuda.max_memory_allocated() - before)
    assert peaks[0] <= peaks[1] * 1.02 + (2 << 20), peaks
