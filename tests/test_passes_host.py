"""What decides whether a pass is issued as one host call (passes.py), as far as no GPU is needed: models that it does not cover, changes
of a model that a table must notice."""

import copy
import ctypes
import io
import os
import pickle
import re

import pytest
import torch
from torch.nn.utils import prune

import fogilix_cases
import nufasun_cases
from gpt_triton_b200 import kernels as K
from gpt_triton_b200 import mixers, passes
from gpt_triton_b200.fogilix import Fogilix, FogilixConfig
from gpt_triton_b200.gpt import FusedAttention, FusedGPT, GPTConfig
from gpt_triton_b200.module_base import parameter_tags
from gpt_triton_b200.nufasun import Nufasun, NufasunConfig


def _gpt():
    return FusedGPT(GPTConfig(vocab_size=64, block_size=16, n_layer=2, n_head=2, n_embd=32)).eval()


def _decoder(kind):
    if kind == "fogilix":
        return Fogilix(FogilixConfig.from_dict(fogilix_cases.CONFIGS["mixed"])).bfloat16().eval()
    return Nufasun(NufasunConfig.from_dict(nufasun_cases.CONFIGS["mixed"])).bfloat16().eval()


def _is_stock(model):
    """Whether the checks in front of a table let the model through (what follows them launches kernels)."""
    class Passed(Exception):
        pass

    def derived(*args):
        raise Passed

    model._operand.derived = derived
    try:
        return model._table() is not None
    except Passed:
        return True
    finally:
        del model._operand.derived


def _blocks(model):
    return [tuple(b.children()) for b in model.blocks]


@pytest.mark.parametrize("slot,name", [(0, "c_attn_weight"), (0, "layer_norm_bias"), (1, "ffn2_bias")])
def test_a_gpt_weight_that_is_no_parameter_is_not_covered(slot, name):
    model = _gpt()
    prune.random_unstructured(model.blocks[1][slot], name, amount=0.5)
    assert passes._gpt_table(model, _blocks(model), folded=False) is None


@pytest.mark.parametrize("kind", ["fogilix", "nufasun"])
def test_pruning_is_noticed_and_not_covered(kind):
    """Also of the last parameter of a module, whose successor `..._orig` takes its place."""
    for name in ("mix.o", "mix.q", "mlp.down", "mlp.up", "norm1"):
        model = _decoder(kind)
        assert _is_stock(model)
        owner, _, weight = name.rpartition(".")
        before = parameter_tags(model, structure=True)
        assert parameter_tags(model, structure=True) == before
        prune.random_unstructured(model.layers[0].get_submodule(owner), weight, amount=0.5)
        assert parameter_tags(model, structure=True) != before
        assert not _is_stock(model)


@pytest.mark.parametrize("kind", ["fogilix", "nufasun"])
def test_weights_of_other_sizes_types_and_places_are_not_covered(kind):
    """The constants of the modules size the workspace, so weights of other sizes stay with the operators, which go by the weights."""
    def wider(model):
        mlp = model.layers[0].mlp
        for name, dim in (("gate", 0), ("up", 0), ("gate_b", 0), ("up_b", 0), ("down", 1)):
            if name in mlp._parameters:
                p = mlp._parameters[name]
                setattr(mlp, name, torch.nn.Parameter(torch.cat([p.data, p.data], dim)))

    def deeper(model):
        model.layers[0].mix.o = torch.nn.Parameter(torch.zeros(144, 8).bfloat16())

    def float32(model):
        model.layers[1].mix.q.data = model.layers[1].mix.q.data.float()

    def transposed(model):
        model.embed.data = model.embed.data.t().contiguous().t()

    def elsewhere(model):
        model.layers[0].mix.q = torch.nn.Parameter(model.layers[0].mix.q.data.to("meta"))

    for change in ((wider,) if kind == "nufasun" else ()) + (deeper, float32, transposed, elsewhere):
        model = _decoder(kind)
        assert _is_stock(model)
        before = parameter_tags(model, structure=True)
        change(model)
        assert not _is_stock(model), change
        assert parameter_tags(model, structure=True) != before


@pytest.mark.parametrize("make", [_gpt, lambda: _decoder("fogilix"), lambda: _decoder("nufasun")])
def test_a_model_with_a_table_can_be_copied_and_saved(make):
    model = make()
    model._operand._slots[("pass",)] = ("tags", passes.Table((passes.Sublayer * 2)(), []))
    model._operand._slots[("gpt pass", True)] = ("tags", passes.Table((passes.GptBlock * 2)(), []))
    file = io.BytesIO()
    torch.save(model, file)
    file.seek(0)
    for other in (copy.deepcopy(model), pickle.loads(pickle.dumps(model)), torch.load(file, weights_only=False)):
        assert other._operand is not model._operand and not other._operand._slots and len(model._operand._slots) == 2
        assert all(torch.equal(a, b) and a.data_ptr() != b.data_ptr() for a, b in zip(model.parameters(), other.parameters()))


def test_a_model_saved_by_an_earlier_version():
    """Its caches came with slots and without a count, its feed-forwards without a width."""
    model = _decoder("fogilix")
    for m in model.modules():
        if "_operand" in m.__dict__:
            cache = object.__new__(type(m._operand))
            cache.__dict__["_slots"] = {}
            m._operand = cache
    assert not hasattr(model.layers[0].mlp, "ff")
    tags = parameter_tags(model, structure=True)
    assert _is_stock(model)
    model.refresh_operands()
    assert parameter_tags(model, structure=True) != tags


def test_functions_that_are_not_the_packages_own(monkeypatch):
    gpt, fogilix = _gpt(), _decoder("fogilix")
    pairs, subs = [m for b in _blocks(gpt) for m in b], [s for layer in fogilix.layers for s in (layer.mix, layer.mlp) if s is not None]
    assert passes.own(pairs) and passes.own(subs) and not passes.own([torch.nn.Identity()])
    for model, module, name, others in ((gpt, pairs[2], "forward_folded", pairs), (gpt, pairs[1], "forward", pairs), (fogilix, subs[0], "prompt", subs),
                                        (fogilix, subs[1], "_stacked", subs)):
        before = parameter_tags(model, structure=True)
        setattr(module, name, lambda *args, **kwargs: None)
        assert not passes.own(others) and parameter_tags(model, structure=True) != before
        assert model is gpt or not _is_stock(model)
        delattr(module, name)
        assert passes.own(others) and parameter_tags(model, structure=True) == before
    kind, before = type(subs[0]), parameter_tags(fogilix, structure=True)
    subs[0].__class__ = type("Other", (kind,), {"prompt": lambda *args: None})
    assert not passes.own(subs) and not _is_stock(fogilix) and parameter_tags(fogilix, structure=True) != before
    subs[0].__class__ = kind
    assert _is_stock(fogilix)
    for owner, name in ((K, "linear"), (K, "fused_ffn"), (FusedAttention, "decode"), (mixers.LightningAttention, "_mix"), (mixers._Sublayer, "_stacked")):
        with monkeypatch.context() as m:
            m.setattr(owner, name, lambda *args, **kwargs: None)
            assert not passes.unchanged()
        assert passes.unchanged()


def test_blocks_of_other_kinds_run_their_own_code():
    """In front of anything that needs the GPU."""
    for change in ("container", "block"):
        model = _gpt()
        if change == "container":
            model.blocks[1].__class__ = type("Pair", (torch.nn.Sequential,), {})
        else:
            model.blocks[1][0].__class__ = type("Other", (FusedAttention,), {})
        assert passes.gpt_body(model, torch.zeros((1, 4), dtype=torch.int64), None, None, FusedAttention, type(model.blocks[0][1])) is None


@pytest.mark.parametrize("dtype,folded,aligned,per_value", [("float16", 1, 1, 10), ("bfloat16", 0, 1, 10), ("float32", 0, 1, 18), ("float32", 0, 0, 28)])
def test_workspace_of_a_gpt_pass(dtype, folded, aligned, per_value):
    """What the operators hold at a time beside the result, in bytes per row and column of the stream (of which the result has one value):
    16 bits: the stream 2, the feed-forward's middle 8 (with the result 12); float32 with operands as fp16: stream 4, q | k | v 12, attention's
    output 2 (22); with products that convert their rows: stream 4, middle 16, converted 8 (32)."""
    from gpt_triton_b200._lib import dtype_code

    B, L, H = 16, 300, 768
    blocks = (passes.GptBlock * 2)()
    for i, b in enumerate(blocks):
        b.qkv_bias = b.up_bias = 4096 if aligned or i == 0 else 4100
    args = passes.GptPassArgs(blocks=ctypes.addressof(blocks), out=4096, n_blocks=2, heads=12, B=B, L=L, V=100, P=512, H=H, eps=1e-5,
                              dtype=dtype_code(getattr(torch, dtype)), folded=folded)
    need = passes._passes.b200_gpt_pass_workspace_bytes(ctypes.byref(args))
    statistics = B * L * (8 + 64 * 2 + 8 * (H // 64 + 1)) if folded else 0
    assert per_value * B * L * H <= need <= per_value * B * L * H + statistics + 8 * 256


def test_structures_are_those_of_the_header():
    """Names, order and kinds of the fields, which the libraries compare by size only."""
    from conftest import ROOT

    text = re.sub(r"/\*.*?\*/", "", open(os.path.join(ROOT, "include", "b200_passes.h")).read(), flags=re.S)
    declared = {name: body for body, name in re.findall(r"typedef struct \{(.*?)\} (\w+);", text, flags=re.S)}
    kinds = {"int64_t": ctypes.c_int64, "int": ctypes.c_int, "float": ctypes.c_float}
    for name, ours in (("b200_gpt_block", passes.GptBlock), ("b200_gpt_pass_args", passes.GptPassArgs), ("b200_sublayer", passes.Sublayer),
                       ("b200_decoder_pass_args", passes.DecoderPassArgs)):
        fields = []
        for line in declared.pop(name).split(";"):
            first, *others = [part.strip() for part in line.split(",")]
            if not first:
                continue
            kind = first.replace("const", "").split()[0].rstrip("*")
            for part in (first, *others):
                ident, length = re.search(r"(\w+)(?:\[(\d+)\])?$", part).groups()
                plain = ctypes.c_void_p if "*" in part else kinds[kind]
                fields.append((ident, plain * int(length) if length else plain))
        assert fields == list(ours._fields_), name
    assert not declared and f"#define B200_PASSES_VERSION {passes.VERSION}\n" in text
    assert passes._passes.b200_passes_version() == passes.VERSION


@pytest.mark.parametrize("kind,fields", [(passes.DENSE, {"ff": 96}), (passes.GATED, {"ff": 96}), (passes.LIGHTNING, {"heads": 4, "dim": 16, "vdim": 24}),
                                         (passes.DELTA, {"heads": 4, "kv_heads": 2, "dim": 16, "vdim": 24, "conv_cols": 160, "taps": 4})])
def test_an_output_product_of_another_depth_is_refused(kind, fields):
    sub = (passes.Sublayer * 1)()
    sub[0].kind, sub[0].k_out, sub[0].n_in = kind, 96, 192
    for name, value in fields.items():
        setattr(sub[0], name, value)
    args = passes.DecoderPassArgs(subs=ctypes.addressof(sub), n_subs=1, B=1, n=5, V=10, W=64, ld_out=64, both_norms=int(kind in (passes.DELTA, passes.GATED)))
    assert passes._passes.b200_decoder_pass_workspace_bytes(ctypes.byref(args)) > 0
    sub[0].k_out = 104
    assert passes._passes.b200_decoder_pass_workspace_bytes(ctypes.byref(args)) == 0
    args.ids = args.table = args.out = args.sumsq_out = args.workspace = 4096
    assert passes._passes.b200_decoder_pass(ctypes.byref(args), None) == 1


def test_tags_of_models_that_are_no_modules():
    """A session's model offers `parameters()`; it need not be an nn.Module."""
    class Model:
        def __init__(self):
            self.weights = [torch.zeros(3), torch.ones(2, 2)]

        def parameters(self):
            return iter(self.weights)

    model = Model()
    before = parameter_tags(model)
    assert len(before) == 2 and parameter_tags(model) == before
    model.weights[1].add_(1)
    assert parameter_tags(model) != before
    holder = torch.nn.Module()
    holder._modules["part"] = model
    assert len(parameter_tags(holder)) == 2
