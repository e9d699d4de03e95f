"""Whole passes over a model as one host call (libb200passes.so, declared in include/b200_passes.h).

A pass makes the library calls that the operators of kernels.py make one by one, in the same order and with the same arguments:
the same results, without 15 to 30 us of Python per launch.  What a pass reads of a model (operand and vector addresses) is a table
that is kept with the model's derived operands and rebuilt when a parameter changes; what it reads of a call is passed each time.
Where a model or a call is not what the passes cover, the functions here return None and the caller runs the operators: weights that are
no parameters of their modules, sizes other than the modules' constants, subclasses, replaced functions, hooks that would be called.

So does a pass that is being captured: a replay costs the host the same either way, and graphs of the operators, each with buffers of
its own, replay faster (one sequence of 37 tokens, GPT-2 124M: 398-403 us against 405-415, whatever the workspace's address).

What a pass costs the host, 124M and decoders of width 1024 with 8 layers, operators -> here: GPT-2 fp16 logits 2240 -> 390 us, float32
hidden rows 1810 -> 380, Fogilix prompt 1370 -> 350, Nufasun prompt 1890 -> 500; most of what is left are the launches.  The first pass of a
model, and the first after a change of its weights, runs the operators and costs what they do; the second makes the table.
"""

import ctypes
import operator
import os

import torch
from torch import nn
from torch.nn.modules import module as _nn_module

from . import _lib
from . import kernels as K
from ._lib import c_i64, c_void_p, check, dtype_code, on_device, stream_ptr
from .build import PASSES_PATH
from .module_base import parameter_tags

_F = _lib._fields


class GptBlock(ctypes.Structure):
    """b200_gpt_block of include/b200_passes.h, field for field (as the classes below)."""

    _fields_ = _F("ptr ln1_w ln1_b ln2_w ln2_b qkv qkv_bias qkv_ext proj proj_bias up up_bias up_ext down down_bias; i64 ld_qkv ld_proj ld_up ld_down; ptr kv")


class GptPassArgs(ctypes.Structure):
    _fields_ = _F("ptr blocks ids wte wpe pos_dev out; i64 n_blocks heads B L V P H cache_len; float eps; int dtype folded; ptr workspace; "
                  "i64 workspace_bytes; ptr status_word")


class Sublayer(ctypes.Structure):
    _fields_ = (_F("int kind act; ptr w_in; i64 n_in ld_in") + [("off", c_i64 * 6)]
                + _F("ptr w_out; i64 k_out ld_out; ptr w_mid w_uk w_uv; i64 n_mid ld_mid off_mid; ptr decay norm norm2 sink freq lambda_ conv_w a_log dt_bias "
                     "bias_in bias_out; i64 heads kv_heads dim vdim rank window reach rot_dims taps conv_cols ff source; "
                     "float scale softcap eps out_scale limit alpha q_scale unit_eps; int v_dtype; ptr gain behind shift; int add_embedding"))


LIGHTNING, LATENT, DENSE, DIFFERENTIAL, DELTA, GATED = range(6)


class DecoderPassArgs(ctypes.Structure):
    _fields_ = _F("ptr subs mem0 mem1 ring ids table first_gain final_gain pos_dev out sumsq_out; i64 n_subs B n start V W ld_out; float eps table_scale; "
                  "int both_norms; ptr workspace; i64 workspace_bytes; ptr status_word")


VERSION = 1  # of the structures above (B200_PASSES_VERSION)


def _load():
    if not os.path.exists(PASSES_PATH):
        raise ImportError(f"{PASSES_PATH} is missing: run `python -m gpt_triton_b200.build`")
    _lib.load()  # first: the passes call it
    lib = ctypes.CDLL(PASSES_PATH)
    sizes = (c_i64 * 4)()
    if hasattr(lib, "b200_passes_struct_bytes"):
        lib.b200_passes_struct_bytes(sizes)
    if list(sizes) != [ctypes.sizeof(c) for c in (GptBlock, GptPassArgs, Sublayer, DecoderPassArgs)] or lib.b200_passes_version() != VERSION:
        raise ImportError(f"{PASSES_PATH} was built from another version of include/b200_passes.h: run `python -m gpt_triton_b200.build`")
    for name, args in (("b200_gpt_pass", GptPassArgs), ("b200_decoder_pass", DecoderPassArgs)):
        size, run = getattr(lib, name + "_workspace_bytes"), getattr(lib, name)
        size.restype, size.argtypes = c_i64, [ctypes.POINTER(args)]
        run.restype, run.argtypes = ctypes.c_int, [ctypes.POINTER(args), c_void_p]
    return lib


_passes = _load()


class Table:
    """What a pass reads of a model, and the tensors whose addresses stand in it."""

    __slots__ = ("entries", "tensors", "extra")

    def __init__(self, entries, tensors, **extra):
        self.entries, self.tensors, self.extra = entries, tensors, extra


def table_of(model, key, build):
    """`build()` (a Table, or None: not covered) kept with the model's derived operands until a parameter, a module or a cache of
    derived operands in it changes.  The first call after such a change gets None: it derives the operands between the launches that
    read them, while a table would have them all in front of the first launch (0.5 to 1.8 ms of a first pass)."""
    slots = model._operand._slots
    slot = slots.get(key)
    if slot is None:
        slots[key] = (None, None)
        return None
    tags = parameter_tags(model, structure=True)
    if slot[0] is None:
        slot = slots[key] = (tags, build())
    elif slot[0] != tags:
        slots[key] = (None, None)
        return None
    return slot[1]


_replaced = {}  # owner -> (its namespace, reads the names out of it, the functions): what a pass runs in the place of
_methods = {}  # class of a module -> the names of its functions


def stands_for(owner, *names):
    """Passes run in the place of the functions `names` of kernels.py, or of all functions of a module's class."""
    places = [(owner, names)]
    if isinstance(owner, type):
        places = [(c, [n for n, f in vars(c).items() if callable(f)]) for c in owner.__mro__[:owner.__mro__.index(nn.Module)]]
        _methods[owner] = {n for _, names in places for n in names}
    for place, names in places:
        read = operator.itemgetter(*names)
        _replaced[place] = (vars(place), read, read(vars(place)))


def own(modules):
    """Whether modules are of the package's classes exactly, with no function set on an instance (at the making of a table: its tags
    show what changes later)."""
    return all(type(m) in _methods and _methods[type(m)].isdisjoint(m.__dict__) for m in modules)


def unchanged():
    """Whether every function of a class or of kernels.py that a pass would run in the place of is the package's own."""
    return all([read(space) == functions for space, read, functions in _replaced.values()])


stands_for(K, "fused_embeddings", "fused_layer_norm", "fused_ffn", "takes_operand_rows", "operand_ffn", "operand_ffn_residual", "kv_cache_fill", "split_qkv",
           "flash_attention_v1", "attention_decode", "embedding_rms", "linear", "linear_residual", "latent_append", "window_attention", "latent_decode",
           "decayed_attention", "stream_update", "gated_linear", "rotary_append", "pair_attention", "gated_delta")


def _hooked(modules):
    if _nn_module._global_forward_hooks or _nn_module._global_forward_pre_hooks:
        return True
    return any(m._forward_hooks or m._forward_pre_hooks for m in modules)


def _run(name, args, device):
    size, run = getattr(_passes, name + "_workspace_bytes"), getattr(_passes, name)
    with on_device(device):
        need = size(ctypes.byref(args))
        ws = torch.empty((max(need, 256),), device=device, dtype=torch.uint8)
        args.workspace, args.workspace_bytes = ws.data_ptr(), need
        check(run(ctypes.byref(args), stream_ptr(device)), name)


def registered(module, names):
    """Whether the weights `names` of a module are parameters of its own.  Others (computed, or put beside the parameter as pruning does)
    change without a trace that a table's tags would show; the operators read them anew in every pass."""
    return all(module._parameters.get(n) is not None for n in names)


# ----------------------------------------------------------------------------- FusedGPT
def _gpt_table(model, blocks, folded):
    h, wte = model.config.n_embd, model.wte_weight
    heads = blocks[0][0].num_heads
    if h % 8 or h % heads or h // heads not in (16, 32, 64, 128, 256):
        return None
    shapes = ({"layer_norm_weight": (h,), "layer_norm_bias": (h,), "c_attn_weight": (h, 3 * h), "c_attn_bias": (3 * h,), "c_proj_weight": (h, h), "c_proj_bias": (h,)},
              {"layer_norm_weight": (h,), "layer_norm_bias": (h,), "ffn1_weight": (h, 4 * h), "ffn1_bias": (4 * h,), "ffn2_weight": (4 * h, h), "ffn2_bias": (h,)})
    if model.wpe_weight.shape[1] != h or wte.shape[1] != h or not (wte.is_contiguous() and model.wpe_weight.is_contiguous()) or model.wpe_weight.dtype != wte.dtype:
        return None
    for pair in blocks:
        if not own(pair) or pair[0].num_heads != heads:
            return None
        for m, want in zip(pair, shapes):
            if not registered(m, want) or any(tuple(m._parameters[n].shape) != s or m._parameters[n].dtype != wte.dtype or m._parameters[n].device != wte.device
                                              or not m._parameters[n].is_contiguous() for n, s in want.items()):
                return None
    entries, tensors = (GptBlock * len(blocks))(), []
    for entry, (att, mlp) in zip(entries, blocks):
        if folded:
            qkv = att._operand.folded(att.c_attn_weight, att.layer_norm_weight, att.layer_norm_bias, att.c_attn_bias)
            up = mlp._operand.folded(mlp.ffn1_weight, mlp.layer_norm_weight, mlp.layer_norm_bias, mlp.ffn1_bias)
            entry.qkv_ext, entry.up_ext = qkv.ext.data_ptr(), up.ext.data_ptr()
        else:
            qkv, up = att._operand(att.c_attn_weight), mlp._operand(mlp.ffn1_weight)
        proj, down = att._operand(att.c_proj_weight), mlp._operand(mlp.ffn2_weight)
        vectors = {"ln1_w": att.layer_norm_weight, "ln1_b": att.layer_norm_bias, "ln2_w": mlp.layer_norm_weight, "ln2_b": mlp.layer_norm_bias,
                   "qkv_bias": att.c_attn_bias, "proj_bias": att.c_proj_bias, "up_bias": mlp.ffn1_bias, "down_bias": mlp.ffn2_bias}
        for name, p in vectors.items():
            setattr(entry, name, p.data_ptr())
        for name, w in (("qkv", qkv), ("proj", proj), ("up", up), ("down", down)):
            setattr(entry, name, w.data.data_ptr())
            setattr(entry, "ld_" + name, w.data.stride(0))
        tensors += [qkv, proj, up, down, *(p.data for p in vectors.values())]
    return Table(entries, tensors, heads=heads)


def gpt_body(model, ids, kv_caches, pos, attention_type, mlp_type):
    """FusedGPT's blocks over ids (B, L) -> the residual stream (B, L, H); `pos`: a decode step (L = 1)."""
    wte, wpe = model.wte_weight, model.wpe_weight
    if type(model.blocks) is not nn.ModuleList or any(type(b) is not nn.Sequential for b in model.blocks._modules.values()):
        return None
    blocks = [tuple(b._modules.values()) for b in model.blocks._modules.values()]
    if not blocks or any(len(b) != 2 or type(b[0]) is not attention_type or type(b[1]) is not mlp_type or b[0].training or b[1].training for b in blocks):
        return None
    if not unchanged():
        return None
    folded = model._folds()
    if not folded and _hooked(m for b in blocks for m in b):
        return None
    B, L = ids.shape
    if not (ids.is_cuda and ids.dtype == torch.int64 and ids.is_contiguous() and ids.device == wte.device and 0 < B * L and L <= wpe.shape[0]):
        return None
    if torch.cuda.is_current_stream_capturing():
        return None
    table = table_of(model, ("gpt pass", folded), lambda: _gpt_table(model, blocks, folded))
    if table is None:
        return None
    H, heads = model.config.n_embd, table.extra["heads"]
    if pos is not None and (H // heads not in (32, 64, 128) or pos.dtype != torch.int32 or pos.numel() < 2 or pos.device != wte.device):
        return None
    entries, cache_len = table.entries, 0
    if kv_caches is not None:
        cache_len = kv_caches[0].shape[1]
        shape = (B, cache_len, 2 * H)
        if len(kv_caches) != len(blocks) or cache_len < L or any(c.shape != shape or c.dtype != wte.dtype or c.device != wte.device or not c.is_contiguous()
                                                                 for c in kv_caches):
            return None
        entries = type(entries).from_buffer_copy(entries)  # (the table is shared by sessions and threads)
        for entry, cache in zip(entries, kv_caches):
            entry.kv = cache.data_ptr()
    dev = wte.device
    out = torch.empty((B, L, H), device=dev, dtype=wte.dtype)
    args = GptPassArgs(blocks=ctypes.addressof(entries), ids=ids.data_ptr(), wte=wte.data_ptr(), wpe=wpe.data_ptr(), pos_dev=K._ptr(pos), out=out.data_ptr(),
                       n_blocks=len(blocks), heads=heads, B=B, L=L, V=wte.shape[0], P=wpe.shape[0], H=H, cache_len=cache_len, eps=K.LN_EPS,
                       dtype=dtype_code(wte.dtype), folded=int(folded), status_word=K._status_ptr(dev))
    _run("b200_gpt_pass", args, dev)
    return out


# ----------------------------------------------------------------------------- decoders with an fp32 residual stream
def stock(model, norms, layers):
    """Whether a decoder is what a table describes: `norms`: (name, shape) of weights of its own, `layers`: (layer, names of its norms'
    weights), each with a mixer `mix` and a feed-forward `mlp` or None, of the package's own kinds.  Every weight has the shape that the modules' constants give (those
    size the workspace: wider weights would be written past it), the type of the embeddings, and lies where they do."""
    embed, W = model.embed, model.config.width
    weights = [(model, {"embed": (embed.shape[0], W), **dict(norms)})] + [(layer, dict.fromkeys(names, (W,))) for layer, names in layers]
    weights += [(s, s._shapes(W)) for layer, _ in layers for s in (layer.mix, layer.mlp) if s is not None]
    return embed.is_contiguous() and own(m for m, _ in weights[1 + len(layers):]) and all(registered(m, shapes) and all(p.shape == shape and p.dtype == embed.dtype and p.device == embed.device
                                                                       for p, shape in ((m._parameters[n], shapes[n]) for n in shapes))
                                         for m, shapes in weights)


def operand(entry, name, weight):
    """A (N, K) operand into the fields `name`, n_ / ld_ of the same suffix."""
    setattr(entry, "w_" + name, weight.data_ptr())
    setattr(entry, "ld_" + name, max(weight.stride(0), weight.shape[1]))
    if name != "out":
        setattr(entry, "n_" + name, weight.shape[0])


def sections(entry, starts):
    for i, s in enumerate(starts):
        entry.off[i] = s


def decoder_rows(model, ids, ctx, step, table, memories):
    """ids (rows,) -> (rows behind the last norm as written, sums of squares or None); `memories`: one tuple of tensors (or None)
    per sublayer, as its `memory` gave them."""
    embed, extra, subs = model.embed, table.extra, table.entries
    dev, n_subs, T, W = embed.device, len(subs), ids.numel(), embed.shape[1]
    B = ctx.batch
    n = T // B
    out = K._rows_empty(T, W, embed.dtype, dev)
    sumsq = None
    args = DecoderPassArgs(subs=ctypes.addressof(subs), ids=ids.data_ptr(), table=embed.data_ptr(), first_gain=extra.get("first_gain"),
                           final_gain=extra.get("final_gain"), out=out.data_ptr(), n_subs=n_subs, B=B, n=n, V=embed.shape[0], W=W,
                           ld_out=max(out.stride(0), W), eps=extra["eps"], table_scale=extra.get("table_scale", 1.0), both_norms=int(extra["both_norms"]),
                           status_word=K._status_ptr(dev))
    if not extra["both_norms"]:
        cols = _lib.load().b200_linear_slice_cols(T, _lib.BF16)
        sumsq = torch.empty(((W + cols - 1) // cols, T), device=dev, dtype=torch.float32)
        args.sumsq_out = sumsq.data_ptr()
    if step:
        args.pos_dev = ctx.pos.data_ptr()
    else:
        args.start = ctx.start
    keep = None
    if memories is not None:
        keep = ((c_void_p * n_subs)(), (c_void_p * n_subs)(), (c_i64 * n_subs)())
        for i, tensors in enumerate(memories):
            if tensors is not None:
                keep[0][i] = tensors[0].data_ptr()
                if len(tensors) > 1:
                    keep[1][i] = tensors[1].data_ptr()
                keep[2][i] = tensors[0].shape[1 if len(tensors) == 1 else 2]  # (of a ring; unused elsewhere)
        args.mem0, args.mem1, args.ring = (ctypes.addressof(k) for k in keep)
    _run("b200_decoder_pass", args, dev)
    return out, sumsq


def call_ok(model, ids, ctx, step):
    """Whether a call is one the passes cover: bf16, ids and positions where the model is, nothing being captured."""
    embed = model.embed
    dev = embed.device
    if embed.dtype != torch.bfloat16 or not (embed.is_contiguous() and ids.is_cuda and ids.device == dev and ids.dtype == torch.int64 and ids.is_contiguous()):
        return False
    if ids.numel() == 0 or ids.numel() % ctx.batch or torch.cuda.is_current_stream_capturing():
        return False
    if step:
        return ids.numel() == ctx.batch and ctx.cache is not None and ctx.pos.dtype == torch.int32 and ctx.pos.device == dev
    return ctx.cache is not None or ctx.start == 0


def tensor_ok(t, shape, dtype, device):
    """`shape`: a number, or None for any."""
    return (isinstance(t, torch.Tensor) and t.dtype == dtype and t.device == device and t.is_contiguous() and t.dim() == len(shape)
            and all(w is None or w == s for w, s in zip(shape, t.shape)))
