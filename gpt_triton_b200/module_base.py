"""What the model modules of this package share: derived-operand caching and the eval-only base class."""

from torch import nn

from . import kernels as K


class _OperandCache:
    """Derived operands (PackedWeight and friends) per parameter; rebuilt when the parameter is replaced, cast,
    moved or written in place.  The tag uses the Parameter's own ``_version``, which ``load_state_dict``,
    ``param.copy_`` and optimizer steps bump (``param.data`` is a fresh tensor object whose counter always reads 0,
    so it cannot serve).  Writes made *through* ``param.data`` (``param.data.mul_(2)``) bump no counter torch
    exposes: after such a write call ``refresh_operands()`` on the model."""

    cleared = 0  # times; what is derived from these operands elsewhere goes with them (of the class: files of earlier versions have none)

    def __init__(self):
        self._slots = {}

    def __reduce__(self):
        """A copied or pickled model starts without: everything here can be derived again, and what holds addresses (passes.Table) would
        name the original's operands."""
        return type(self), ()

    def clear(self):
        self._slots.clear()
        self.cleared += 1

    @staticmethod
    def _tag(param):
        return (param.data_ptr(), param._version, param.dtype, param.device, param.shape)

    def derived(self, key, params, make):
        """`make()` cached under `key` until one of `params` changes."""
        tag = tuple(self._tag(p) for p in params)
        slot = self._slots.get(key)
        if slot is None or slot[0] != tag:
            slot = (tag, make())
            self._slots[key] = slot
        return slot[1]

    def __call__(self, param, weight_is_nk=False):
        return self.derived(("packed", id(param), weight_is_nk), (param,),
                            lambda: K.pack_weight(param.data.contiguous(), weight_is_nk=weight_is_nk))

    def folded(self, weight, ln_weight, ln_bias, bias):
        """FoldedWeight of `weight` with the LayerNorm (ln_weight, ln_bias) in front of it and `bias` behind."""
        return self.derived(("folded", id(weight)), (weight, ln_weight, ln_bias, bias),
                            lambda: K.fold_layer_norm(weight.data.contiguous(), ln_weight.data.contiguous(), ln_bias.data.contiguous(),
                                                      bias.data.contiguous()))


_PLAIN = {int, float, str, tuple, type(None)}


def parameter_tags(module, structure=False):
    """What tells whether a parameter of `module` or of one below it was replaced, cast, moved or written in place: equal lists, no
    change.  With `structure` also whether one was renamed, added or taken away (a weight that is pruned, say, is no parameter any more), a
    module exchanged, one of its constants set, an attribute (a function, say) set on one below, or derived operands dropped.  (A walk
    over the module tree's own dictionaries: Module.parameters() takes 3 us per parameter, as long as a launch.)"""
    tags, stack = [], [module]
    while stack:
        m = stack.pop()
        d = m.__dict__
        params = d.get("_parameters")
        if params is None:  # (a model, or a part of one, that is no nn.Module or keeps its parameters elsewhere)
            tags += [(p.data_ptr(), p._version, p.dtype, p.device, p.shape) for p in m.parameters()]
            continue
        if structure:
            cache = d.get("_operand")
            if cache is not None:
                tags.append((cache.cleared, d.get("config"), [v for v in d.values() if v.__class__ in _PLAIN]))
            tags += (m.__class__, m is module or len(d), *params)
            # (the device goes with the address)
            tags += [(p.data_ptr(), p._version, p.dtype, p.shape) for p in params.values() if p is not None]
        else:
            tags += [(p.data_ptr(), p._version, p.dtype, p.device, p.shape) for p in params.values() if p is not None]
        stack.extend([c for c in d["_modules"].values() if c is not None])
    return tags


class _EvalOnly(nn.Module):
    def _check_eval(self):
        if self.training:
            raise NotImplementedError("libb200gpt implements the forward/eval path only: call .eval() first")

    def refresh_operands(self):
        """Drop every cached derived operand (packed weights) of this module and its children; the next forward
        rebuilds them from the parameters.  Needed only after writes through ``param.data``, which torch's version
        counters do not see; ``load_state_dict``, ``copy_``, casts and moves are noticed without it."""
        for m in self.modules():
            cache = getattr(m, "_operand", None)
            if isinstance(cache, _OperandCache):
                cache.clear()
