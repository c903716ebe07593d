"""A layer's weights as the native layer loops take them: a C struct of raw handles, made from the layer's dict.

The dict stays the one place where a layer's weights are: before the struct is used, its sources are compared with the dict's
entries and with the handles they hold now, and it is made anew when one was replaced (and refused when one was freed).
"""
from __future__ import annotations

from operator import attrgetter

_handle = attrgetter("h")


class LayerWeights:
    """What `make(layer)` returned, with the entries (and the handles in them) that it was made from.  One look at them costs
    about 1.5 us of host time a layer."""

    __slots__ = ("entries", "tensors", "handles", "struct")

    def __init__(self, layer: dict, keys, make):
        self.entries = tuple(map(layer.get, keys))
        self.tensors = tuple(dict.fromkeys(_tensors(self.entries)))
        self.handles = list(map(_handle, self.tensors))
        self.struct = make(layer)

    def current(self, layer: dict, keys) -> bool:
        return tuple(map(layer.get, keys)) == self.entries and list(map(_handle, self.tensors)) == self.handles


def _tensors(entries):
    """The handles' owners among the entries: tensors and packed payloads, in tuples and in weight objects too."""
    for e in entries:
        if isinstance(e, (tuple, list)):
            yield from _tensors(e)
        elif hasattr(e, "h"):
            yield e
        elif e is not None and not isinstance(e, (int, float, str)):
            yield from _tensors(getattr(e, n, None) for n in ("t", "q", "s", "scale"))


def native_struct(layer: dict, keys, make):
    """The struct of a layer that has one ("native" in the layer), up to date with the layer's entries; None when `make`
    declines what they are now."""
    kept = layer["native"]
    if not kept.current(layer, keys):
        kept = layer["native"] = LayerWeights(layer, keys, make)
    return kept.struct


def fused_from(layer: dict, fused: str, parts) -> bool:
    """Whether layer[fused], one matrix made of several at load time, still stands for them: layer[fused + "_of"] holds the
    entries that it was made from."""
    made_of = layer.get(fused + "_of")
    return layer.get(fused) is not None and (made_of is None or all(map(_same, map(layer.get, parts), made_of)))


def _same(a, b) -> bool:
    return a is b
