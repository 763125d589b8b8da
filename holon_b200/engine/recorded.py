"""What a recorded step reads, held against what the model is now.

A CUDA graph of a step holds addresses, sizes and numbers as they were when it was recorded, and none of the Python that a step
runs. So a step may be replayed only while running the model's parts again would enqueue the same kernels with the same arguments:
nothing that the parts, their context, the kernel table or the cache hold may have been replaced since, and no part may do anything
else than enqueue kernels. `Reads.of` looks for all of it, and answers None for a model that holds anything it does not understand:
a part whose own class does not say `recordable` (a subclass does not inherit it), a function set on a part or on the kernel table, an
object of an unknown type. `Reads.same` compares what it found with what is there now, by identity: a derived tensor that `finalize` made
again, a number, a list's member, another storage behind a tensor, a method set on a class or an object.
"""
from __future__ import annotations

import dataclasses
import operator
import types
import weakref
from itertools import chain

import torch

from ..parts.base import Param, Part

_PLAIN = frozenset((type(None), bool, int, float, complex, str, bytes, torch.dtype, torch.device, torch.Size))


class _NotUnderstood(Exception):
    pass


def _dead() -> None:
    return None


def _own_method(v, name: str, x) -> bool:
    """Whether `x` is nothing but the method `name` that `v` has from its class (who watches a method and puts it back may leave it on the object)."""
    return isinstance(x, types.MethodType) and x.__self__ is v and x.__func__ is getattr(type(v), name, None)


class Reads:
    """`views`: live views of every dict, list and class that a step reads; `values`: their members when this was made, one after the
    other. Parameters' tensors are held weakly (whoever replaces a model's weights gets the old ones' memory back); what parts
    derived from them is held like everything else until a later step finds it replaced."""

    def __init__(self) -> None:
        self.views, self.values, self.params, self.weak, self.tensors, self.pointers = [], [], [], [], [], []
        self.tables: list[tuple] = []                # (vars, names, how many in all, values) of objects with counters
        self.objects, self.types = [], []            # what declares itself, and the classes it was of
        self.classes: dict[type, None] = {}          # these and their bases
        self._seen: dict[int, object] = {}

    @classmethod
    def of(cls, *roots) -> "Reads | None":
        reads = cls()
        reads.roots = roots
        try:
            for root in roots:
                reads._look(root)
        except _NotUnderstood:
            return None
        for c in reads.classes:
            reads.views.append(vars(c).values())
        reads.values = list(chain.from_iterable(reads.views))
        reads.weak = [weakref.ref(p.tensor) if p.tensor is not None else _dead for p in reads.params]
        reads.pointers = reads._pointers()
        reads._seen = {}
        return reads

    @staticmethod
    def declared(part: Part) -> bool:
        """Whether every part below this one is of a class that says it may be recorded: what can be told without looking further."""
        return vars(type(part)).get("recordable") is True and all(map(Reads.declared, part._children.values()))

    def same(self, *roots) -> bool:
        """Whether these are the roots it was made of and all that they read is as it was."""
        return len(roots) == len(self.roots) and all(map(operator.is_, roots, self.roots)) \
            and all(map(operator.is_, map(type, self.objects), self.types)) \
            and sum(map(len, self.views)) == len(self.values) \
            and all(map(operator.is_, chain.from_iterable(self.views), self.values)) \
            and all(p.tensor is r() for p, r in zip(self.params, self.weak)) and self._pointers() == self.pointers \
            and all(len(d) == n and all(d.get(name, self) is v for name, v in zip(names, values))
                    for d, names, n, values in self.tables)

    def _pointers(self) -> list[int]:
        return [t.data_ptr() for t in self.tensors] + [p.tensor.data_ptr() for p in self.params if p.tensor is not None]

    def _look(self, v) -> None:
        t = type(v)
        if t in _PLAIN or id(v) in self._seen:
            return
        self._seen[id(v)] = v
        if t is tuple:
            for x in v:
                self._look(x)
        elif t is Param:
            if v.tensor is not None and type(v.tensor) is not torch.Tensor:
                raise _NotUnderstood
            self.params.append(v)
        elif t is torch.Tensor:
            self.tensors.append(v)
        elif vars(t).get("recordable") is True:
            self._look_at_object(v)
        elif t is list:
            self.views.append(v)
            for x in v:
                self._look(x)
        elif t is dict:
            self.views.append(v.values())
            for x in v.values():
                self._look(x)
        elif not (dataclasses.is_dataclass(t) and t.__dataclass_params__.frozen):    # (such an object cannot change; its holder is asked
            raise _NotUnderstood                                                     # whether it is still the same)

    def _look_at_object(self, v) -> None:
        self.objects.append(v)
        self.types.append(type(v))
        if type(v) not in self.classes:
            self.classes.update(dict.fromkeys(type(v).__mro__[:-1]))
        counters = getattr(type(v), "counters", None)
        if counters is None:
            held, part = vars(v), isinstance(v, Part)
            self.views.append(held.values())
            for name, x in held.items():
                if type(x) not in _PLAIN and not (part and name in ("_params", "_children")) and not _own_method(v, name, x):
                    self._look(x)                    # (what a step reads of those two it reads by their own names)
            return
        # A kernel table: what it holds decides which kernels it launches, except its counters; nothing in it is walked into
        if any(callable(getattr(type(v), name, None)) and not _own_method(v, name, x) for name, x in vars(v).items()):
            raise _NotUnderstood
        names = tuple(name for name in vars(v) if name not in counters)
        self.tables.append((vars(v), names, len(vars(v)), tuple(vars(v)[name] for name in names)))
