"""What `Reads` notices of a model's changes between the steps of a recording, without a GPU (engine/recorded.py)."""
import types

import pytest
import torch

import bukuvik_tools
import gegunex_tools
import kasovik_tools
import rulorax_tools
import tilarax_tools
import vobosun_tools
from helpers import TINY_A, TINY_B
from holon_b200.engine import build
from holon_b200.engine.recorded import Reads
from holon_b200.parts.attention import GQA
from holon_b200.parts.linear import Linear
from holon_b200.weights import RandomSource, load_weights
from ref_kernels import RefKernels

DESIGNS = {"qwen3 a": TINY_A, "qwen3 b": TINY_B}
for tools in (rulorax_tools, kasovik_tools, tilarax_tools, vobosun_tools, gegunex_tools, bukuvik_tools):
    DESIGNS |= {f"{tools.__name__[:-6]} {name}": config for name, config in tools.CONFIGS.items()}


class Kernels(RefKernels):
    recordable, counters = True, frozenset(("launches",))

    def __init__(self):
        self.launches, self.switch = 0, "auto"


def made(config=TINY_A, kernels=None):
    built = build(RandomSource(config, seed=3, dtype=torch.float32), dtype="float32", device="cpu", kernels=kernels or Kernels(), page_size=4, max_seqs=2,
                  max_model_len=32, max_step_tokens=32, pages=16)
    return built, Reads.of(*built.runner._read())


def same(built, reads):
    return reads.same(*built.runner._read())


@pytest.mark.parametrize("name", sorted(DESIGNS))
def test_every_design_is_understood(name):
    built, reads = made(DESIGNS[name])
    assert reads is not None and same(built, reads)
    built.ctx.kernels.launches += 7                       # a counter
    assert same(built, reads)
    for _, p in built.model.params():                     # values may change where they are
        if p.tensor is not None and p.tensor.is_floating_point():
            p.tensor.mul_(1.5)
    assert same(built, reads)


def test_weights_that_are_loaded_again():
    """The parameters' tensors stay; what latent attention derives from them does not."""
    built, reads = made(rulorax_tools.CONFIGS["a"])
    source = RandomSource(rulorax_tools.CONFIGS["a"], seed=4, dtype=torch.float32)
    load_weights(built.model, built.model.spec, source.tensors(), torch.float32, "cpu")
    assert not same(built, reads)


def test_weights_swapped_and_swapped_back():
    built, reads = made(rulorax_tools.CONFIGS["a"])
    old = {n: p.tensor for n, p in built.model.params()}
    for _, p in built.model.params():
        p.tensor = p.tensor.clone()
    built.model.finalize()
    assert not same(built, reads)
    for n, p in built.model.params():
        p.tensor = old[n]
    built.model.finalize()
    assert not same(built, reads)                         # (what was derived has been made again)


def test_parameters_are_not_kept_alive():
    import weakref
    built, reads = made()
    p = next(p for n, p in built.model.params() if "down_proj" in n)
    gone = weakref.ref(p.tensor)
    p.tensor = p.tensor.clone()
    assert gone() is None and not same(built, reads)


class Changed(GQA):
    pass


def storage(b):
    next(p for n, p in b.model.params() if "down_proj" in n).tensor.data = torch.zeros(64, 128)


def moved(b):
    t = next(p for n, p in b.model.params() if "down_proj" in n).tensor
    t.set_(torch.zeros_like(t))


def number(b):
    b.model.layers[1].mixer.scale = 0.5


def layer(b):
    b.model.layers[0] = b.model.layers[1]


def forward(b):
    own = b.model.head.forward
    b.model.head.forward = lambda x: own(x)


def attribute(b):
    b.model.layers[0].kept = []


def switch(b):
    b.ctx.kernels.switch = "other"


def wrapped(b):
    b.ctx.kernels.linear = lambda *a: RefKernels.linear(b.ctx.kernels, *a)


def another_class(b):
    b.model.layers[1].mixer.__class__ = Changed


def pages(b):
    b.cache.kv_of_entry = dict(b.cache.kv_of_entry)


def table(b):
    b.cache.groups[0].table_device = b.cache.groups[0].table_device.clone()


def model(b):
    b.runner.model = types.SimpleNamespace(spec=b.model.spec)


@pytest.mark.parametrize("change", [storage, moved, number, layer, forward, attribute, switch, wrapped, another_class, pages, table, model])
def test_changes_are_noticed(change):
    built, reads = made()
    change(built)
    assert not same(built, reads)


def test_a_method_set_on_a_class(monkeypatch):
    built, reads = made()
    own = Linear.forward
    monkeypatch.setattr(Linear, "forward", lambda self, *a, **k: own(self, *a, **k))
    assert not same(built, reads)
    monkeypatch.undo()
    assert same(built, reads)


def test_a_method_that_was_watched_and_put_back():
    built, reads = made()
    k, head = built.ctx.kernels, built.model.head
    own = k.linear, head.forward
    k.linear, head.forward = (lambda *a: own[0](*a)), (lambda x: own[1](x))
    assert not same(built, reads) and Reads.of(*built.runner._read()) is None
    k.linear, head.forward = own
    assert not same(built, reads) and Reads.of(*built.runner._read()) is not None
    k.linear = head.forward                               # (somebody else's)
    assert Reads.of(*built.runner._read()) is None


def test_what_is_not_understood_is_not_recorded():
    built, _ = made()

    def reads():
        return Reads.of(*built.runner._read())

    assert reads() is not None
    forward(built)                                        # a function in a part's place
    assert reads() is None
    del built.model.head.forward
    assert reads() is not None
    built.model.layers[0].mixer.__class__ = Changed       # a class of somebody else's
    assert reads() is None
    built.model.layers[0].mixer.__class__ = GQA
    built.model.layers[0].note = object()
    assert reads() is None
    del built.model.layers[0].note
    wrapped(built)                                        # a kernel table whose calls somebody watches
    assert reads() is None
    del built.ctx.kernels.linear
    assert reads() is not None
    assert made(kernels=RefKernels())[1] is None          # and one that says nothing
