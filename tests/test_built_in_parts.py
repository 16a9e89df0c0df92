"""Which models count as made of the package's own parts only (the 32-bit path captures the steps of those): parts anywhere inside other
parts are looked at, and methods that were replaced on an instance or a class count as foreign."""
import gc
import weakref

import pytest

import infer_b200.models  # noqa: F401  (registers the architectures)
from infer_b200.engine.model import Model
from infer_b200.parts.attention import Attention
from infer_b200.parts.base import CHANGES, Block, Mixer, watch
from infer_b200.parts.linear import Linear
from infer_b200.parts.rmsnorm import RMSNorm
from infer_b200.parts.side_by_side import SideBySide


class Foreign(Mixer):
    pass


class ForeignProduct(Linear):
    pass


def _bare(cls, **attributes):
    part = cls.__new__(cls)
    part.spec = part.rt = None
    for k, v in attributes.items():
        setattr(part, k, v)
    return part


def _model(mixer, block_class=Block):
    model = Model.__new__(Model)
    model.spec = model.rt = None
    model.embedding = model.head = model.final_norm = _bare(RMSNorm)
    model.stream = None
    model.blocks = [block_class(norm=_bare(RMSNorm), mixer=mixer)]
    return model


def _sides(second):
    return _bare(SideBySide, sides={"first": _bare(Attention), "second": second})


def test_own_parts():
    assert _model(_bare(Attention, qkv=_bare(Linear))).built_in()
    assert _model(_sides(_bare(Attention))).built_in()


@pytest.mark.parametrize("mixer", [
    lambda: _bare(Foreign),
    lambda: _sides(_bare(Foreign)),
    lambda: _bare(Attention, more=[_bare(RMSNorm), _bare(Foreign)]),
    lambda: _bare(Attention, more=(({"deep": [_bare(Foreign)]},),)),
    lambda: _sides(_bare(Attention, forward=lambda *a, **k: None)),
    lambda: _bare(Attention, qkv=_bare(ForeignProduct)),
], ids=["itself", "in a dict", "in a list", "deeper", "replaced method", "a foreign product"])
def test_a_foreign_part_anywhere(mixer):
    assert not _model(mixer()).built_in()


def test_a_foreign_block():
    class Mine(Block):
        pass
    assert not _model(_bare(Attention), Mine).built_in()


def test_a_method_replaced_on_a_class_or_a_block(monkeypatch):
    model = _model(_bare(Attention))
    model.blocks[0].forward = lambda *a: None
    assert not model.built_in()
    monkeypatch.setattr(RMSNorm, "forward", lambda *a, **k: None)
    assert not _model(_bare(Attention)).built_in()


def test_parts_that_know_each_other():
    a, b = _bare(Attention), _bare(Attention)
    a.other, b.other = b, a
    assert _model(a).built_in()


def test_looking_at_the_parts_keeps_none_of_them():
    """A model's weights go with the model, without waiting for a collection."""
    collecting = gc.isenabled()
    gc.disable()
    try:
        model = _model(_sides(_bare(Attention)))
        part = weakref.ref(model.blocks[0].mixer.sides["second"])
        assert model.built_in() and len(model.made_of()) > 3
        del model
        assert part() is None
    finally:
        if collecting:
            gc.enable()


def test_containers_that_hold_themselves():
    a = _bare(Attention)
    a.more = [a]
    a.more.append(a.more)
    assert _model(a).built_in()


def test_only_what_is_watched_is_counted():
    """The parts of other models, a model that is being built and one whose steps nobody keeps cost and count nothing."""
    model, other = _model(_sides(_bare(Attention))), _model(_bare(Attention))
    before = model.made_of()
    watch(before[::3])
    n = CHANGES[0]
    other.blocks[0].mixer.scale = 2.0
    _model(_bare(Attention, qkv=_bare(Linear)))
    assert CHANGES[0] == n and len(model.made_of()) == len(before)
    model.blocks[0].mixer.sides["second"].scale = 2.0
    model.blocks[0].extra = 1
    del model.blocks[0].extra
    model.final_norm = _bare(RMSNorm)
    assert CHANGES[0] == n + 4
