"""What the event brackets around launches see (no GPU needed: events and libraries are stand-ins)."""
import inspect
import re

import pytest
import torch

from cisr_b200.ops import kernels


class Event:
    def __init__(self, enable_timing):
        pass

    def record(self):
        pass


@pytest.fixture
def stand_ins(monkeypatch):
    class Library:
        def __getattr__(self, name):
            return lambda *a: 0

    monkeypatch.setattr(torch.cuda, "Event", Event)
    monkeypatch.setattr(kernels, "_need", lambda *a, **kw: None)
    monkeypatch.setattr(kernels, "_stream", lambda: 0)
    monkeypatch.setattr(kernels, "_skinny", Library)
    monkeypatch.setattr(kernels, "_elementwise", Library)


def test_both_products_of_a_feed_forward_are_seen(stand_ins):
    t = lambda *s: torch.zeros(*s, dtype=torch.bfloat16)
    with kernels.timed_launches() as timed:
        kernels.skinny_mlp(t(4, 64), t(96, 64), t(24, 48))
    assert [(name, shape) for name, shape, *_ in timed.records] == [("skinny_gemm", (4, 96, 64, kernels.EPI_SWIGLU, False)), ("skinny_gemm", (4, 24, 48, kernels.EPI_PLAIN, False))]


def test_every_function_that_launches_is_described():
    source = open(kernels.__file__).read()
    launches = {m.group(1) for f in re.split(r"\n(?=def )", source) for m in [re.match(r"def ([a-z]\w*)", f)] if m and "_check(" in f}
    seen_by_parts = {"skinny_mlp"}                       # as the products it is made of
    not_launches = {"attention_library"}                 # an init call
    assert launches - set(kernels._DESCRIBE) == seen_by_parts | not_launches


def test_a_context_inside_another_leaves_the_outer_one_open(stand_ins):
    x = torch.zeros(4, 8)
    plain = kernels.scale_
    with kernels.timed_launches() as outer:
        kernels.scale_(x, 2.0)
        with kernels.timed_launches() as inner:
            kernels.scale_(x, 2.0)
        kernels.scale_(x, 2.0)
    assert len(outer.records) == 2 and len(inner.records) == 1 and kernels.scale_ is plain
    first, second = kernels.timed_launches(), kernels.timed_launches()
    first.__enter__(), second.__enter__(), first.__exit__()
    kernels.scale_(x, 2.0)
    second.__exit__()
    assert len(second.records) == 1 and not first.records and kernels.scale_ is plain


def test_a_description_takes_every_call_that_its_function_takes():
    for name, describe in kernels._DESCRIBE.items():
        parameters = inspect.signature(kernels._untimed[name]).parameters.values()
        given = [object() for p in parameters if p.kind == p.POSITIONAL_OR_KEYWORD and p.default is p.empty]
        inspect.signature(describe).bind(*given, **{p.name: p.default for p in parameters if p.kind == p.KEYWORD_ONLY or p.default is not p.empty})
