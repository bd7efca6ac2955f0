"""The decode operator's two forms for short contexts are made together, before either is needed a second time."""
import ctypes as C
import threading

import pytest
import torch

from blockgtq_b200 import _lib, attention, layer

SEGS = [[3, 0, 128, 0, 0, 0]]
MERGING, NARROW, PD = _lib.DEC_NARROW | 8 << _lib.DEC_CLUSTER_SHIFT, _lib.DEC_NARROW, _lib.DEC_PROGRAMMATIC


@pytest.fixture
def operator(monkeypatch):
    """call(tokens, ...) -> the flags of the plan that was passed on; ``made``: flags of the plans made, with their threads."""
    made, passed = [], []
    make = layer.make_decode_plan

    def make_plan(desc, n_kv, flags, device, **kw):
        made.append((flags, threading.get_ident()))
        return make(desc, n_kv, flags, device, **kw)

    class Host:
        def attend(self, plan, *args):
            passed.append(plan)
            return None, None, None

    monkeypatch.setattr(attention, "make_decode_plan", make_plan)
    def forms(B, n_kv, T, *shape):
        split = NARROW if T <= 9000 else 0
        return MERGING if T <= 3000 else split, split, MERGING

    monkeypatch.setattr(attention, "growing_forms", forms)
    monkeypatch.setattr(_lib, "host", lambda: Host())

    def call(T, lut, row=48):
        cb = torch.arange(8).half()
        q, kn, vn = (torch.zeros(*s, dtype=torch.float16) for s in ((1, 4, 1, 128), (1, 1, T, 1), (1, 1, T)))
        kp = torch.zeros(1, 1, T, row, dtype=torch.uint8)[..., :48]
        attention.fused_blockgtq_decode_attention(q, kp, kn, cb, None, None, SEGS, kp, vn, lut, v_bits=3)
        lt = attention._layer_for(SEGS, cb, lut, 3, 1, torch.device("cpu"))
        return next(f for f, e in lt._plans.items() if C.addressof(e[0]) == passed[-1])

    return call, made


@pytest.mark.parametrize("first", [100, 5000])
def test_a_context_that_grows_compiles_nothing_on_its_way(operator, first):
    call, made = operator
    lut = torch.full((8,), float(first)).half()         # (tables of its own)
    want = {100: MERGING | PD, 5000: NARROW | PD, 9500: PD}
    assert call(first, lut) == want[first]
    assert sorted(f for f, _ in made) == sorted([NARROW | PD, MERGING | PD])
    for T in (100, 5000, 100):
        assert call(T, lut) == want[T] and len(made) == 2
    assert call(9500, lut) == want[9500] and len(made) == 3          # the wide tile, as long contexts always did


def test_under_capture_only_what_is_there(operator, monkeypatch):
    call, made = operator
    lut = torch.full((8,), 7.0).half()
    assert call(9500, lut) == PD
    monkeypatch.setattr(attention, "_capturing", lambda lt: True)
    assert call(100, lut) == NARROW | PD            # (which has to be there on a GPU)


def test_padded_rows_take_the_split_form(operator):
    call, made = operator
    lut = torch.full((8,), 9.0).half()
    assert call(100, lut, row=96) == MERGING | PD
    assert call(100, lut, row=97) == NARROW | PD and len(made) == 2
