"""What an attention call hands to the library by address is alive until the library returns."""
import copy
import ctypes as C
import threading
import weakref

import pytest
import torch

from blockgtq_b200 import _lib, attention, layer

SEGS = [[3, 0, 128, 0, 0, 0]]
B, N_KV, GQA, T = 1, 2, 2, 5


class _Host:
    """Stands in for the native calls: `attend` records what is alive, and does nothing else."""

    def __init__(self, watched):
        self.watched, self.alive = watched, None

    def attend(self, *args):
        self.alive = [r() is not None for r in self.watched]
        return None, None, None


def _args():
    q = torch.zeros(B, N_KV * GQA, 1, 128, dtype=torch.float16)
    kp, vp = (torch.zeros(B, N_KV, T, 48, dtype=torch.uint8) for _ in range(2))
    kn, vn = torch.ones(B, N_KV, T, 1, dtype=torch.float16), torch.ones(B, N_KV, T, dtype=torch.float16)
    cb = lut = torch.arange(8).half()
    return q, kp, kn, cb, None, None, SEGS, vp, vn, lut


@pytest.mark.parametrize("shape,dtype,step", [((128, 128), torch.float32, 1), ((N_KV, 128, 128), torch.float16, 1),
                                              ((N_KV, 128, 128), torch.float32, 2)])
def test_a_converted_rotation_outlives_the_call(monkeypatch, shape, dtype, step):
    """One matrix for all heads, another type, another layout: each makes a tensor that only the call holds."""
    made = []
    rotation = attention._rotation

    def watch(*args):
        r = rotation(*args)
        made.append(weakref.ref(r))
        return r

    host = _Host(made)
    monkeypatch.setattr(attention, "_rotation", watch)
    monkeypatch.setattr(attention, "growing_forms", lambda *shape: (0, 0, 0))
    monkeypatch.setattr(_lib, "host", lambda: host)
    rot = torch.ones(*shape[:-1], shape[-1] * step, dtype=dtype)[..., ::step]
    attention.fused_blockgtq_decode_attention(*_args(), v_bits=3, v_rotation=rot)
    assert len(made) == 1 and made[0]() is None         # (it was a temporary)
    assert host.alive == [True]


def test_rotation_and_status_passed_as_temporaries(monkeypatch):
    q, kp, kn, cb, _, _, _, vp, vn, lut = _args()
    lt = attention._layer_for(SEGS, cb, lut, 3, N_KV, torch.device("cpu"))
    watched = []

    def temporary(*shape, dtype):
        t = torch.zeros(*shape, dtype=dtype)
        watched.append(weakref.ref(t))
        return t

    host = _Host(watched)
    monkeypatch.setattr(_lib, "host", lambda: host)
    layer.attend(lt, q, kp, kn, vp, vn, 0, T, rotate=False, v_rot=temporary(N_KV, 128, 128, dtype=torch.float32),
                 status=temporary(1, dtype=torch.int32))
    assert host.alive == [True, True]


class _Calls:
    def __init__(self):
        self.plans = []

    def attend(self, plan, *args):
        self.plans.append(plan)
        return None, None, None


def _layer(kind):
    if kind == "operator":
        return attention._AdHocLayer(SEGS, [0] * 8, [0] * 8, 3, N_KV, (128, 0), torch.device("cpu"))
    from helpers import tables_for
    return layer.LayerTables(*zip(*[tables_for("a3_1to8", h) for h in range(N_KV)]), "cpu")


@pytest.mark.parametrize("kind", ["operator", "layer"])
def test_threads_making_the_first_call_share_one_plan(monkeypatch, kind):
    """Each of four threads makes a plan of its own; one of them is kept, and every call passes that one on."""
    n = 4
    together, host, make = threading.Barrier(n), _Calls(), layer.make_decode_plan

    def make_at_once(*args, **kwargs):
        together.wait(60)
        made = make(*args, **kwargs)
        together.wait(60)
        return made

    for module in (layer, attention):
        monkeypatch.setattr(module, "make_decode_plan", make_at_once)
    monkeypatch.setattr(_lib, "host", lambda: host)
    lt = _layer(kind)
    q, kp, kn, *_, vp, vn, _ = _args()

    def call():
        layer.attend(lt, q, kp, kn, vp, vn, 0, T, rotate=False)

    for _ in range(2):
        threads = [threading.Thread(target=call) for _ in range(n)]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    assert len(host.plans) == 2 * n and len(lt._plans) == 1
    assert set(host.plans) == {C.addressof(lt.plan(_lib.DEC_PROGRAMMATIC))}


def test_a_copied_layer_passes_its_own_plan(monkeypatch):
    host = _Calls()
    monkeypatch.setattr(_lib, "host", lambda: host)
    lt = _layer("layer")
    q, kp, kn, *_, vp, vn, _ = _args()
    for x in (lt, copy.deepcopy(lt)):
        for _ in range(2):
            layer.attend(x, q, kp, kn, vp, vn, 0, T, rotate=True)
        assert set(host.plans) == {C.addressof(x.plan(_lib.DEC_PROGRAMMATIC))}
        host.plans.clear()
    twin = copy.deepcopy(lt)        # (with its plans made)
    layer.attend(twin, q, kp, kn, vp, vn, 0, T, rotate=True)
    assert host.plans == [C.addressof(twin.plan(_lib.DEC_PROGRAMMATIC))] != [C.addressof(lt.plan(_lib.DEC_PROGRAMMATIC))]
