"""The native calls take their numbers as Python takes them: one that is no number, or does not fit, is an exception."""
import pytest
import torch

from blockgtq_b200 import _lib

X3, X4 = torch.zeros(1, 4, 128, dtype=torch.float16), torch.zeros(1, 1, 4, 128, dtype=torch.float16)
U8, N3 = torch.zeros(1, 1, 4, 48, dtype=torch.uint8), torch.zeros(1, 1, 4, dtype=torch.float16)
CALLS = {       # function: (arguments, {position: kind of number})
    "layer_step": ([0, 0, X4, X4, X4, None, None], {0: "ptr", 1: "i32"}),
    "layer_encode": ([0, 0, X4, X4, 0, 0], {0: "ptr", 1: "i32", 4: "i32", 5: "i32"}),
    "encode": ([0, 0, 0, 1, 48, X4, X4, 0, U8, X4, U8, N3, 0], {0: "ptr", 1: "ptr", 2: "ptr", 3: "i32", 4: "i32", 7: "i32", 12: "i32"}),
    "compress": ([0, 0, 1, X3, 48, 0, 0], {0: "ptr", 1: "ptr", 2: "i32", 4: "i32", 5: "i32", 6: "i32"}),
    "attend": ([0, 0, None, X3, U8, X4, U8, N3, 0, 4, 1, 1.0, None, None, None, False, False, None, 1],
               {0: "ptr", 1: "ptr", 2: "ptr", 8: "i32", 9: "i32", 10: "i32", 11: "real", 12: "ptr", 15: "truth", 16: "truth", 17: "ptr",
                18: "i32"}),
    "rotate_rows": ([0, 0, 1, X4], {0: "ptr", 1: "ptr", 2: "i32"}),
    "prefill": ([0, 1, X4, U8, X4, U8, N3, 4, 0, True, 1.0, 0, None, 1 << 40],
                {0: "ptr", 1: "i32", 7: "i32", 8: "i32", 9: "truth", 10: "real", 11: "i32", 12: "ptr", 13: "i64"}),
}


class NoTruth:
    def __bool__(self):
        raise ValueError("no truth")


@pytest.mark.parametrize("name", list(CALLS))
def test_bad_numbers_raise(name):
    fn = getattr(_lib.host(), name)
    args, numbers = CALLS[name]
    assert fn(*args) is None                     # CPU tensors: left to the Python wrapper
    for i, kind in numbers.items():
        bad = {"truth": [(NoTruth(), ValueError)], "real": [("1.0", TypeError)],
               "i32": [("3", TypeError), (2.0, TypeError), (1 << 40, OverflowError), (-(1 << 31) - 1, OverflowError)],
               "i64": [("3", TypeError), (1 << 70, OverflowError)], "ptr": [("3", TypeError), (-1, OverflowError)]}[kind]
        for value, error in bad:
            with pytest.raises(error):
                fn(*args[:i], value, *args[i + 1:])
    if name == "attend":                          # -1 is a number like any other, but no count of splits
        assert fn(*args[:8], -1, *args[9:]) is None
        assert fn(*args[:10], -1, *args[11:]) == -1


def test_bind_takes_addresses_only():
    with pytest.raises(TypeError):
        _lib.host().bind(*["x"] * 8)
    with pytest.raises(ValueError):
        _lib.host().bind(0)


def test_strides_of_single_heads_and_batches_do_not_matter():
    """Queries in the packed basis have to lie one behind the other; with one head or one batch entry any stride of that
    dim says so.  (A plan without a table image is refused before anything is launched: -1, where strides are -2.)"""
    import ctypes as C
    L, plan = _lib.lib(), _lib.DecodePlan()
    buf = C.create_string_buffer(1 << 16)
    a = (C.addressof(buf) + 255) & ~255

    def attend(B, n_q, sb, sh):
        return L.bgtq_attend(C.addressof(plan), None, None, a, sb, sh, a, 0, 0, 48, a, 0, 0, 2, a, 0, 0, 48, a, 0, 0, 1, B, n_q, 1, 0, 4, 1,
                             1.0, None, None, None, a, a, None, None, None, None)

    assert attend(1, 4, 7, 128) == attend(1, 1, 7, 4096) == attend(3, 1, 128, 4096) == attend(2, 4, 512, 128) == -1
    assert attend(1, 4, 512, 4096) == attend(2, 1, 4096, 128) == attend(2, 4, 1024, 128) == -2


def test_a_preparation_with_nothing_to_do_launches_nothing():
    import ctypes as C
    L = _lib.lib()
    buf = C.create_string_buffer(1 << 12)
    a = (C.addressof(buf) + 255) & ~255

    def prepare(flags, q=None):
        return L.bgtq_step_prepare(a, a, a, q, 0, 128, q, 1, a, 0, 128, a, 0, 128, 1, 1, 0, a, 0, 0, 48, 48, a, 0, 0, 2, 2, a, 0, 0, 48,
                                   a, 0, 0, 1, flags | _lib.ENC_PROGRAMMATIC, None, 4, None, None)

    assert prepare(_lib.ENC_SKIP_K | _lib.ENC_SKIP_V) == 0
    if not torch.cuda.is_available():       # (everything else is launched, and there is nothing to launch on)
        assert prepare(_lib.ENC_SKIP_K) == prepare(_lib.ENC_SKIP_K | _lib.ENC_SKIP_V, a) == -4
