"""The native way to call an entry point (csrc/entry.c) hands every argument over as ctypes does."""
import ctypes
import random

import pytest

from burn_lm_b200.csrc import build

Entry = build.entry_type()
pytestmark = pytest.mark.skipif(Entry is None, reason="no C compiler here: ctypes calls the entry points")


@pytest.mark.parametrize("ints,floats", [(0, 0), (1, 0), (6, 8), (7, 1), (20, 3), (45, 4), (64, 8)])
def test_arguments_arrive(ints, floats):
    rng, seen = random.Random(ints * 10 + floats), []
    kinds = ["i"] * ints + ["f"] * floats
    rng.shuffle(kinds)
    types = {"i": (ctypes.c_int, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_size_t), "f": (ctypes.c_float,)}
    argtypes = [rng.choice(types[k]) for k in kinds]
    back = ctypes.CFUNCTYPE(ctypes.c_int, *argtypes)(lambda *a: seen.extend(a) or 7)
    values = []
    for t in argtypes:
        values.append(rng.choice((-0.5, 1, 3.25)) if t is ctypes.c_float else rng.choice((None, 0x7fff12345678)) if t is ctypes.c_void_p
                      else rng.choice((True, 0, 5)) if t is ctypes.c_int else rng.getrandbits(62))
    call = Entry(ctypes.cast(back, ctypes.c_void_p).value, "".join(kinds))
    assert call(*values) == 7
    assert seen == [v if v is None else type(t().value or 0)(v) if t is ctypes.c_int else v for t, v in zip(argtypes, values)]


def test_results_and_refusals():
    wide = ctypes.CFUNCTYPE(ctypes.c_longlong, ctypes.c_longlong)(lambda v: v)
    at = ctypes.cast(wide, ctypes.c_void_p).value
    assert Entry(at, "i", True)(1 << 40) == 1 << 40 and Entry(at, "i")(-3) == -3
    assert Entry(at, "i")(ctypes.c_longlong(12)) == 12
    for bad in ((), (1, 2), ("x",), (1.5,)):
        with pytest.raises(TypeError):
            Entry(at, "i")(*bad)
    with pytest.raises(ValueError):
        Entry(at, "f" * 9)
