"""How a launcher's arguments reach it: every integer, pointer and float in its place, natively and by ctypes."""

import ctypes
import random

import pytest

from lite_lang_b200.csrc import build

_KINDS = {"int": ctypes.c_int, "long": ctypes.c_long, "pointer": ctypes.c_void_p, "float": ctypes.c_float}


def _calls():
    native = build._native_call()
    yield "ctypes", lambda f, args: build._by_ctypes(f, args)
    if native is not None:
        yield "native", lambda f, args: native(ctypes.cast(f, ctypes.c_void_p).value, *args)


@pytest.mark.parametrize("seed", range(8))
def test_arguments_reach_a_launcher(seed):
    rng = random.Random(seed)
    kinds = [rng.choice(("int", "long", "pointer", "pointer", "int")) for _ in range(rng.choice((1, 5, 6, 7, 23, 50)))]
    for _ in range(rng.randint(0, 8)):
        kinds.insert(rng.randint(0, len(kinds)), "float")
    make = {"int": lambda: rng.choice((0, 1, -1, 2 ** 31 - 1, -2 ** 31, True)), "long": lambda: rng.choice((0, -5, 2 ** 62, -2 ** 63)),
            "pointer": lambda: rng.choice((None, 0, 2 ** 47 + 16)), "float": lambda: rng.choice((0.0, -1.5, 2.0 ** 100))}
    args, seen = [make[k]() for k in kinds], []

    def launcher(*got):
        seen.append(got)
        return len(got)

    proto = ctypes.CFUNCTYPE(ctypes.c_int, *(_KINDS[k] for k in kinds))(launcher)
    want = tuple((a or None) if k == "pointer" else a for k, a in zip(kinds, args))
    for name, call in _calls():
        assert call(ctypes.CFUNCTYPE(ctypes.c_int)(ctypes.cast(proto, ctypes.c_void_p).value) if name == "ctypes" else proto,
                    args) == len(args)
        assert seen.pop() == want, name
        wrapped = [_KINDS[k](a) for k, a in zip(kinds, args)]              # objects of ctypes
        if name == "native":
            assert call(proto, wrapped) == len(args) and seen.pop() == want


def test_other_arguments_are_refused():
    native = build._native_call()
    if native is None:
        pytest.skip("launchers are called by ctypes here")
    proto = ctypes.CFUNCTYPE(ctypes.c_int)(lambda: 0)
    address = ctypes.cast(proto, ctypes.c_void_p).value
    for bad in (("x",), ([1],), (1.0,) * 9, (1,) * 59):
        with pytest.raises(TypeError):
            native(address, *bad)
    with pytest.raises(ValueError):
        native(0)
    assert native(address) == 0
