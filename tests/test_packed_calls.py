"""The argument blocks of the packed calls: every field arrives in its place, and values that do not pack go
argument by argument as before (no GPU: the library's own argument checks answer)."""
import ctypes as C

import numpy as np
import pytest

from conftest import pulpnn

api = pulpnn.api


def test_every_argument_arrives(monkeypatch):
    """A C callback in the place of the entry point sees the arguments as the caller wrote them."""
    lib = pulpnn.load_library()
    seen = []
    kinds = [C.c_void_p] * 7 + [C.c_uint16] * 16 + [C.c_int] * 2
    entry = C.CFUNCTYPE(None, *kinds)(lambda *a: seen.append(a))
    f = lib.pulpnn_packed_conv_bn32
    proto = C.CFUNCTYPE(C.c_int, C.c_void_p, C.c_char_p)
    args = list(range(1001, 1008)) + list(range(11, 27)) + [-1, 7]
    block = api._Packed("conv", "=7Q16H2i", "x").pack(*args)
    assert proto(C.cast(f, C.c_void_p).value)(C.cast(entry, C.c_void_p), block) == 0
    assert list(seen[0]) == args
    seen.clear()
    kinds = [C.c_void_p] * 8 + [C.c_uint16] * 16 + [C.c_int8] * 2
    entry = C.CFUNCTYPE(None, *kinds)(lambda *a: seen.append(a))
    args = list(range(1001, 1009)) + list(range(11, 27)) + [-1, 7]
    block = api._Packed("depthwise", "=8Q16H2b", "x").pack(*args)
    assert proto(C.cast(lib.pulpnn_packed_depthwise_bn64, C.c_void_p).value)(C.cast(entry, C.c_void_p), block) == 0
    assert list(seen[0]) == args


def test_what_does_not_pack_is_not_taken():
    add = api._Packed("add", "=3Q6H")
    assert add(32, 0, 0, 0, 65536, 1, 0, 4, 4, 16) is False        # ctypes cuts it to 0
    assert add(32, 0, 0, 0, 1.5, 1, 0, 4, 4, 16) is False          # ctypes refuses it
    assert add(32, 0, 0, 0, None, 1, 0, 4, 4, 16) is False
    a = np.zeros(16, np.uint8)
    with pytest.raises(TypeError):
        api.pulp_nn_add(32, a, a, a, 1.5, 1, 0, 1, 1, 16)
    with pytest.raises(TypeError):
        api.pulp_nn_add(32, a, a, "text", 1, 1, 0, 1, 1, 16)
    with pytest.raises(ValueError):
        api.pulp_nn_add(16, a, a, a, 1, 1, 0, 1, 1, 16)
    with pytest.raises(AssertionError):
        api.pulp_nn_add(32, a[::2], a, a, 1, 1, 0, 1, 1, 16)
