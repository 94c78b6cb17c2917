"""Uniform words of the encryptor's sampling: the library's draws are numpy's, and leave the generator where numpy's leave it."""
import ctypes as C

import numpy as np
import pytest

from cerium_b200 import _capi

WORD = (1 << 64) - 1


def draw(lib, rng, below, count):
    st = rng.bit_generator.state
    at, inc = st["state"]["state"], st["state"]["inc"]
    state, buffered = (C.c_uint64 * 4)(at >> 64, at & WORD, inc >> 64, inc & WORD), (C.c_uint32 * 2)(st["has_uint32"], st["uinteger"])
    out = np.empty(count, dtype=np.uint32)
    lib.check(lib.dll.cerium_pcg64_uniform(state, buffered, below, out.ctypes.data, count))
    st["state"]["state"] = state[0] << 64 | state[1]
    st["has_uint32"], st["uinteger"] = buffered[0], buffered[1]
    rng.bit_generator.state = st
    return out


@pytest.mark.parametrize("below", [1, 2, 3, 1 << 21, 268369921, (1 << 30) - 35, (1 << 31) + 1, (1 << 32) - 1])
def test_words_are_numpys(below):
    lib = _capi.load()      # host code: no device needed
    ours, numpys = np.random.default_rng([below, 5]), np.random.default_rng([below, 5])
    for count in (1, 2, 0, 3, 4, 5, 8, 511, 1023, 1024, 1025, 4099, 65536):     # odd ones leave a half behind
        assert np.array_equal(draw(lib, ours, below, count), numpys.integers(0, below, size=count, dtype=np.uint32)), count
        assert ours.bit_generator.state == numpys.bit_generator.state, count


def test_bad_arguments():
    lib = _capi.load()
    state, buffered, out = (C.c_uint64 * 4)(), (C.c_uint32 * 2)(), np.empty(4, dtype=np.uint32)
    for args in ((None, buffered, 5, out.ctypes.data, 4), (state, None, 5, out.ctypes.data, 4), (state, buffered, 5, None, 4), (state, buffered, 0, out.ctypes.data, 4)):
        with pytest.raises(_capi.CeriumError) as e:
            lib.check(lib.dll.cerium_pcg64_uniform(*args))
        assert e.value.code == _capi.ERR_INVALID
