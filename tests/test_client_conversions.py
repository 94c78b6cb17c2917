"""Residues of integer-valued doubles and exact CRT composition, against Python integers (exact: whole numbers, and one
rounding to the nearest double)."""
import numpy as np
import pytest

from cerium_b200 import _capi, params

N = 1 << 16


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


def words(be, a):
    """64-bit patterns of a double array in a backend buffer."""
    return be.to_dev(np.ascontiguousarray(a).view(np.uint64))


@pytest.mark.parametrize("word_bits", [32, 64])
def test_residues(be, word_bits):
    mods = params.reference_primes_28bit(3) if word_bits == 32 else params.ntt_primes_below(50, 2, 16) + params.ntt_primes_below(60, 1, 16)
    ctx = _capi.Context(be.lib, mods, word_bits)
    rng = np.random.default_rng(3)
    v = np.rint(rng.standard_normal(N) * 2.0 ** rng.integers(0, 200, N))
    v[:8] = [0.0, -0.0, 1.0, -1.0, 2.0 ** 53, -(2.0 ** 53 - 1), float(mods[0]), 2.0 ** 1000]
    small = rng.integers(-21, 22, N).astype(np.int32)
    small[0] = -5
    out = be.empty((3, N), np.uint32 if word_bits == 32 else np.uint64)
    dv, ds = words(be, v), be.to_dev(small.view(np.uint32))
    for s in (None, small):
        ctx.residues(be.ptr(out), be.ptr(dv), [0, 1, 2], small=be.ptr(ds) if s is not None else 0)
        got = be.to_host(out)
        for l, q in enumerate(mods):
            want = [(int(x) + (int(s[i]) if s is not None else 0)) % q for i, x in enumerate(v)]
            assert np.array_equal(got[l], np.array(want, dtype=np.uint64))


@pytest.mark.parametrize("limbs", [1, 2, 17, 64, 255])
def test_compose(be, limbs):
    mods = params.reference_primes_28bit(64)[:limbs] if limbs <= 64 else params.ntt_primes_below(30, limbs, 16)
    ctx = _capi.Context(be.lib, mods, 32)
    big = 1
    for q in mods:
        big *= q
    rng = np.random.default_rng(limbs)
    # magnitudes from a few bits up to the whole range, and the values where the rounding or the sign turns
    vals = [int.from_bytes(rng.bytes(240 if limbs <= 64 else 1000), "little") % max(2, big >> int(rng.integers(0, big.bit_length())))
            for _ in range(N if limbs <= 64 else 1024)] * (1 if limbs <= 64 else N // 1024)
    vals = [(-x if i & 1 else x) for i, x in enumerate(vals)]
    vals[:6] = [0, 1, -1, big // 2, -(big // 2), big // 2 - 1]
    if limbs > 2:
        vals[6:10] = [(1 << 53) + 1, (1 << 54) + 3, -((1 << 54) + 2), (1 << 70) + (1 << 17) + 1]
    x = np.stack([np.array([v % q for v in vals], dtype=np.uint32) for q in mods])
    out = be.empty((N,), np.uint64)
    dx = be.to_dev(x)
    _capi.Composer(ctx, range(limbs)).apply(be.ptr(out), be.ptr(dx))
    got = be.to_host(out).view(np.float64)

    def nearest(v):
        v = (v + big // 2) % big - big // 2
        try:
            return float(v)
        except OverflowError:
            return np.inf if v > 0 else -np.inf
    assert np.array_equal(got, np.array([nearest(v) for v in vals]))
