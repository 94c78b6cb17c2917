"""Plaintext multiply-accumulate: every kind of sum (primes of 50, 55 and 60 bits, mixed, 32-bit words), group sizes on both
sides of a launch's, more sources than a sum of doubles holds before it is reduced, absent plaintexts.  Exact against integers."""
import numpy as np
import pytest

from cerium_b200 import params
from tests import parity_cases as pc


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


@pytest.mark.parametrize("bits", [(50,), (55, 50), (60, 50), (28,)])
@pytest.mark.parametrize("n_out,n_src", [(1, 1), (5, 3), (8, 2), (9, 16)])
def test_sums(be, bits, n_out, n_src):
    mods = [params.ntt_primes_below(b, 1, pc.LOGN)[0] for b in bits]
    word_bits = 32 if bits[0] < 32 else 64
    h = pc.Harness(be, word_bits, mods)
    idx = list(range(len(mods)))
    rng = np.random.default_rng(n_out)
    src = [[pc.rand_limbs(rng, mods, idx) for _ in range(n_src)] for _ in range(2)]
    src[0][0] = pc.edge_limbs(mods, idx)
    pts = [pc.edge_limbs(mods, idx) if k % 5 == 0 else None if k % 7 == 3 else pc.rand_limbs(rng, mods, idx) for k in range(n_out * n_src)]
    d_src = [[h.up(s) for s in row] for row in src]
    d_pts = [None if p is None else h.up(p) for p in pts]
    outs = [[h.new(len(idx), pc.N) for _ in range(n_out)] for _ in range(2)]
    h.ctx.plaintext_mac([h.p(o) for o in outs[0]], [h.p(o) for o in outs[1]], [h.p(s) for s in d_src[0]], [h.p(s) for s in d_src[1]],
                        [0 if p is None else h.p(p) for p in d_pts], idx)
    q = np.array(mods, dtype=object)[:, None]
    at = np.concatenate([np.arange(64), pc.N // 2 + np.arange(64), pc.N - 64 + np.arange(64)])  # big integers: a part of the words
    for i in range(n_out):
        for p in range(2):
            want = sum((src[p][j][:, at].astype(object) * pts[i * n_src + j][:, at].astype(object)
                        for j in range(n_src) if pts[i * n_src + j] is not None), np.zeros((len(idx), len(at)), dtype=object)) % q
            assert np.array_equal(h.down(outs[p][i])[:, at].astype(object), want)
