"""Row pass of the raised digits inside the inner product of a key switch: every arithmetic (primes of 60, 51 and 50 bits),
more digits than a sum of doubles holds before it is reduced, and keys that are aligned to 16 bytes only, which take the
separate kernels."""
import numpy as np
import pytest

from cerium_b200 import _capi, params
from tests import parity_cases as pc


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


def _params(word_bits, L, K, dnum):
    if word_bits == 32:
        return pc.small_params(32, L, K, dnum)
    p60 = params.ntt_primes_below(60, K + 1, pc.LOGN)
    q = [p60[0]] + params.ntt_primes_below(51, 1, pc.LOGN) + params.ntt_primes_below(50, L - 2, pc.LOGN)
    return params.CkksParams(pc.LOGN, 64, q + p60[1:], L, K, dnum)


@pytest.mark.parametrize("word_bits,L,K,dnum", [(64, 3, 1, 3), (64, 12, 1, 12), (64, 15, 2, 10), (32, 9, 2, 5)])
@pytest.mark.parametrize("offset", [0, 16])
def test_key_switch(be, word_bits, L, K, dnum, offset):
    prm = _params(word_bits, L, K, dnum)
    h = pc.Harness(be, word_bits, prm.moduli)
    c0, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(dnum), prm)
    if offset == 0:  # the largest key words
        evk[..., ::2] = np.array([prm.moduli[p] - 1 for p in prm.q_idx + prm.p_idx], dtype=np.uint64)[:, None]
    modes = (_capi.BCONV_EXACT, _capi.ROUND_HALF) if word_bits == 64 else (_capi.BCONV_LAZY, _capi.ROUND_FLOOR)
    ks = _capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, dnum, *modes)
    words = offset * 8 // word_bits
    d_evk = h.up(np.concatenate([np.zeros(words, dtype=np.uint64), evk.reshape(-1)]))
    d_c0, d_c1 = h.up(c0), h.up(c1)
    o = h.new(2, L, pc.N)
    second = h.p(o) + L * pc.N * word_bits // 8
    ks.apply(h.p(o), second, h.p(d_c1), h.p(d_evk) + offset)
    assert np.array_equal(h.down(o), np.stack(h.orc.keyswitch(*modes, prm.q_idx, prm.p_idx, dnum, c1, evk)))
    elt = be.lib.galois_elt_from_step(7, pc.LOGN)
    ks.hrot(h.p(o), second, h.p(d_c0), h.p(d_c1), h.p(d_evk) + offset, elt)
    assert np.array_equal(h.down(o), np.stack(h.orc.hrot(*modes, prm.q_idx, prm.p_idx, dnum, elt, c0, c1, evk)))
    # a multiplication: the products of the tensor are taken where they are read
    b0, b1 = (pc.rand_limbs(np.random.default_rng(8 + k), prm.moduli, prm.q_idx) for k in range(2))
    d_b0, d_b1 = h.up(b0), h.up(b1)
    ks.hmult(h.p(o), second, h.p(d_c0), h.p(d_c1), h.p(d_b0), h.p(d_b1), h.p(d_evk) + offset, 0)
    assert np.array_equal(h.down(o), np.stack(h.orc.hmult_relin(*modes, False, prm.q_idx, prm.p_idx, dnum, c0, c1, b0, b1, evk)))
    ks.close()


@pytest.mark.parametrize("bits", [28, 32, 33, 34, 50])
def test_integer_butterflies_of_small_primes(be, monkeypatch, bits):
    """With integer butterflies asked for, 64-bit words of any prime; the sums of products want 34 bits."""
    monkeypatch.setenv("CERIUM_B200_NTT_ARITH", "int")
    L, K = (6, 3) if be.name == "emu" else (20, 7)   # rows for every warp of the device
    mods = params.ntt_primes_below(bits, L + K, pc.LOGN)
    prm = params.CkksParams(pc.LOGN, 64, mods, L, K, 3)
    h = pc.Harness(be, 64, mods)
    c0, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(bits), prm)
    evk[..., ::2] = np.array(mods, dtype=np.uint64)[:, None] - 1
    modes = (_capi.BCONV_EXACT, _capi.ROUND_HALF)
    ks = _capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, 3, *modes)
    d_evk, d_c0, d_c1, o = h.up(evk), h.up(c0), h.up(c1), h.new(2, L, pc.N)
    second = h.p(o) + L * pc.N * 8
    ks.apply(h.p(o), second, h.p(d_c1), h.p(d_evk))
    assert np.array_equal(h.down(o), np.stack(h.orc.keyswitch(*modes, prm.q_idx, prm.p_idx, 3, c1, evk)))
    ks.hmult(h.p(o), second, h.p(d_c0), h.p(d_c1), h.p(d_c1), h.p(d_c0), h.p(d_evk), 0)
    assert np.array_equal(h.down(o), np.stack(h.orc.hmult_relin(*modes, False, prm.q_idx, prm.p_idx, 3, c0, c1, c1, c0, evk)))
    ks.close()
