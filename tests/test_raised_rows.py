"""Row pass of the raised digits inside the inner product of a key switch: every arithmetic (primes of 60, 51 and 50 bits),
more digits than a sum of doubles holds before it is reduced, for one warp to a row and for each of two, and keys that are
aligned to 16 bytes only, which take the separate kernels with 64-bit words.  The launches are counted, so that a call that
takes another path than the one it is here for fails."""
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


# the last column: whether the plan has the rows for it on a GPU of 148 SMs (1.8 for each of 16 warps an SM, 1.4 from 12 digits
# on); 12 digits in 13 limbs and 10 in 17 are just past the line, 19 and 25 limbs well
SHAPES = [(64, 3, 1, 3, False), (64, 12, 1, 12, True), (64, 15, 2, 10, True), (32, 9, 2, 5, True), (64, 20, 5, 4, True)]


@pytest.mark.parametrize("word_bits,L,K,dnum,rows,offset", [s + (o,) for o in (0, 16) for s in SHAPES] + [(64, 18, 1, 18, True, 0), (32, 12, 1, 12, True, 0)])
def test_key_switch(be, word_bits, L, K, dnum, rows, offset):
    if be.name == "emu" and L == 20:
        L, K, dnum = 8, 2, 4   # the emulated device has the rows for any plan
    prm = _params(word_bits, L, K, dnum)
    h = pc.Harness(be, word_bits, prm.moduli)
    c0, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(dnum), prm)
    if offset == 0:  # the largest key words
        evk[..., ::2] = np.array([prm.moduli[p] - 1 for p in prm.q_idx + prm.p_idx], dtype=np.uint64)[:, None]
    modes = (_capi.BCONV_EXACT, _capi.ROUND_HALF) if word_bits == 64 else (_capi.BCONV_LAZY, _capi.ROUND_FLOOR)
    shape = (prm.q_idx, prm.p_idx, dnum)
    ks = _capi.KeySwitch(h.ctx, *shape[:2], dnum, *modes)
    words = offset * 8 // word_bits
    d_evk = h.up(np.concatenate([np.zeros(words, dtype=np.uint64), evk.reshape(-1), np.zeros(4, dtype=np.uint64)]))
    key = h.p(d_evk) + offset
    d_c0, d_c1 = h.up(c0), h.up(c1)
    o = h.new(2, L, pc.N)
    second = h.p(o) + L * pc.N * word_bits // 8
    ks.apply(h.p(o), second, h.p(d_c1), key)
    assert np.array_equal(h.down(o), np.stack(h.orc.keyswitch(*modes, *shape, c1, evk)))
    elt = be.lib.galois_elt_from_step(7, pc.LOGN)
    ks.hrot(h.p(o), second, h.p(d_c0), h.p(d_c1), key, elt)
    assert np.array_equal(h.down(o), np.stack(h.orc.hrot(*modes, *shape, elt, c0, c1, evk)))
    # a multiplication: the products of the tensor are taken where they are read
    b0, b1 = (pc.rand_limbs(np.random.default_rng(8 + k), prm.moduli, prm.q_idx) for k in range(2))
    d_b0, d_b1 = h.up(b0), h.up(b1)
    inputs = [h.p(d_c0), h.p(d_c1), h.p(d_b0), h.p(d_b1)]
    ks.hmult(h.p(o), second, *inputs, key, 0)
    assert np.array_equal(h.down(o), np.stack(h.orc.hmult_relin(*modes, False, *shape, c0, c1, b0, b1, evk)))
    r = h.new(2, L - 1, pc.N)
    # with a rescale, after the division and in it
    for levels, want in ((1, lambda: h.orc.hmult_relin(*modes, True, *shape, c0, c1, b0, b1, evk)),
                         (2, lambda: h.orc.hmult_relin_fused(*modes, *shape, c0, c1, b0, b1, evk)))[:2 if K > 1 else 0]:
        ks.hmult(h.p(r), h.p(r) + (L - 1) * pc.N * word_bits // 8, *inputs, key, levels)
        assert np.array_equal(h.down(r), np.stack(want())), levels
    # which kernels these were: the row pass is one of its own, or not, and the tensor product likewise
    one = (word_bits == 32 or offset == 0) and (rows or be.name == "emu")
    integers = word_bits == 64 and 2 * sum(prm.moduli[p] >> 50 > 0 for p in prm.q_idx + prm.p_idx) > L + K
    tensor = one and not integers and (word_bits == 32 or dnum < 12)
    converted = int(dnum != L)     # every digit's conversion in one launch
    assert be.launches(lambda st: ks.hoisted_begin(h.p(d_c1), st)) == 4 + converted
    switch = 9 + converted + (not one)
    assert be.launches(lambda st: ks.apply(h.p(o), second, h.p(d_c1), key, stream=st)) == switch
    assert be.launches(lambda st: ks.hmult(h.p(o), second, *inputs, key, 0, st)) == switch + (not tensor)
    ks.close()


@pytest.mark.parametrize("word_bits,L,K,dnum,conversions", [(64, 9, 5, 2, 1), (64, 17, 9, 2, 2), (32, 17, 9, 2, 1)])
def test_digits_of_two_sizes(be, word_bits, L, K, dnum, conversions):
    """A digit takes a step more to share the launch of a longer one, but not where the longer one's fragments leave the registers
    (9 limbs of 64-bit words)."""
    prm = _params(word_bits, L, K, dnum)
    h = pc.Harness(be, word_bits, prm.moduli)
    _c0, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(L), prm)
    modes = (_capi.BCONV_EXACT, _capi.ROUND_HALF) if word_bits == 64 else (_capi.BCONV_LAZY, _capi.ROUND_FLOOR)
    ks = _capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, dnum, *modes)
    d_c1, d_evk, o = h.up(c1), h.up(evk), h.new(2, L, pc.N)
    ks.apply(h.p(o), h.p(o) + L * pc.N * word_bits // 8, h.p(d_c1), h.p(d_evk))
    assert np.array_equal(h.down(o), np.stack(h.orc.keyswitch(*modes, prm.q_idx, prm.p_idx, dnum, c1, evk)))
    assert be.launches(lambda st: ks.hoisted_begin(h.p(d_c1), st)) == 4 + conversions   # two passes each way
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
    assert be.launches(lambda st: ks.hoisted_begin(h.p(d_c1), st)) == 5
    assert be.launches(lambda st: ks.apply(h.p(o), second, h.p(d_c1), h.p(d_evk), stream=st)) == 10 + (bits < 34)
    ks.close()


@pytest.mark.parametrize("L,K,dnum,rows", [(16, 1, 16, False), (20, 5, 4, True), (16, 5, 4, False)])
def test_plans_of_60_bit_primes(be, L, K, dnum, rows):
    """Integer butterflies: the kernels stay apart below 2.5 rows for each of 16 warps an SM, a row keeps one warp, and the tensor
    product is a kernel of its own."""
    if be.name == "emu":
        L, K, dnum = (6, 1, 6) if dnum == L else (6, 2, 3)
    mods = params.ntt_primes_below(60, L + K, pc.LOGN)
    h = pc.Harness(be, 64, mods)
    shape = (list(range(L)), list(range(L, L + K)), dnum)
    c0, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(L), params.CkksParams(pc.LOGN, 64, mods, L, K, dnum, q_idx=shape[0], p_idx=shape[1]))
    evk[..., ::2] = np.array(mods, dtype=np.uint64)[:, None] - 1
    modes = (_capi.BCONV_EXACT, _capi.ROUND_HALF)
    ks = _capi.KeySwitch(h.ctx, *shape, *modes)
    d_evk, d_c0, d_c1, o = h.up(evk), h.up(c0), h.up(c1), h.new(2, L, pc.N)
    second = h.p(o) + L * pc.N * 8
    ks.apply(h.p(o), second, h.p(d_c1), h.p(d_evk))
    assert np.array_equal(h.down(o), np.stack(h.orc.keyswitch(*modes, *shape, c1, evk)))
    ks.hmult(h.p(o), second, h.p(d_c0), h.p(d_c1), h.p(d_c1), h.p(d_c0), h.p(d_evk), 0)
    assert np.array_equal(h.down(o), np.stack(h.orc.hmult_relin(*modes, False, *shape, c0, c1, c1, c0, evk)))
    converted = int(dnum != L)
    assert be.launches(lambda st: ks.hoisted_begin(h.p(d_c1), st)) == 4 + converted
    switch = 9 + converted + (not rows and be.name != "emu")
    assert be.launches(lambda st: ks.apply(h.p(o), second, h.p(d_c1), h.p(d_evk), stream=st)) == switch
    assert be.launches(lambda st: ks.hmult(h.p(o), second, h.p(d_c0), h.p(d_c1), h.p(d_c1), h.p(d_c0), h.p(d_evk), 0, st)) == switch + 1
    ks.close()
