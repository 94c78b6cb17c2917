"""Operands that are not 16-byte aligned: the kernels move 16 bytes at a time, so a call refuses such an operand or takes a
way that does not."""
import numpy as np
import pytest

import oracle
from cerium_b200 import _capi
from tests import parity_cases as pc

L, K, DNUM = 3, 2, 2


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


class Plan:
    def __init__(self, be, word_bits):
        prm = self.prm = pc.small_params(word_bits, L, K, DNUM)
        self.h = pc.Harness(be, word_bits, prm.moduli)
        self.c0, self.c1, self.evk = pc.make_keyswitch_inputs(np.random.default_rng(5), prm)
        self.d_c0, self.d_c1, self.d_evk = self.h.up(self.c0), self.h.up(self.c1), self.h.up(self.evk)
        self.ks = _capi.KeySwitch(self.h.ctx, prm.q_idx, prm.p_idx, DNUM, _capi.BCONV_LAZY, _capi.ROUND_FLOOR)


@pytest.mark.parametrize("word_bits", [64, 32])
@pytest.mark.parametrize("levels", [0, 1, 2])
def test_additions_of_a_key_switch_are_refused(be, word_bits, levels):
    t = Plan(be, word_bits)
    h, word = t.h, word_bits // 8
    o = h.new(2, L - levels, pc.N)
    spare = h.new(L + 1, pc.N)
    o1 = h.p(o) + (L - levels) * pc.N * word
    for add0, add1 in ((h.p(spare) + word, 0), (0, h.p(spare) + 8), (h.p(t.d_c0), h.p(spare) + word)):
        with pytest.raises(_capi.CeriumError) as e:
            t.ks.apply_rescale(h.p(o), o1, h.p(t.d_c1), h.p(t.d_evk), levels, add0, add1)
        assert e.value.code == _capi.ERR_INVALID
    be.sync()
    t.ks.close()


@pytest.mark.parametrize("word_bits", [64, 32])
def test_hoisted_rotation_into_outputs_aligned_to_words(be, word_bits):
    t = Plan(be, word_bits)
    h, word, prm = t.h, word_bits // 8, t.prm
    elt = be.lib.galois_elt_from_step(-3, pc.LOGN)
    k0, k1 = h.orc.keyswitch(_capi.BCONV_LAZY, _capi.ROUND_FLOOR, prm.q_idx, prm.p_idx, DNUM, t.c1, t.evk)
    k0 = np.stack([oracle.ew("add", prm.moduli[p], k0[i], t.c0[i]) for i, p in enumerate(prm.q_idx)])
    want = [np.stack([oracle.apply_galois_ntt(elt, pc.LOGN, k[i]) for i in range(L)]) for k in (k0, k1)]
    buf = [h.new((L + 1) * pc.N) for _ in range(2)]
    t.ks.hoisted_begin(h.p(t.d_c1))
    t.ks.hoisted_rotate(h.p(buf[0]) + word, h.p(buf[1]) + 3 * word, h.p(t.d_c0), h.p(t.d_c1), h.p(t.d_evk), elt)
    for b, at, w in zip(buf, (1, 3), want):
        assert np.array_equal(h.down(b)[at:at + L * pc.N].reshape(L, pc.N), w)
    # outputs on top of the inputs: refused
    with pytest.raises(_capi.CeriumError) as e:
        t.ks.hoisted_rotate(h.p(t.d_c0) + word, h.p(t.d_c1), h.p(t.d_c0), h.p(t.d_c1), h.p(t.d_evk), elt)
    assert e.value.code == _capi.ERR_INVALID
    be.sync()
    t.ks.close()


@pytest.mark.parametrize("word_bits,world", [(64, 2), (32, 2), (64, 1)])
def test_sharded_key_switch_from_a_gather_buffer_aligned_to_words(be, word_bits, world):
    prm = pc.small_params(word_bits, 4, 2, 2)
    h, word = pc.Harness(be, word_bits, prm.moduli), word_bits // 8
    _c0, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(6), prm)
    want = h.orc.keyswitch(_capi.BCONV_EXACT, _capi.ROUND_HALF, prm.q_idx, prm.p_idx, 2, c1, evk)
    plans = [_capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, 2, _capi.BCONV_EXACT, _capi.ROUND_HALF, rank=r, world=world) for r in range(world)]
    g = -(-4 // world)
    gathered = np.zeros((world * g, pc.N), dtype=h.dt)
    for r, ks in enumerate(plans):     # what the ranks send, one after another
        send, mine = h.new(g, pc.N), h.up(c1[r::world])
        ks.sharded_begin(h.p(send), h.p(mine))
        gathered[r * g:(r + 1) * g] = be.to_host(send)
    flat = be.to_dev(np.concatenate([np.zeros(1, dtype=h.dt), gathered.ravel(), np.zeros(3, dtype=h.dt)]))
    for r, ks in enumerate(plans):
        local = list(range(r, 4, world))
        key = evk[:, :, local + [4, 5]]
        o = [h.new(len(local), pc.N) for _ in range(2)]
        d_c1, d_key = h.up(c1[local]), h.up(key)
        ks.sharded_finish(h.p(o[0]), h.p(o[1]), h.p(flat) + word, h.p(d_c1), h.p(d_key))
        for out, w in zip(o, want):
            assert np.array_equal(h.down(out), w[local])
        ks.close()
