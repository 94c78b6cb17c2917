"""A handle can be used on any stream as soon as the call that made it returns: its tables are on the device, not on their
way there on the default stream, which a non-blocking stream does not wait for."""
import numpy as np
import pytest

from cerium_b200 import _capi
from tests import backends, parity_cases as pc


@pytest.mark.parametrize("word_bits", [64, 32])
def test_tables_are_in_place_when_a_handle_is_made(word_bits):
    be = backends.EmuBackend()
    early = be.lib.dll.cerium_emu_early_launches
    prm = pc.small_params(word_bits, 4, 2, 2)
    before = early()
    h = pc.Harness(be, word_bits, prm.moduli)
    x = h.up(pc.rand_limbs(np.random.default_rng(1), prm.moduli, prm.q_idx))
    h.ctx.ntt_forward(h.p(x), h.p(x), prm.q_idx)
    assert early() == before, "context"
    bc = _capi.BaseConverter(h.ctx, prm.q_idx, prm.p_idx, _capi.BCONV_LAZY)
    out = h.new(2, pc.N)
    bc.apply(h.p(out), h.p(x))
    assert early() == before, "converter"
    ks = _capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, 2, _capi.BCONV_EXACT, _capi.ROUND_HALF)
    ks.hoisted_begin(h.p(x))
    assert early() == before, "key switch"
    if word_bits == 32:
        comp, values = _capi.Composer(h.ctx, prm.q_idx), be.empty((pc.N,), np.float64)
        comp.apply(be.ptr(values), h.p(x))
        assert early() == before, "composition"
