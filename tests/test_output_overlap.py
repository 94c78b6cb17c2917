"""Key switch with an output on top of an addition: whichever polynomial's it is, it is read before it is overwritten."""
import numpy as np
import pytest

import oracle
from cerium_b200 import _capi
from tests import parity_cases as pc


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


@pytest.mark.parametrize("word_bits,L", [(64, 4), (32, 1), (32, 7)])
def test_outputs_over_additions(be, word_bits, L):
    prm = pc.small_params(word_bits, L, 4, min(L, 2))
    h = pc.Harness(be, word_bits, prm.moduli)
    add, c1, evk = pc.make_keyswitch_inputs(np.random.default_rng(3), prm)
    ks = _capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, prm.dnum, _capi.BCONV_EXACT, _capi.ROUND_HALF)
    plain = h.orc.keyswitch(_capi.BCONV_EXACT, _capi.ROUND_HALF, prm.q_idx, prm.p_idx, prm.dnum, c1, evk)
    added = [np.stack([oracle.ew("add", prm.moduli[p], w[i], add[i]) for i, p in enumerate(prm.q_idx)]) for w in plain]
    d_evk = h.up(evk)
    for reads in (0, 1):            # the polynomial that the addition belongs to
        for over in (0, 1):         # the one that is written over it
            d_c1, d_add = h.up(c1), h.up(add)
            outs = [h.new(L, pc.N), h.new(L, pc.N)]
            outs[over] = d_add
            ks.apply(h.p(outs[0]), h.p(outs[1]), h.p(d_c1), h.p(d_evk), *(h.p(d_add) if p == reads else 0 for p in (0, 1)))
            for p in (0, 1):
                assert np.array_equal(h.down(outs[p]), added[p] if p == reads else plain[p]), (reads, over, p)
    ks.close()
