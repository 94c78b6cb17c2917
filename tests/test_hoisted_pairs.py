"""Baby steps of a linear transform, which rotate in pairs: an even and an odd number of them, and a plan whose work buffers
have no room for a second rotation (three extension limbs beside three limbs)."""
import pytest

from cerium_b200 import _capi
from tests import parity_cases as pc


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


@pytest.mark.parametrize("word_bits,L,K,dnum,g", [(64, 3, 2, 2, 3), (64, 4, 2, 2, 4), (64, 3, 3, 2, 3), (32, 4, 2, 2, 4), (32, 4, 2, 2, 5)])
def test_linear_transform(be, word_bits, L, K, dnum, g):
    modes = (_capi.BCONV_EXACT, _capi.ROUND_HALF) if word_bits == 64 else (_capi.BCONV_LAZY, _capi.ROUND_FLOOR)
    pc.case_bsgs(be, word_bits, L, K, dnum, *modes, g=g, n_giant=2, r=0)


@pytest.mark.gpu
def test_the_largest_plan():
    """64 limbs: both polynomials of a rotation fill the final transform's launch."""
    from tests import backends
    pc.case_bsgs(backends.CudaBackend(), 32, 64, 16, 4, _capi.BCONV_LAZY, _capi.ROUND_FLOOR, g=3, n_giant=2, r=0)


def test_a_rescale_without_a_rotated_diagonal_is_refused(be):
    """The rotated giant step has a key and no diagonal: there is no ModDown that could divide, and the sums do not fit the outputs."""
    prm = pc.small_params(64, 3, 1, 3)
    h = pc.Harness(be, 64, prm.moduli)
    ks = _capi.KeySwitch(h.ctx, prm.q_idx, prm.p_idx, 3, _capi.BCONV_EXACT, _capi.ROUND_HALF)
    limbs, key, work = h.new(5, 3, pc.N), h.new(3, 2, 4, pc.N), h.new(ks.bsgs_work_limbs(1, 2), pc.N)
    poly = 3 * pc.N * 8
    p = [h.p(limbs) + k * poly for k in range(5)]
    call = lambda r, pts: ks.bsgs_apply(p[0], p[1], p[2], p[3], 1, 2, pts, [0], [1], [0, h.p(key)], [1, 5], r, h.p(work))  # noqa: E731
    for r in (1, 2):
        with pytest.raises(_capi.CeriumError) as e:
            call(r, [p[4], 0])
        assert e.value.code == _capi.ERR_UNSUPPORTED
    call(0, [p[4], 0])
    call(1, [0, p[4]])
    be.sync()
    ks.close()
