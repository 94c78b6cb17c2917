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
