"""Base conversion at the edges of its tensor-core kernel: numbers of inputs around a step of 32 bytes and around the
fragments kept in registers, numbers of outputs around a group, primes of every quotient class.  Exact, against Python
integers on the coefficients that sit at tile and stage edges and on random ones."""
import numpy as np
import pytest

from cerium_b200 import _capi, params

N = 1 << 16


@pytest.fixture(scope="module", params=["emu", pytest.param("cuda", marks=pytest.mark.gpu)])
def be(request):
    from tests import backends
    return backends.EmuBackend() if request.param == "emu" else backends.CudaBackend()


@pytest.mark.parametrize("word_bits,n_in,n_out,mode", [
    (64, 1, 1, _capi.BCONV_LAZY), (64, 4, 8, _capi.BCONV_EXACT), (64, 5, 9, _capi.BCONV_LAZY), (64, 9, 17, _capi.BCONV_EXACT),
    (64, 33, 3, _capi.BCONV_LAZY), (64, 64, 6, _capi.BCONV_LAZY), (64, 8, 16, _capi.BCONV_LAZY), (64, 32, 7, _capi.BCONV_EXACT),
    (64, 9, 35, _capi.BCONV_EXACT), (64, 33, 33, _capi.BCONV_EXACT),       # more warps than an SM holds at 128 registers
    (32, 1, 1, _capi.BCONV_LAZY), (32, 8, 9, _capi.BCONV_EXACT), (32, 17, 16, _capi.BCONV_LAZY), (32, 21, 25, _capi.BCONV_EXACT),
    (32, 32, 17, _capi.BCONV_LAZY), (32, 33, 8, _capi.BCONV_EXACT),
])
def test_bconv_edges(be, word_bits, n_in, n_out, mode):
    if word_bits == 64:     # outputs of 30 to 60 bits in one conversion, inputs of 60 and 50 bits
        widths = (59, 49, 47, 39, 30) if n_in < 64 else (59, 49, 48, 40, 30)    # most inputs: classes at their upper ends
        ins = params.ntt_primes_below(60, (n_in + 1) // 2, 16) + params.ntt_primes_below(50, n_in // 2, 16)
        pools = [params.ntt_primes_below(b, n_out, 16, exclude=ins) for b in widths]
        outs = [pools[j % 5][j] for j in range(n_out)]
    else:
        mods = params.reference_primes_28bit(n_in + n_out)
        ins, outs = mods[:n_in], mods[n_in:]
    ctx = _capi.Context(be.lib, ins + outs, word_bits)
    bc = _capi.BaseConverter(ctx, range(n_in), range(n_in, n_in + n_out), mode)
    dt = np.uint64 if word_bits == 64 else np.uint32
    rng = np.random.default_rng(n_in * 100 + n_out)
    x = np.stack([rng.integers(0, q, N, dtype=dt) for q in ins])
    x[:, 0], x[:, 1] = 0, [q - 1 for q in ins]
    x[:, 2] = [(1 << (q.bit_length() - 1)) - 1 for q in ins]    # low bytes of 255
    dx, out = be.to_dev(x), be.empty((n_out, N), dt)
    bc.apply(be.ptr(out), be.ptr(dx))
    got = be.to_host(out)
    big = 1
    for q in ins:
        big *= q
    hats = [big // q for q in ins]
    invs = [pow(h % q, -1, q) for h, q in zip(hats, ins)]
    at = sorted({0, 1, 2, 7, 8, 127, 128, 383, 384, N - 129, N - 1} | set(int(c) for c in rng.integers(0, N, 200)))
    for j, p in enumerate(outs):
        for c in at:
            if mode == _capi.BCONV_LAZY:
                want = sum(int(x[i, c]) * (invs[i] * hats[i] % p) for i in range(n_in)) % p
            else:
                want = sum(int(x[i, c]) * invs[i] % ins[i] * hats[i] for i in range(n_in)) % p
            assert int(got[j, c]) == want, (j, c)


def test_conversions_of_different_sizes_from_several_threads(be):
    """Conversions that need more than 48 KB of shared memory, 30 and 20 inputs of 64-bit words: neither takes away the
    limit that the other's launch counts on, and both are right when two threads launch them at once."""
    from concurrent.futures import ThreadPoolExecutor
    mods = params.ntt_primes_below(50, 31, 16)
    ctx = _capi.Context(be.lib, mods, 64)
    rng = np.random.default_rng(7)
    x = np.stack([rng.integers(0, q, N, dtype=np.uint64) for q in mods[:30]])
    dx = be.to_dev(x)
    made = [(_capi.BaseConverter(ctx, range(n), [30], _capi.BCONV_LAZY), be.empty((1, N), np.uint64)) for n in (30, 20)]

    def run(k, times):
        for _ in range(times):
            made[k][0].apply(be.ptr(made[k][1]), be.ptr(dx))

    for k in (0, 1, 0):
        run(k, 1)
    if be.name == "emu":
        assert be.lib.dll.cerium_emu_lowered_smem_limits() == 0
    else:
        with ThreadPoolExecutor(2) as pool:
            list(pool.map(run, (0, 1), (2000, 2000)))
    for n, (_bc, out) in zip((30, 20), made):
        got, big = be.to_host(out), 1
        for q in mods[:n]:
            big *= q
        f = [big // q * pow(big // q, -1, q) % mods[30] for q in mods[:n]]
        for c in (0, 1, 127, 128, N - 1):
            assert int(got[0, c]) == sum(int(x[i, c]) * f[i] for i in range(n)) % mods[30]
