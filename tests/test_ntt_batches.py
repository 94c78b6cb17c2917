"""Transforms on both sides of the batch size where the passes change from small tiles (64 limbs of 64-bit words, 74
of 32-bit words on 148 SMs) to usual ones, for every arithmetic (64-bit words: primes of 60, 51 and 50 bits), batches that go on
in a second and a third launch, and two polynomials around the largest launch that holds both: exact against the oracle, forward
and inverse."""
import numpy as np
import pytest

from cerium_b200 import _capi, params
from tests import backends, parity_cases as pc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("word_bits", [64, 32])
@pytest.mark.parametrize("count", [1, 27, 64, 65, 74, 75])
def test_ntt_batch_sizes(word_bits, count):
    mods = pc.moduli_for(word_bits, 3, 1)
    if word_bits == 64:
        mods = mods + params.ntt_primes_below(51, 1, 16)
    h = pc.Harness(backends.CudaBackend(), word_bits, mods)
    idx = [(count + b) % len(mods) for b in range(count)]
    x = pc.rand_limbs(np.random.default_rng(count), mods, idx)
    want = h.orc.ntt_forward(x, idx)
    d = h.up(x)
    h.ctx.ntt_forward(h.p(d), h.p(d), idx)
    assert np.array_equal(h.down(d), want)
    h.ctx.ntt_inverse(h.p(d), h.p(d), idx)
    assert np.array_equal(h.down(d), x)


@pytest.mark.parametrize("word_bits", [64, 32])
@pytest.mark.parametrize("count", [577, 1153])
def test_batches_of_several_launches(word_bits, count):
    """A launch holds 576 limbs: the next one starts at its own slots, primes and strides."""
    mods = pc.moduli_for(word_bits, 3, 1)
    h = pc.Harness(backends.CudaBackend(), word_bits, mods)
    idx = [(7 * b + b // 5) % len(mods) for b in range(count)]
    own = 8     # limbs of their own, each in turn under a prime of its own choice
    base = pc.rand_limbs(np.random.default_rng(count), [min(mods)], [0] * own)
    want = {(k, p): h.orc.ntt_forward(base[k:k + 1], [p])[0] for k in range(own) for p in range(len(mods))}
    stride = pc.N + 16 // h.ctx.word_bytes
    x = np.zeros((count, stride), dtype=h.dt)
    x[:, :pc.N] = base[np.arange(count) % own]
    d = h.up(x)
    out = h.new(count, pc.N)
    h.ctx.ntt_forward(h.p(out), h.p(d), idx, pc.N, stride)
    got = h.down(out)
    assert all(np.array_equal(got[b], want[b % own, idx[b]]) for b in range(count))
    h.ctx.ntt_inverse(h.p(d), h.p(out), idx, stride, pc.N)
    assert np.array_equal(h.down(d), x)


@pytest.mark.parametrize("word_bits,L", [(64, 49), (64, 50), (64, 65), (32, 52)])
def test_two_polynomials_of_a_rescale_in_one_launch(word_bits, L):
    """A launch holds 128 limbs, two polynomials of 64; it held 96."""
    pc.case_rescale(backends.CudaBackend(), word_bits, _capi.ROUND_HALF, L=L)
