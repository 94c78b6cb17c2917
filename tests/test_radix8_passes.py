"""Transforms on both sides of the batch sizes where a pass changes between eight words a thread and sixteen, for every arithmetic (64-bit
words: 32 limbs forward, 23, 35, 64 and 128 inverse; 32-bit words: 27, 55, 74 and 90 inverse), as stacks and as pointer tables, and
limbs of 64-bit words that are aligned to 16 bytes only, whose rows move as pairs of words: exact against the oracle."""
import numpy as np
import pytest

from cerium_b200 import _capi, params
from tests import parity_cases as pc


def gpu(*args):
    return pytest.param(*args, marks=pytest.mark.gpu)


def harness(name, word_bits):
    from tests import backends
    mods = pc.moduli_for(word_bits, 3, 1)
    if word_bits == 64:
        mods = mods + params.ntt_primes_below(51, 1, 16)
    return pc.Harness(backends.EmuBackend() if name == "emu" else backends.CudaBackend(), word_bits, mods)


@pytest.mark.parametrize("name,word_bits,count", [("emu", 64, 4), ("emu", 32, 3)] + [
    gpu("cuda", 64, c) for c in (1, 24, 25, 32, 33, 64, 65, 128, 129, 256, 257)] + [gpu("cuda", 32, c) for c in (1, 28, 29, 33, 280, 281)])
def test_batch_sizes(name, word_bits, count):
    h = harness(name, word_bits)
    idx = [(count + b) % len(h.moduli) for b in range(count)]
    x = pc.rand_limbs(np.random.default_rng(count), h.moduli, idx)
    x[0] = pc.edge_limbs(h.moduli, idx[:1])[0]
    d = h.up(x)
    h.ctx.ntt_forward(h.p(d), h.p(d), idx)
    assert np.array_equal(h.down(d), h.orc.ntt_forward(x, idx))
    h.ctx.ntt_inverse(h.p(d), h.p(d), idx)
    assert np.array_equal(h.down(d), x)


@pytest.mark.parametrize("name,word_bits,integers,count", [("emu", 64, False, 3), ("emu", 32, False, 2)] + [
    gpu("cuda", 64, i, c) for c in (23, 24, 35, 36, 64, 65, 129) for i in (False, True)] + [
    gpu("cuda", 32, False, c) for c in (27, 28, 55, 56, 74, 75, 90, 91)])
def test_lines_of_the_inverse_passes(name, word_bits, integers, count):
    from tests import backends
    mods = params.ntt_primes_below(60, 3, pc.LOGN) if integers else pc.moduli_for(word_bits, 3, 1)
    be = backends.EmuBackend() if name == "emu" else backends.CudaBackend()
    h = pc.Harness(be, word_bits, mods)
    idx = [b % len(mods) for b in range(count)]
    want = pc.rand_limbs(np.random.default_rng(count), mods, idx)
    x = h.orc.ntt_forward(want, idx)
    d, out = h.up(x), h.new(count, pc.N)
    h.ctx.ntt_inverse(h.p(out), h.p(d), idx)
    assert np.array_equal(h.down(out), want)
    at = lambda b: be.to_dev(np.array([h.p(b) + k * pc.N * h.ctx.word_bytes for k in range(count)], dtype=np.uint64))  # noqa: E731
    outs, ins, bases = at(out), at(d), be.to_dev(np.array(idx, dtype=np.uint32))
    h.ctx.ntt_inverse_ptrs(be.ptr(outs), be.ptr(ins), be.ptr(bases), count)
    assert np.array_equal(h.down(out), want)
    h.ctx.ntt_forward_ptrs(be.ptr(outs), be.ptr(outs), be.ptr(bases), count)
    assert np.array_equal(h.down(out), x)


@pytest.mark.parametrize("name", ["emu", gpu("cuda")])
def test_limbs_aligned_to_two_words(name):
    h = harness(name, 64)
    stride, idx = pc.N + 2, list(range(len(h.moduli)))
    x = pc.rand_limbs(np.random.default_rng(3), h.moduli, idx)
    flat = np.zeros((len(idx) + 1) * stride, dtype=np.uint64)
    limbs = lambda a: np.lib.stride_tricks.as_strided(a[2:], (len(idx), pc.N), (8 * stride, 8))  # noqa: E731
    limbs(flat)[...] = x
    d, out = h.up(flat), h.new(flat.size)
    h.ctx.ntt_forward(h.p(out) + 16, h.p(d) + 16, idx, stride, stride)
    assert np.array_equal(limbs(h.down(out)), h.orc.ntt_forward(x, idx))
    h.ctx.ntt_inverse(h.p(d) + 16, h.p(out) + 16, idx, stride, stride)
    assert np.array_equal(limbs(h.down(d)), x)
    # division by the last limb, whose row pass reads what it subtracts from as well
    div, scratch, packed = h.new(flat.size), h.new(pc.N), h.up(np.concatenate([np.zeros(2, np.uint64), x.ravel()]))
    h.ctx.rescale(h.p(div) + 16, h.p(packed) + 16, idx, 1, h.p(scratch), _capi.ROUND_HALF)
    want = h.orc.rescale(_capi.ROUND_HALF, idx, x)
    assert np.array_equal(h.down(div)[2:2 + want.size].reshape(want.shape), want)
