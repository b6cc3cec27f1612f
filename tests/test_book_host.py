"""The host codebook builder against the oracle where its merge can go wrong: few symbols (levels
shorter than the cuts they are merged in), ties everywhere, every number of symbols, counts that use
all 32 bits, depths that reach the 16-bit limit."""
import numpy as np
import pytest

import huffman_coding_gap_arrays_b200 as H
from oracle import oracle as O


def _same(h):
    b, z = H.Codebook.from_histogram(h)
    o = O.codebook(h)
    n = b.symbol_count
    assert n == int((h > 0).sum())
    assert np.array_equal(b.symbols, o.symbols[:n]) and np.array_equal(b.lengths, o.lengths[:n])
    assert np.array_equal(b.code, o.code) and np.array_equal(b.length, o.length)
    assert z.bits == o.total_bits


@pytest.mark.parametrize("n", range(1, 257))
def test_every_symbol_count(n):
    rng = np.random.default_rng(n)
    at = rng.permutation(256)[:n]
    for counts in (np.ones(n), rng.integers(1, 4, n), rng.integers(1, 2**32, n, dtype=np.uint64),
                   np.maximum(1, 1e9 * 0.55 ** np.arange(n)), 1 + 1e7 * np.arange(1, n + 1.0) ** -1.3):
        h = np.zeros(256, np.uint32)
        h[at] = np.asarray(counts).astype(np.uint64).astype(np.uint32)
        _same(h)


@pytest.mark.parametrize("seed", range(20))
def test_random_histograms(seed):
    rng = np.random.default_rng(1000 + seed)
    for _ in range(50):
        h = (rng.random(256) < rng.random()) * rng.integers(0, 2 ** int(rng.integers(1, 33)), 256, dtype=np.uint64)
        if h.any():
            _same(h.astype(np.uint32))
