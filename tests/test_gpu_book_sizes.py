"""Device-built codebooks around the sum of counts where their weights change from 32 to 64 bits,
small and large ones side by side in every order, against the host builder."""
import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import batch as B

pytestmark = pytest.mark.gpu

LIMIT = (1 << 24) - 1


def _hist(total, n, seed):
    """n symbols whose counts add up to `total`, of very different sizes."""
    rng = np.random.default_rng(seed)
    p = rng.random(n) ** 12 + 1e-9
    c = np.maximum(1, (p / p.sum() * (total - n)).astype(np.int64))
    c[0] += total - c.sum()
    h = np.zeros(256, np.uint32)
    h[rng.permutation(256)[:n]] = c.astype(np.uint32)
    assert int(h.sum(dtype=np.uint64)) == total
    return h


@pytest.mark.parametrize("n", [1, 2, 3, 17, 255, 256])
@pytest.mark.parametrize("order", [0, 1, 2])
def test_books_at_the_weight_limit(n, order):
    totals = [LIMIT - 1, LIMIT, LIMIT + 1, 300, 2**32 - 1, 5000, LIMIT * 7]
    hs = np.stack([_hist(t, n, 7 * i + n) for i, t in enumerate(np.roll(totals, order))])
    books, sizes = B.device_codebooks(torch.from_numpy(hs.view(np.int32)).cuda())
    for h, b, z in zip(hs, books, sizes):
        hb, hz = H.Codebook.from_histogram(h)
        assert np.array_equal(b.symbols, hb.symbols) and np.array_equal(b.lengths, hb.lengths)
        assert np.array_equal(b.code, hb.code) and np.array_equal(b.length, hb.length)
        assert (z.bits, z.words, z.segments, z.gap_words) == (hz.bits, hz.words, hz.segments, hz.gap_words)
