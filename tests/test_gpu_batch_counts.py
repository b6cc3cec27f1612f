"""Batches whose number of buffers lies at the edges of the setup scans (256 buffers a CTA, at
most 64 CTAs, then 1024 buffers a step), empty buffers and large ones among them: entries consistent, everything
decoded, sampled streams equal to the single-buffer path's."""
import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import batch as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("region_chunks", [1, 8])
@pytest.mark.parametrize("count", [1, 2, 255, 256, 257, 1025, 4097, 16385, 33000, 66000])
def test_counts(count, region_chunks):
    rng = np.random.default_rng(count)
    sizes = rng.integers(0, 60, count)
    sizes[rng.integers(0, count, max(1, count // 50))] = 0
    big = rng.integers(0, count, 5)
    sizes[big] = rng.integers(1, 200_000, big.size)
    at = np.concatenate([[0], np.cumsum(sizes)])
    data = torch.from_numpy(np.minimum(rng.geometric(0.1, int(at[-1]) + 1) - 1, 255).astype(np.uint8)).cuda()
    back = torch.zeros_like(data)
    ins = [data[at[i]:at[i + 1]] for i in range(count)]
    outs = [back[at[i]:at[i + 1]] for i in range(count)]
    plan = B.BatchCodec(sizes, B.LaunchConfig(region_chunks=region_chunks), inputs=ins, outputs=outs)
    plan.compress()
    plan.check_compress()
    plan.decompress()
    plan.check_decompress()
    assert torch.equal(back[:int(at[-1])], data[:int(at[-1])])
    entries = plan.entries_host()
    ob = og = 0
    for e, n in zip(entries, sizes):
        assert (e.n, e.status, e.bits_offset, e.gaps_offset) == (n, 0, ob, og)
        ob += (e.words + 3) // 4 * 4
        og += e.gap_words
    for i in sorted(set([0, count - 1, *big.tolist(), *rng.integers(0, count, 5).tolist()])):
        if sizes[i] == 0:
            assert entries[i].words == 0
            continue
        c, s = H.compress(ins[i].clone()), plan.stream(i, entries[i])
        assert torch.equal(c.bits, s.bits) and torch.equal(c.gaps, s.gaps)
        assert np.array_equal(c.book.lengths, s.book.lengths) and np.array_equal(c.book.symbols, s.book.symbols)
