"""The encoder at the edges of its units on the GPU, bit for bit against the oracle: a lane's 32
bytes, a warp's 1 KiB, a step's 16 KiB, a region's end, every input alignment, an output that is
not 16-byte aligned, and bytes whose codes are the longest where a warp's words do not fit its
image in shared memory."""
import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu

WARP, STEP = 1024, 16384


def _check(x, offsets, out_shift=0):
    book_o = O.codebook(O.histogram(x))
    bits_o, gaps_o, _ = O.encode(x, book_o)
    book, sizes = H.Codebook.from_histogram(O.histogram(x))
    enc = H.Encoder(x.size)
    for off in offsets:
        # the bytes around the input are others than those in it
        whole = torch.from_numpy(np.resize(np.arange(255, -1, -1, dtype=np.uint8), x.size + 64)).cuda()
        d = whole[off:off + x.size]
        d.copy_(torch.from_numpy(x))
        bits = torch.zeros(sizes.words + 4, dtype=torch.int32, device="cuda")[out_shift:]
        gaps = torch.zeros(sizes.gap_words + 4, dtype=torch.int32, device="cuda")[out_shift:]
        b, g = enc.encode(d, book, sizes, bits=bits, gaps=gaps)
        assert np.array_equal(b.cpu().numpy().view(np.uint32), bits_o), (x.size, off, out_shift)
        assert np.array_equal(g.cpu().numpy().view(np.uint32), gaps_o), (x.size, off, out_shift)
        assert int(bits[sizes.words:].abs().sum()) == 0 and int(gaps[sizes.gap_words:].abs().sum()) == 0


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, WARP - 16, WARP - 1, WARP, WARP + 1, WARP + 33, STEP - 1, STEP,
                               STEP + 1, STEP + WARP, 2 * STEP + 17, 65536 - 15, 65536, 65536 + 15])
def test_sizes_and_alignments(n):
    rng = np.random.default_rng(n)
    _check(rng.zipf(1.4, n).clip(1, 256).astype(np.int64).__sub__(1).astype(np.uint8), range(16))


@pytest.mark.parametrize("symbols", [1, 2, 3])
def test_shortest_codes(symbols):
    """1-bit codes: a lane's 32 bytes are exactly one word, or a word and a little."""
    rng = np.random.default_rng(symbols)
    x = rng.choice(symbols, 3 * STEP + 100, p=np.array([0.9, 0.06, 0.04][:symbols]) / sum([0.9, 0.06, 0.04][:symbols]))
    _check(x.astype(np.uint8), (0, 1, 15))


def _with_rare_run(n, at, run, seed):
    """Mostly one byte value, and a run of ~200 others that together are rare: 13- to 16-bit codes."""
    rng = np.random.default_rng(seed)
    x = np.where(rng.random(n) < 0.9, 7, 9).astype(np.uint8)
    x[at:at + run] = rng.integers(40, 240, run)
    return x


@pytest.mark.parametrize("at,run", [(0, 700), (5000, WARP), (5 * WARP, WARP), (3 * WARP - 100, 2300), (STEP - 600, 1200),
                                    (1 << 20, 3000), ((3 << 20) - 2500, 2500), ((3 << 20) - 400, 400)])
def test_longest_codes(at, run):
    _check(_with_rare_run(3 << 20, at, run, at + run), (0, 3))


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_unaligned_output(shift):
    rng = np.random.default_rng(shift)
    _check(rng.integers(0, 100, 40000).astype(np.uint8), (0, 7), out_shift=shift)
    _check(_with_rare_run(1 << 20, 9000, 2500, shift), (2,), out_shift=shift)


@pytest.mark.parametrize("tail", [0, 1, 40, WARP + 5])
def test_many_regions(tail):
    """Regions of several chunks, whose ends fall anywhere in a word and a gap word."""
    rng = np.random.default_rng(100 + tail)
    _check(np.minimum(rng.geometric(0.08, (5 << 20) + tail) - 1, 255).astype(np.uint8), (0, 13))
