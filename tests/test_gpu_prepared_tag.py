"""A prepared encode takes the histograms of the last histogram pass in its workspace, and only those of its
own input: another pass since then, over an input of any other size, is refused with nothing written."""
import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from oracle import oracle as O

pytestmark = pytest.mark.gpu

INVALID_ARG = 1
MiB = 1 << 20


def _bytes(n, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return (torch.rand(n, device="cuda", generator=g) ** 3 * 250).to(torch.uint8)


@pytest.mark.parametrize("first,second", [(256 * MiB, 4 * MiB), (4 * MiB, 256 * MiB), (16 * MiB, 1000), (1000, 16 * MiB),
                                          (16 * MiB, 15 * MiB), (3 * MiB, 3 * MiB)])
def test_another_pass_since(first, second):
    a, b = _bytes(first, 1), _bytes(second, 2)
    enc = H.Encoder(max(first, second))
    books = [H.Codebook.from_histogram(enc.histogram(x).cpu()) for x in (a, b)]
    book, sizes = books[0]
    bits = torch.full((sizes.words,), 0x5A5A5A5A, dtype=torch.int32, device="cuda")
    gaps = torch.full((sizes.gap_words,), 0x5A5A5A5A, dtype=torch.int32, device="cuda")
    for _ in range(2):
        with pytest.raises(H.HgapError) as e:
            enc.encode(a, book, sizes, bits=bits, gaps=gaps, prepared=True)
        assert e.value.status == INVALID_ARG
        assert bool((bits == 0x5A5A5A5A).all()) and bool((gaps == 0x5A5A5A5A).all())
    # the refused calls leave the second input's histograms as they are, for as many calls as there are
    ref = H.compress(b)
    for _ in range(3):
        x, y = enc.encode(b, *books[1], prepared=True)
        assert torch.equal(x, ref.bits) and torch.equal(y, ref.gaps)


@pytest.mark.parametrize("n", [1000, 4 * MiB + 3, 100 * MiB])
def test_prepared_with_several_books(n):
    """One histogram pass, then any number of encodes, each with its own codebook."""
    x = _bytes(n, n)
    enc = H.Encoder(n)
    hist = enc.histogram(x).cpu().numpy().view(np.uint32)
    host = x.cpu().numpy()
    for k in range(4):
        h = hist.astype(np.uint64) + k * np.random.default_rng(k).integers(1, 1 + n // 50, 256, dtype=np.uint64)
        book, _ = H.Codebook.from_histogram(h.astype(np.uint32))
        bits_o, gaps_o, total = O.encode(host, O.codebook(h.astype(np.uint32)))
        assert total == book.encoded_bits(hist)
        words, segs = (total + 31) // 32, (total + 127) // 128
        bits, gaps = enc.encode(x, book, H.StreamSizes(total, words, segs, (segs + 7) // 8), prepared=True)
        assert np.array_equal(bits.cpu().numpy().view(np.uint32), bits_o)
        assert np.array_equal(gaps.cpu().numpy().view(np.uint32), gaps_o)
