"""Batched decompress of books that the compressor does not make: incomplete ones of every shortest code
(one launch serves them all), and complete ones whose longest code lies around the table's prefix of 10 bits
(shortest code 1 bit) or 11 bits.  Streams come from the oracle; every buffer is decoded by both paths."""
import ctypes as C

import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import batch as B
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _ladder(first, last):  # complete: first, first + 1, ..., last, last, and the rest of the codes of `first` bits
    return [first] * ((1 << first) - 1) + list(range(first + 1, last + 1)) + [last]


def _full(head, last):  # head, and the rest of the code space in codes of `last` bits
    left = (1 << last) - sum(1 << (last - l) for l in head)
    assert 0 < left <= 256 - len(head)
    return head + [last] * left


INCOMPLETE = [[1], [1, 2], [1, 3, 16], [2], [2, 2, 2], [2, 3, 4, 11, 12], [3] * 5, [3, 3, 7, 12, 12, 16],
              [4] * 7 + [5, 6, 11, 12, 16], [5] * 20, [8] * 100, [16] * 40]
COMPLETE = ([_ladder(1, k) for k in (2, 9, 10, 11, 12, 16)] + [_ladder(2, k) for k in (3, 10, 11, 12, 16)] +
            [_full([1, 2, 3], 10), _full([1, 2, 3, 4], 11), _full([1, 2, 3, 4, 5], 12), _full([1, 2, 3, 4, 5, 6], 13),
             _full([2, 2, 2, 3, 4], 11), _full([2, 2, 2, 3, 4, 5], 12), _full([3] * 7 + [4], 11), _full([4] * 15 + [5], 12)])


@pytest.mark.parametrize("books", [INCOMPLETE, COMPLETE], ids=["incomplete", "complete"])
@pytest.mark.parametrize("n", [1, 4097, 70001])
def test_hand_made_books(books, n):
    r = np.random.default_rng(n)
    streams = []
    for lengths in books:
        syms = r.permutation(256)[:len(lengths)].astype(np.uint8)
        p = 0.9 * 2.0 ** -np.array(lengths)
        p = p / p.sum() * 0.9 + 0.1 / len(lengths)
        x = r.choice(syms, n, p=p / p.sum())
        bits, gaps, _ = O.encode(x, O.codebook_from_list(syms, lengths))
        streams.append((x, syms, lengths, bits, gaps))
    count = len(streams)
    outs = [torch.full((n,), 0x5A, dtype=torch.uint8, device="cuda") for _ in streams]
    plan = B.BatchCodec([max(n, 4 * s[3].size) for s in streams])  # (room for the longest stream)
    at_bits, at_gaps = 0, 0
    entries = (B.BatchEntry * count)()
    whole_bits = np.zeros(sum((s[3].size + 3) & ~3 for s in streams) + 4, np.uint32)
    whole_gaps = np.zeros(sum(s[4].size for s in streams), np.uint32)
    for e, (x, syms, lengths, bits, gaps) in zip(entries, streams):
        e.n, e.words, e.bits = n, bits.size, 32 * bits.size
        e.segments, e.gap_words = (bits.size + 3) // 4, gaps.size
        e.bits_offset, e.gaps_offset = at_bits, at_gaps
        e.symbol_count = len(lengths)
        for i, (s, l) in enumerate(zip(syms, lengths)):
            e.symbols[i].symbol, e.symbols[i].length = int(s), int(l)
        whole_bits[at_bits:at_bits + bits.size] = bits
        whole_gaps[at_gaps:at_gaps + gaps.size] = gaps
        at_bits += (bits.size + 3) & ~3
        at_gaps += gaps.size
    plan.bits = torch.from_numpy(whole_bits.view(np.int32)).cuda()
    plan.gaps = torch.from_numpy(whole_gaps.view(np.int32)).cuda()
    plan.entries.copy_(torch.frombuffer(bytearray(bytes(entries)), dtype=torch.uint8)[:C.sizeof(entries)].cuda())
    for mask in (0, B.decoder_class_mask(list(entries))):
        for o in outs:
            o.fill_(0x5A)
        plan.config = B.LaunchConfig(dec_class_mask=mask)
        plan._outputs = outs
        plan.d_out.copy_(torch.tensor([o.data_ptr() for o in outs], dtype=torch.int64))
        plan.decompress()
        plan.check_decompress()
        for o, (x, _, lengths, _, _) in zip(outs, streams):
            assert np.array_equal(o.cpu().numpy(), x), (mask, lengths)
    for x, syms, lengths, bits, gaps in streams:
        z = H.StreamSizes.from_words(bits.size)
        y = H.Decoder(z.segments).decode(torch.from_numpy(bits.view(np.int32)).cuda(),
                                         torch.from_numpy(gaps.view(np.int32)).cuda(), z,
                                         H.Codebook.from_symbols(syms, lengths), n)
        assert np.array_equal(y.cpu().numpy(), x), lengths
