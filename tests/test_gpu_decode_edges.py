"""The decoder at the edges of its units on the GPU, through the single-buffer and the batched path:
streams that end around a warp's 32 segments and a tile's 256 or 512, every class of shortest code,
books whose table needs two levels, streams and outputs at other alignments than 16 bytes."""
import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import HgapError
from huffman_coding_gap_arrays_b200 import batch as B
from oracle import oracle as O

pytestmark = pytest.mark.gpu

# per kind: symbol probabilities, shortest code 1 (up to three symbols a lookup), 2, 3, 4 and 8 bits
KINDS = {
    "len1": [0.7, 0.2, 0.06, 0.03, 0.01],
    "len2": [0.3, 0.3, 0.2, 0.1, 0.05, 0.03, 0.02],
    "len3": [0.2] * 3 + [0.1] * 2 + [0.2 / 40] * 40,
    "len4": [1 / 16] * 16,
    "len8": [1 / 256] * 256,
}


def _data(kind, n, seed):
    p = np.array(KINDS[kind])
    return np.random.default_rng(seed).choice(len(p), n, p=p / p.sum()).astype(np.uint8)


def _wide(short):
    """A complete book of one or two very frequent bytes, a hundred of 12 to 13 bits and some of 16:
    one table for all lengths would have thousands of entries, so it gets two levels."""
    x = [np.repeat(np.arange(130, dtype=np.uint8), 30), np.repeat(np.arange(130, 140, dtype=np.uint8), 2),
         np.full(70000, 200, np.uint8)]
    if not short:
        x += [np.full(50000, 201, np.uint8), np.full(30000, 202, np.uint8)]
    x = np.concatenate(x)
    return np.random.default_rng(short).permutation(x)


def _check_single(x, shifts=(0,), outs=(0,)):
    book_o = O.codebook(O.histogram(x))
    bits_o, gaps_o, _ = O.encode(x, book_o)
    book, z = H.Codebook.from_histogram(O.histogram(x))
    dec = H.Decoder(z.segments)
    for s in shifts:
        bits = torch.zeros(z.words + 8, dtype=torch.int32, device="cuda")[s:s + z.words]
        gaps = torch.zeros(z.gap_words + 8, dtype=torch.int32, device="cuda")[s:s + z.gap_words]
        bits.copy_(torch.from_numpy(bits_o.view(np.int32)))
        gaps.copy_(torch.from_numpy(gaps_o.view(np.int32)))
        for o in outs:
            out = torch.full((x.size + 64,), 0x5A, dtype=torch.uint8, device="cuda")
            y = dec.decode(bits, gaps, z, book, x.size, out=out[o:])
            assert np.array_equal(y.cpu().numpy(), x), (x.size, s, o)
            rest = out.cpu().numpy()
            assert (rest[:o] == 0x5A).all() and (rest[o + x.size:] == 0x5A).all()


@pytest.mark.parametrize("kind", sorted(KINDS))
@pytest.mark.parametrize("segments", [1, 2, 31, 32, 33, 63, 64, 65, 255, 256, 257, 511, 512, 513, 1025, 5000])
def test_stream_lengths(kind, segments):
    p = np.array(KINDS[kind])
    per_seg = 128 / -(p * np.log2(p)).sum()
    for d in (-0.6, 0.0, 0.4):
        n = max(1, int((segments + d) * per_seg))
        _check_single(_data(kind, n, segments), outs=(0, 5))


@pytest.mark.parametrize("kind", sorted(KINDS))
def test_alignments(kind):
    _check_single(_data(kind, 30011, 7), shifts=(0, 1, 2, 3), outs=range(16))


@pytest.mark.parametrize("short", [0, 1])
def test_two_level_tables(short):
    x = _wide(short)
    assert O.codebook(O.histogram(x)).lengths.max() > 12
    _check_single(x, shifts=(0, 1), outs=(0, 9))


@pytest.mark.parametrize("tile", [0, 256, 512])
def test_batch_of_all_kinds(tile):
    xs = [_data(k, n, 11 * i + n) for i, k in enumerate(sorted(KINDS)) for n in (1, 100, 4097, 20000, 300001)]
    xs += [_wide(0), _wide(1), np.full(5000, 9, np.uint8)]
    ins = [torch.from_numpy(x).cuda() for x in xs]
    whole = torch.full((sum(x.size for x in xs) + len(xs),), 0x5A, dtype=torch.uint8, device="cuda")
    outs, at = [], 0
    for x in xs:  # packed one byte apart: every output alignment
        outs.append(whole[at:at + x.size])
        at += x.size + 1
    plan = B.BatchCodec([x.size for x in xs], B.LaunchConfig(dec_tile_segs=tile))
    plan.bind(ins, outs)
    plan.compress()
    for _ in range(2):
        whole.fill_(0x5A)
        plan.decompress()
        plan.check()
        for x, o in zip(xs, outs):
            assert np.array_equal(o.cpu().numpy(), x)
        assert int((whole == 0x5A).sum()) >= len(xs)


@pytest.mark.parametrize("kind", ["len1", "len2", "len3", "len8"])
def test_wrong_gap_entry_is_found(kind):
    x = _data(kind, 100000, 3)
    bits, gaps, _ = O.encode(x, O.codebook(O.histogram(x)))
    book, z = H.Codebook.from_histogram(O.histogram(x))
    for k in (0, 30, 31, 32, 255, 256, 511, 512, z.segments - 2):
        bad = gaps.copy()
        bad[k >> 3] ^= np.uint32(1 << (4 * (k & 7)))
        with pytest.raises(HgapError) as e:
            H.Decoder(z.segments).decode(torch.from_numpy(bits.view(np.int32)).cuda(),
                                         torch.from_numpy(bad.view(np.int32)).cuda(), z, book, x.size)
        assert e.value.status in (4, 5), k
