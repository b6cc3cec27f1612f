"""The encoder where a warp's 1 KiB has more code bits than its image in shared memory holds (348 words,
the first 8 slack), so that it packs its two halves one after the other: at a job's start, in its middle and at
its end, at every input alignment, as a single buffer, as a part of a split stream and in a packed batch.
Every case counts the bits of its warps first."""
import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import batch as B
from huffman_coding_gap_arrays_b200 import parallel as PL
from oracle import oracle as O

pytestmark = pytest.mark.gpu

WARP, STEP = 1024, 16384
ROOM = 348 * 32 - 256  # bits of a warp that never fit, wherever in a segment they start

# 1 to 9 bits, and 128 bytes of 16 bits: the longest codes, complete
DEEP_SYMBOLS = np.arange(60, 60 + 137, dtype=np.uint8)
DEEP_LENGTHS = np.array(list(range(1, 10)) + [16] * 128, np.uint8)
LONG = DEEP_SYMBOLS[9:]


def _warp_bits(x, length, off):
    """Code bits of each of the encoder's warps for x at an address 16 k + off."""
    b = np.concatenate([np.zeros(off, np.int64), length[x].astype(np.int64)])
    return np.add.reduceat(b, np.arange(0, b.size, WARP))


def _deep(n, rng, spans):
    """Short codes, and the longest ones in the given [start, end) spans."""
    x = DEEP_SYMBOLS[np.minimum(rng.geometric(0.5, n) - 1, 8)]
    for a, b in spans:
        x[a:b] = rng.choice(LONG, b - a)
    return x


def _at(x, off):
    """x on the device at an address 16 k + off, among bytes that it does not hold."""
    whole = torch.full((x.size + 48,), 255, dtype=torch.uint8, device="cuda")
    d = whole[off:off + x.size]
    d.copy_(torch.from_numpy(x))
    return d


def _sizes(bits_total):
    words = (bits_total + 31) // 32
    segs = (bits_total + 127) // 128
    return H.StreamSizes(bits_total, words, segs, (segs + 7) // 8)


CASES = {  # bytes, spans of 16-bit codes
    "first": (3 * WARP, [(0, WARP)]),
    "middle": (40 * WARP + 77, [(19 * WARP, 22 * WARP)]),
    "step ends": (3 * STEP, [(STEP - 2 * WARP, STEP + 2 * WARP)]),
    "last": (5 * WARP + 900, [(4 * WARP, 5 * WARP + 900)]),
    "alone": (900, [(0, 900)]),
    "first and last": (2 * WARP + 800, [(0, 2 * WARP + 800)]),
}


@pytest.mark.parametrize("where", sorted(CASES))
def test_kept_book(where):
    n, spans = CASES[where]
    x = _deep(n, np.random.default_rng(n), spans)
    book_o = O.codebook_from_list(DEEP_SYMBOLS, DEEP_LENGTHS)
    bits_o, gaps_o, total = O.encode(x, book_o)
    book, sizes = H.Codebook.from_symbols(DEEP_SYMBOLS, DEEP_LENGTHS), _sizes(total)
    enc = H.Encoder(n)
    for off in range(16):
        w = _warp_bits(x, book_o.length, off)
        assert w.max() > ROOM
        if "first" in where:
            assert w[0] > ROOM
        if where == "last":
            assert w[-1] > ROOM or w[-2] > ROOM
        bits, gaps = enc.encode(_at(x, off), book, sizes)
        assert np.array_equal(bits.cpu().numpy().view(np.uint32), bits_o), (where, off)
        assert np.array_equal(gaps.cpu().numpy().view(np.uint32), gaps_o), (where, off)


@pytest.mark.parametrize("short", [0, 20])
def test_records_of_two_steps_fill_their_ring(short):
    """Regions of 48 KiB whose steps of 16 KiB each close 2048 segments (or a few less, in a region's first step),
    where the ring of gap records holds 4096: gap words are written before the next records reach theirs."""
    region = 3 * STEP
    n = 12 << 20
    x = np.random.default_rng(short).choice(LONG, n)
    for i in range(short):
        x[100 + i::region] = DEEP_SYMBOLS[0]
    x = np.concatenate([x, LONG[:333]])
    book_o = O.codebook_from_list(DEEP_SYMBOLS, DEEP_LENGTHS)
    bits_o, gaps_o, total = O.encode(x, book_o)
    per_step = book_o.length[x[:n]].astype(np.int64).reshape(-1, STEP).sum(1) // 128
    two = per_step[0::3] + per_step[1::3]
    assert ((two >= 4096 - 8) & (per_step[0::3] == 2048 - (3 if short else 0))).all()
    assert (n + 333 + 15) // 8192 + 1 <= 296 * 6 and n > 296 * 5 * 8192  # one region a CTA, two CTAs on each of 148 SMs
    book, sizes = H.Codebook.from_symbols(DEEP_SYMBOLS, DEEP_LENGTHS), _sizes(total)
    enc = H.Encoder(x.size)
    for off in (0, 3, 15):
        bits, gaps = enc.encode(_at(x, off), book, sizes)
        assert np.array_equal(bits.cpu().numpy().view(np.uint32), bits_o), off
        assert np.array_equal(gaps.cpu().numpy().view(np.uint32), gaps_o), off


@pytest.mark.parametrize("cut", [1, 700, WARP + 5, 7 * WARP])
def test_parts_of_a_split_stream(cut):
    """The second part starts anywhere in a word, and with a warp that does not fit."""
    x = _deep(9 * WARP + 50, np.random.default_rng(cut), [(cut, cut + WARP), (8 * WARP, 9 * WARP + 50)])
    book_o = O.codebook_from_list(DEEP_SYMBOLS, DEEP_LENGTHS)
    bits_o, gaps_o, total = O.encode(x, book_o)
    book, sizes = H.Codebook.from_symbols(DEEP_SYMBOLS, DEEP_LENGTHS), _sizes(total)
    counts = [int(book_o.length[p].sum()) for p in (x[:cut], x[cut:])]
    for off in range(16):
        assert _warp_bits(x[cut:], book_o.length, off)[0] > ROOM
        windows = []
        for p, start, k in zip((x[:cut], x[cut:]), PL.part_starts(counts), counts):
            c, d = PL.DevicePartCodec(), _at(p, off)
            c.histogram(d)
            windows.append(c.encode(d, book, start, k))
        bits, gaps = PL.stitch_parts(windows, sizes.words, sizes.gap_words, torch.device("cuda"))
        assert np.array_equal(bits.cpu().numpy().view(np.uint32), bits_o), (cut, off)
        assert np.array_equal(gaps.cpu().numpy().view(np.uint32), gaps_o), (cut, off)


def _with_header(n, sigma, seed):
    """1 KiB of random bytes, then rounded N(128, sigma): a file whose header is unlike its body."""
    rng = np.random.default_rng(seed)
    body = np.clip(np.round(rng.normal(128, sigma, n)), 0, 255).astype(np.uint8)
    return np.concatenate([rng.integers(0, 256, WARP, dtype=np.uint8), body])


@pytest.mark.parametrize("n,sigma", [(64 << 10, 0.5), (64 << 10, 2.0), (200_000, 1.0), (4 << 20, 4.0)])
def test_header_unlike_the_body(n, sigma):
    x = _with_header(n, sigma, n)
    book_o = O.codebook(O.histogram(x))
    bits_o, gaps_o, _ = O.encode(x, book_o)
    for off in (0, 1, 3, 8, 15):
        assert _warp_bits(x, book_o.length, off)[0] > ROOM
        c = H.compress(_at(x, off))
        assert np.array_equal(c.bits.cpu().numpy().view(np.uint32), bits_o), off
        assert np.array_equal(c.gaps.cpu().numpy().view(np.uint32), gaps_o), off
        assert np.array_equal(H.decompress(c).cpu().numpy(), x), off


def test_packed_batch():
    xs = [_with_header(40_000 + 1001 * i, 0.5 + 0.2 * i, i) for i in range(16)]
    at = np.cumsum([0] + [x.size for x in xs])
    whole = torch.from_numpy(np.concatenate(xs)).cuda()
    back = torch.zeros_like(whole)
    books = [O.codebook(O.histogram(x)) for x in xs]
    offs = [int((whole.data_ptr() + a) & 15) for a in at[:-1]]
    assert sum(o != 0 for o in offs) >= 8
    assert all(_warp_bits(x, b.length, o)[0] > ROOM for x, b, o in zip(xs, books, offs))
    plan = B.BatchCodec([x.size for x in xs], inputs=[whole[a:b] for a, b in zip(at, at[1:])],
                        outputs=[back[a:b] for a, b in zip(at, at[1:])])
    plan.compress()
    plan.check_compress()
    for i, (x, b) in enumerate(zip(xs, books)):
        bits_o, gaps_o, _ = O.encode(x, b)
        s = plan.stream(i)
        assert np.array_equal(s.bits.cpu().numpy().view(np.uint32)[:bits_o.size], bits_o), (i, offs[i])
        assert np.array_equal(s.gaps.cpu().numpy().view(np.uint32)[:gaps_o.size], gaps_o), (i, offs[i])
    plan.decompress()
    plan.check()
    assert torch.equal(back, whole)
