"""A withheld look-back record under every shape of the decoder, with many tiles a CTA: every warp that
waits gives up together with its CTA, the kernel ends by itself within a small multiple of the waits' limit,
writes nothing outside the output, reports the timeout, and the workspace serves the next call."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import _lib

pytestmark = pytest.mark.gpu

TIMEOUT = 3
LIMIT_NS = 2_000_000
GUARD = 4096
# symbols' shares by the shortest code: 1, 2, 3 and 8 bits (pairs of symbols where codes are short, none at 8)
KINDS = {
    "len1": [0.7, 0.2, 0.06, 0.03, 0.01],
    "len2": [0.3, 0.3, 0.2, 0.1, 0.05, 0.03, 0.02],
    "len3": [0.2] * 3 + [0.1] * 2 + [0.2 / 40] * 40,
    "len8": [1 / 256] * 256,
}


@pytest.mark.parametrize("hold", [0, 1, 300, 1500])
@pytest.mark.parametrize("kind", sorted(KINDS))
def test_every_shape_ends_and_recovers(kind, hold):
    n = 128 << 20
    g = torch.Generator(device="cuda")
    g.manual_seed(hold)
    edges = torch.tensor(np.cumsum(KINDS[kind])[:-1], device="cuda", dtype=torch.float32)
    x = torch.bucketize(torch.rand(n, device="cuda", generator=g), edges).to(torch.uint8)
    book, sizes = H.Codebook.from_histogram(H.histogram(x).cpu())
    bits, gaps = H.Encoder(n).encode(x, book, sizes)
    assert sizes.segments > 512 * (hold + 500)  # tiles of at most 512 segments: many after the held one
    dec = H.Decoder(sizes.segments)
    whole = torch.full((n + 2 * GUARD,), 0x5A, dtype=torch.uint8, device="cuda")
    out = whole[GUARD:GUARD + n]
    L = _lib.lib()
    stream = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    ws = dec.workspace
    for _ in range(3):
        t0 = time.perf_counter()
        assert L.hgap_decode_hold(bits.data_ptr(), sizes.words, gaps.data_ptr(), sizes.segments, C.byref(book.cstruct),
                                  out.data_ptr(), n, ws.data_ptr(), ws.numel() * 8, stream, hold, LIMIT_NS) == 0
        assert L.hgap_workspace_status(ws.data_ptr(), stream) == TIMEOUT
        assert time.perf_counter() - t0 < 1.0
        assert bool((whole[:GUARD] == 0x5A).all()) and bool((whole[GUARD + n:] == 0x5A).all())
        y = dec.decode(bits, gaps, sizes, book, n, out=out)
        assert torch.equal(y, x)
