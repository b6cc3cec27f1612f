"""The encoder's plan of more regions than its grid takes at once, beside other work: on two streams at the same
time, and while another kernel holds most of the places that its CTAs would take."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

import huffman_coding_gap_arrays_b200 as H
from huffman_coding_gap_arrays_b200 import _lib
from huffman_coding_gap_arrays_b200 import batch as B

pytestmark = pytest.mark.gpu

COUNT = 30_000  # buffers of one region or two: at eight regions a CTA, more than 148 SMs hold CTAs of 256 threads
TIMEOUT = 3


def _batch(seed):
    rng = np.random.default_rng(seed)
    sizes = rng.integers(1, 200, COUNT)
    sizes[rng.integers(0, COUNT, 300)] = rng.integers(8000, 20_000, 300)
    at = np.concatenate([[0], np.cumsum(sizes)])
    data = torch.from_numpy(np.minimum(rng.geometric(0.1, int(at[-1])) - 1, 255).astype(np.uint8)).cuda()
    back = torch.zeros_like(data)
    plan = B.BatchCodec(sizes, B.LaunchConfig(region_chunks=1), inputs=[data[a:b] for a, b in zip(at, at[1:])],
                        outputs=[back[a:b] for a, b in zip(at, at[1:])])
    return plan, data, back


def test_two_streams():
    assert COUNT > 8 * 8 * 148
    batches = [_batch(s) for s in (1, 2)]
    streams = [torch.cuda.Stream() for _ in batches]
    torch.cuda.synchronize()
    for _ in range(5):
        for (plan, _, back), s in zip(batches, streams):
            with torch.cuda.stream(s):
                back.zero_()
                plan.compress()
                plan.decompress()
        for (plan, data, back), s in zip(batches, streams):
            with torch.cuda.stream(s):
                plan.check()
                assert torch.equal(back, data)


def test_beside_a_kernel_that_holds_sms():
    plan, data, back = _batch(3)
    plan.compress()  # (warm: nothing is loaded or allocated below)
    plan.decompress()
    plan.check()
    # another stream: a plan of 256 MiB whose first group withholds its record, so that the CTAs of all
    # others wait, one on nearly every SM (more would leave no room for the batch's largest CTAs)
    n = 1 << 28
    x = torch.randint(0, 250, (n,), dtype=torch.uint8, device="cuda")
    book, sizes = H.Codebook.from_histogram(H.histogram(x).cpu())
    enc = H.Encoder(n)
    bits = torch.empty(sizes.words, dtype=torch.int32, device="cuda")
    gaps = torch.empty(sizes.gap_words, dtype=torch.int32, device="cuda")
    ws = enc.workspace
    side, done = torch.cuda.Stream(), torch.cuda.Event()
    torch.cuda.synchronize()
    L = _lib.lib()
    assert L.hgap_encode_hold(x.data_ptr(), n, C.byref(book.cstruct), bits.data_ptr(), sizes.words, gaps.data_ptr(),
                              sizes.segments, ws.data_ptr(), ws.numel() * 8, C.c_void_p(side.cuda_stream), 0,
                              1_500_000_000) == 0
    done.record(side)
    time.sleep(0.1)
    back.zero_()
    plan.compress()
    plan.check_compress()
    assert not done.query()  # the other plan still holds its places
    plan.decompress()
    plan.check_decompress()
    assert torch.equal(back, data)
    assert L.hgap_workspace_status(ws.data_ptr(), C.c_void_p(side.cuda_stream)) == TIMEOUT
