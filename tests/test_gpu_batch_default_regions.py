"""Batched compress without a region size: 8, 16 or 32 chunks by the regions of 8 chunks that the batch itself
has, on both sides of each limit, whatever the workspace would hold."""
import numpy as np
import pytest
import torch

from huffman_coding_gap_arrays_b200 import batch as B

pytestmark = pytest.mark.gpu

LARGE = 1 << 20  # 16 regions of 8 chunks, 8 of 16, 4 of 32
NITEMS = 64 // 8  # the region count's place in the workspace


@pytest.mark.parametrize("room", [0, 100_000])
@pytest.mark.parametrize("regions,chunks", [(17, 8), (5919, 8), (5920, 16), (23679, 16), (23680, 32)])
def test_by_the_batch(regions, chunks, room):
    count = regions - 16  # buffers of one region, empty ones, and the large one
    rng = np.random.default_rng(regions)
    sizes = np.concatenate([rng.integers(1, 48, count), np.zeros(count // 9, np.int64), [LARGE]])
    sizes = sizes[rng.permutation(sizes.size)]
    at = np.concatenate([[0], np.cumsum((sizes + 15) & ~15)])
    data = torch.from_numpy(np.minimum(rng.geometric(0.1, int(at[-1]) + 16), 255).astype(np.uint8)).cuda()
    ins = [data[a:a + n] for a, n in zip(at, sizes)]
    plan = B.BatchCodec(sizes, inputs=ins)
    # room for that many more regions of 8 + 80 + 1024 bytes
    plan.enc_ws = torch.empty(plan.enc_ws.numel() + 1112 * room // 8, dtype=torch.int64, device="cuda")
    plan.compress()
    plan.check_compress()
    assert int(plan.enc_ws[NITEMS]) == count + LARGE // (chunks * 8192)
    ref = B.BatchCodec(sizes, B.LaunchConfig(region_chunks=8), inputs=ins)
    ref.compress()
    ref.check_compress()
    assert int(ref.enc_ws[NITEMS]) == regions
    i = int(np.argmax(sizes))
    assert torch.equal(plan.entries, ref.entries)
    a, b = ref.stream(i), plan.stream(i)
    assert torch.equal(a.bits, b.bits) and torch.equal(a.gaps, b.gaps)
