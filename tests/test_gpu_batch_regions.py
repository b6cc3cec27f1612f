"""Batched compress without a region size: the library takes 8, 16 or 32 chunks a region by the number of
regions that the workspace holds.  The streams do not depend on it."""
import numpy as np
import pytest
import torch

from huffman_coding_gap_arrays_b200 import batch as B

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("regions", [0, 5919, 5920, 23679, 23680])
def test_streams_do_not_depend_on_the_workspace(regions):
    sizes = [1, 65535, 65536, 131072 + 17, 262144, 1000003, 3000000]
    r = np.random.default_rng(5)
    whole = torch.from_numpy(np.minimum(r.geometric(0.1, sum(sizes) + 32), 255).astype(np.uint8)).cuda()
    ins, at = [], 0
    for n in sizes:  # at every alignment
        ins.append(whole[at:at + n])
        at += n
    outs = [torch.full((n,), 0x5A, dtype=torch.uint8, device="cuda") for n in sizes]
    ref = B.BatchCodec(sizes, B.LaunchConfig(region_chunks=8), inputs=ins)
    ref.compress()
    plan = B.BatchCodec(sizes, inputs=ins, outputs=outs)
    # room for that many regions of 8 + 80 + 1024 bytes beside what the buffers need
    plan.enc_ws = torch.empty((plan.enc_ws.numel() * 8 + 1112 * regions) // 8, dtype=torch.int64, device="cuda")
    plan.compress()
    plan.decompress()
    plan.check()
    for i, (x, o) in enumerate(zip(ins, outs)):
        assert torch.equal(o, x)
        a, b = ref.stream(i), plan.stream(i)
        assert torch.equal(a.bits, b.bits) and torch.equal(a.gaps, b.gaps)
