"""A batch decodes books whose shortest code has 2 bits in tiles of 480 segments: streams that end around one
(and, one by one, in tiles of 512)."""
import numpy as np
import pytest
import torch

from huffman_coding_gap_arrays_b200 import batch as B
from test_gpu_decode_edges import KINDS, _check_single, _data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments", [447, 448, 449, 479, 480, 481, 959, 960, 961, 4800])
def test_tile_edges(segments):
    p = np.array(KINDS["len2"])
    per_seg = 128 / -(p * np.log2(p)).sum()
    xs = [_data("len2", int((segments + d) * per_seg), segments) for d in (-0.6, 0.0, 0.4)]
    for x in xs:
        _check_single(x, shifts=(0, 1), outs=(0, 5))
    xs.append(_data("len2", 400000, 1))  # (over 64 KiB a buffer on the average: not the small batch's tiles)
    ins = [torch.from_numpy(x).cuda() for x in xs]
    for tile in (0, 512):
        outs = [torch.full((x.size,), 0x5A, dtype=torch.uint8, device="cuda") for x in xs]
        plan = B.BatchCodec([x.size for x in xs], B.LaunchConfig(dec_tile_segs=tile), inputs=ins, outputs=outs)
        plan.compress()
        plan.decompress()
        plan.check()
        for x, o in zip(ins, outs):
            assert torch.equal(o, x)
