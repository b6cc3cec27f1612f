"""Batched decompress into buffers packed one byte apart, every book class and tile size among them: the byte
between two buffers keeps its value, compared place by place."""
import numpy as np
import pytest
import torch

from huffman_coding_gap_arrays_b200 import batch as B
from test_gpu_decode_edges import KINDS, _data, _wide

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", [0, 256, 512])
@pytest.mark.parametrize("guard", [0x00, 0x5A, 0xFF])
def test_bytes_between_the_buffers(tile, guard):
    xs = [_data(k, n, 3 * i + n) for i, k in enumerate(sorted(KINDS)) for n in (1, 15, 16, 17, 100, 4097, 20000, 300001)]
    xs += [_wide(0), _wide(1), np.full(5000, 9, np.uint8), np.full(1, 200, np.uint8)]
    xs = [xs[i] for i in np.random.default_rng(guard).permutation(len(xs))]
    ends = np.cumsum([x.size + 1 for x in xs]) - 1  # the byte behind each buffer
    whole = torch.empty(int(ends[-1]) + 1, dtype=torch.uint8, device="cuda")
    plan = B.BatchCodec([x.size for x in xs], B.LaunchConfig(dec_tile_segs=tile),
                        inputs=[torch.from_numpy(x).cuda() for x in xs],
                        outputs=[whole[e - x.size:e] for e, x in zip(ends, xs)])
    plan.compress()
    for _ in range(2):
        whole.fill_(guard)
        plan.decompress()
        plan.check()
        host = whole.cpu().numpy()
        assert (host[ends] == guard).all()
        for e, x in zip(ends, xs):
            assert np.array_equal(host[e - x.size:e], x)
