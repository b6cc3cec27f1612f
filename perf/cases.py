"""The calls this library is used for, as cases that can be timed and compared.

A case names a way of calling (`path`), a direction (`dir`), a size and a
byte distribution:

* path "call"  -- one buffer through ``codec.compress`` / ``codec.decompress``:
                  everything allocated and checked inside the call, as a
                  program does that meets a new buffer now and then;
* path "kept"  -- one buffer through a kept ``Encoder`` (with a codebook the
                  program already has) or a kept ``Decoder`` and output buffer;
* path "batch" -- many buffers, each with its own codebook, through a kept
                  ``BatchCodec``: as plain calls with the status read after
                  each, or (`graph`) as the replay of a captured CUDA graph.

Every output is returned whole: bitstream, gap array and codebook (for a
batch: both arenas and all entries), or the decoded bytes.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

from huffman_coding_gap_arrays_b200 import batch as B
from huffman_coding_gap_arrays_b200 import codec
from huffman_coding_gap_arrays_b200 import workloads as WL

KiB, MiB = 1 << 10, 1 << 20


def listed():
    return [
        # a short message: latency of one whole compress call; odd size, unaligned input
        dict(name="call_compress_4k", path="call", dir="compress", n=4099, dist="zipf", param=1.2, offset=3),
        # a small payload on the way in: latency of one whole decompress call
        dict(name="call_decompress_64k", path="call", dir="decompress", n=65537, dist="gauss", param=2.5, offset=0),
        # an ordinary file of skewed bytes, both directions
        dict(name="call_compress_16m", path="call", dir="compress", n=16 * MiB, dist="zipf", param=1.2, offset=0),
        dict(name="call_decompress_16m", path="call", dir="decompress", n=16 * MiB, dist="zipf", param=1.2, offset=0),
        # the largest single buffer: a GiB of blocks of two kinds, nearly incompressible together
        dict(name="call_compress_1g", path="call", dir="compress", n=1024 * MiB, dist="mixed", param=0.0, offset=0),
        dict(name="call_decompress_1g", path="call", dir="decompress", n=1024 * MiB, dist="mixed", param=0.0,
             offset=0),
        # tensor bytes: the sign|mantissa plane of BF16 weights (near-uniform bytes) encoded with a
        # codebook that is kept, and the exponent plane (very short codes) decoded
        dict(name="kept_encode_mantissa", path="kept", dir="compress", n=256 * MiB, dist="bf16_mantissa", param=0.0,
             offset=0),
        dict(name="kept_decode_exponent", path="kept", dir="decompress", n=256 * MiB, dist="bf16_exponent",
             param=0.0, offset=0),
        # thousands of buffers of uneven size and kind: the throughput workload, replayed as graphs
        dict(name="batch_compress_mix", path="batch", dir="compress", count=4096, lo=4 * KiB, hi=4 * MiB, align=256,
             graph=True),
        dict(name="batch_decompress_mix", path="batch", dir="decompress", count=4096, lo=4 * KiB, hi=4 * MiB,
             align=256, graph=True),
        # thousands of small buffers, packed without alignment: per-buffer work counts
        dict(name="batch_compress_small", path="batch", dir="compress", count=4096, lo=4 * KiB, hi=64 * KiB, align=1,
             graph=False),
        dict(name="batch_decompress_small", path="batch", dir="decompress", count=4096, lo=4 * KiB, hi=64 * KiB,
             align=1, graph=False),
    ]


def _log_uniform(rng: random.Random, lo: float, hi: float) -> int:
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng: random.Random):
    case = dict(path=rng.choice(["call", "call", "kept", "batch", "batch"]), dir=rng.choice(["compress", "decompress"]))
    if case["path"] == "batch":
        lo = _log_uniform(rng, 1 * KiB, 64 * KiB)
        hi = _log_uniform(rng, 2 * lo, 4 * MiB)
        mean = (hi - lo) / math.log(hi / lo)
        case.update(count=_log_uniform(rng, 8, min(4096, 2 ** 31 / mean)), lo=lo, hi=hi,
                    align=rng.choice([256, 16, 1]), graph=rng.random() < 0.5)
        return case
    dist = rng.choice(["zipf", "gauss", "mixed", "bf16_mantissa", "bf16_exponent"])
    param = {"zipf": round(rng.uniform(0.8, 1.6), 3), "gauss": round(rng.uniform(0.5, 4.0), 3)}.get(dist, 0.0)
    lo = 1 * KiB if case["path"] == "call" else 1 * MiB
    case.update(n=_log_uniform(rng, lo, 256 * MiB), dist=dist, param=param, offset=rng.choice([0, 0, rng.randrange(16)]))
    return case


# ------------------------------------------------------------------- inputs ---

def _gauss(n: int, sigma: float, device) -> torch.Tensor:
    g = torch.Generator(device=device)
    g.manual_seed(n)
    z = torch.randn(n, generator=g, device=device, dtype=torch.float32)
    return torch.round(128.0 + sigma * z).clamp_(0, 255).to(torch.uint8)


def _bytes(case, seed: int, device="cuda") -> torch.Tensor:
    """One buffer.  The draws depend on the size alone; the seed then renames the byte values and
    turns the buffer round.  So the counts come in another order for every seed, and with them the
    codebook and every code, while their sum of code bits -- the size of the result -- stays."""
    n, dist = case["n"], case["dist"]
    if dist == "zipf":
        x = WL.zipf_buffer(n, case["param"], n, device)
    elif dist == "gauss":
        x = _gauss(n, case["param"], device)
    elif dist == "mixed":
        x = WL.mixed_buffer(n, n, device=device)
    else:
        x = WL.bf16_planes(n, n, device)[0 if dist == "bf16_exponent" else 1]
    g = torch.Generator(device="cpu")
    g.manual_seed(seed)
    names = torch.randperm(256, generator=g).to(torch.uint8).to(device)
    turn = int(torch.randint(n, (1,), generator=g))
    x = torch.roll(names[x.int()], turn)
    if case["offset"]:  # a view into a larger buffer, at any byte address
        whole = torch.empty(n + 16, dtype=torch.uint8, device=device)
        view = whole[case["offset"]:case["offset"] + n]
        view.copy_(x)
        x = view
    return x


def _slices(sizes, align: int, device="cuda"):
    """One buffer of zeros and a view of it for each size, each starting at a multiple of `align`."""
    at, offsets = 0, []
    for n in sizes:
        at = -(-at // align) * align
        offsets.append(at)
        at += n
    whole = torch.zeros(at, dtype=torch.uint8, device=device)
    return whole, [whole[o:o + n] for o, n in zip(offsets, sizes)]


def _batch_sizes(case):
    return WL.batch_sizes(case["count"], case["lo"], case["hi"])


def _prepare_batch(case, seed: int):
    sizes = _batch_sizes(case)
    _, ins = _slices(sizes, case["align"])
    for j, (v, n) in enumerate(zip(ins, sizes)):
        v.copy_(WL.batch_buffer(n, seed * 1000003 + j))
    out, outs = _slices(sizes, case["align"])
    plan = B.BatchCodec(sizes)
    plan.bits.zero_()  # what no stream covers stays as it is
    plan.gaps.zero_()
    plan.bind(ins, outs)
    plan.compress()
    if case["dir"] == "decompress":
        plan.decompress()
    plan.check_compress()
    graph = None
    if case["graph"]:
        graph = plan.capture(compress=case["dir"] == "compress", decompress=case["dir"] == "decompress")
    if case["dir"] == "decompress":
        out.zero_()
    else:
        plan.bits.zero_()
        plan.gaps.zero_()
        plan.entries.zero_()
    return dict(case=case, plan=plan, graph=graph, out=out)


def prepare(case, seed: int):
    if case["path"] == "batch":
        return _prepare_batch(case, seed)
    x = _bytes(case, seed)
    state = dict(case=case, x=x)
    if case["path"] == "kept" and case["dir"] == "compress":
        book, sizes = codec.Codebook.from_histogram(codec.histogram(x).cpu())
        state.update(encoder=codec.Encoder(x.numel()), book=book, sizes=sizes,
                     bits=torch.zeros(sizes.words, dtype=torch.int32, device="cuda"),
                     gaps=torch.zeros(sizes.gap_words, dtype=torch.int32, device="cuda"))
    elif case["dir"] == "decompress":
        c = codec.compress(x)
        state["x"] = None
        state["stream"] = c
        if case["path"] == "kept":
            whole = torch.zeros(x.numel() + 16, dtype=torch.uint8, device="cuda")
            state.update(decoder=codec.Decoder(c.sizes.segments), out=whole[case["offset"]:case["offset"] + x.numel()])
    return state


# ---------------------------------------------------------------------- run ---

def run(state):
    case = state["case"]
    if case["path"] == "batch":
        plan = state["plan"]
        if case["dir"] == "compress":
            if state["graph"] is not None:
                state["graph"].replay()
            else:
                plan.compress()
                plan.check_compress()
            return plan.entries, plan.bits, plan.gaps
        if state["graph"] is not None:
            state["graph"].replay()
        else:
            plan.decompress()
            plan.check_decompress()
        return state["out"]
    if case["path"] == "call":
        if case["dir"] == "compress":
            c = codec.compress(state["x"])
            return c.bits, c.gaps, np.frombuffer(c.book.cstruct, np.uint8)
        return codec.decompress(state["stream"])
    if case["dir"] == "compress":
        return state["encoder"].encode(state["x"], state["book"], state["sizes"], bits=state["bits"],
                                       gaps=state["gaps"])
    c = state["stream"]
    return state["decoder"].decode(c.bits, c.gaps, c.sizes, c.book, c.n, out=state["out"])


# --------------------------------------------------------------------- work ---

def _entropy(p) -> float:
    p = np.asarray(p, np.float64)
    p = p[p > 0] / p.sum()
    return max(1.0, float(-(p * np.log2(p)).sum()))  # a code has at least one bit


def _normal(edges) -> np.ndarray:
    return np.diff([0.5 * (1.0 + math.erf(e / math.sqrt(2.0))) for e in edges])


def _zipf_p(s: float) -> np.ndarray:
    p = np.arange(1, 257, dtype=np.float64) ** -s
    return p / p.sum()


def _gauss_p(sigma: float) -> np.ndarray:
    return _normal([-40.0] + [(k - 128 + 0.5) / sigma for k in range(255)] + [40.0])


@functools.lru_cache(maxsize=None)
def _bits_per_byte(dist: str, param: float) -> float:
    if dist == "zipf":
        return _entropy(_zipf_p(param))
    if dist == "gauss":
        return _entropy(_gauss_p(param))
    if dist == "mixed":  # half Zipf(1.05), half N(0, 1) clamped to +-3 sigma over 0..255, one codebook
        g = _normal([-40.0] + [(k + 0.5) / 255.0 * 6.0 - 3.0 for k in range(255)] + [40.0])
        return _entropy(0.5 * _zipf_p(1.05) + 0.5 * g)
    if dist == "bf16_exponent":  # |x| in [2^k, 2^(k+1)) of N(0, 0.02)
        cdf = [math.erf(2.0 ** k / 0.02 / math.sqrt(2.0)) for k in range(-40, 2)]
        return _entropy(np.diff([0.0] + cdf))
    if dist == "batch":  # half Zipf(s in [0.8, 1.6]), half Gaussian(sigma in [0.5, 4])
        a = (np.arange(64) + 0.5) / 64
        return float(np.mean([0.5 * _entropy(_zipf_p(0.8 + 0.8 * v)) + 0.5 * _entropy(_gauss_p(0.5 + 3.5 * v))
                              for v in a]))
    return 8.0  # sign and mantissa bits: nearly uniform


def work(case):
    """Raw bytes on one side; on the other the bitstream at the distribution's entropy and its gap
    array (4 bits for every 128)."""
    if case["path"] == "batch":
        n, bits = sum(_batch_sizes(case)), _bits_per_byte("batch", 0.0)
    else:
        n, bits = case["n"], _bits_per_byte(case["dist"], case["param"])
    return {"bytes": n + n * bits / 8 * (1 + 1 / 32), "flops": 0}
