"""The shape that the learned tuner and the server keep when nothing is predicted better is the library's own
(no GPU): regions by the batch, which the networks see as the region size that it stands for."""
import numpy as np
import pytest

from huffman_coding_gap_arrays_b200 import mlp as M
from huffman_coding_gap_arrays_b200 import tuner as T
from huffman_coding_gap_arrays_b200.batch import LaunchConfig

LIBRARY = LaunchConfig(region_chunks=0)


def _features(regions, count):
    return np.array([np.log2((regions - count / 2) * 65536), 4.0, 13.0, 0.0, np.log2(count)], np.float32)


class _Net:
    """Compress time grows with the distance of the region size from `best` (log2), decompress time is flat."""

    def __init__(self, best):
        self.best = best

    def predict(self, X):
        X = np.asarray(X, np.float64)
        return np.stack([0.2 * np.abs(X[:, 5] - self.best), np.zeros(len(X))], axis=1)


@pytest.mark.parametrize("regions,chunks", [(3000, 8), (5800, 8), (6000, 16), (23000, 16), (24000, 32), (100_000, 32)])
@pytest.mark.parametrize("count", [1, 64, 2048])
def test_zero_is_seen_as_what_it_stands_for(regions, chunks, count):
    f = _features(regions, count)
    assert T.default_chunks(f) == chunks
    assert M.config_vector(LIBRARY, f)[0] == np.log2(chunks)
    assert np.array_equal(M.config_vector(LIBRARY, f)[1:], M.config_vector(LaunchConfig(), f)[1:])


@pytest.mark.parametrize("regions,chunks", [(3000, 8), (12_000, 16), (100_000, 32)])  # (features are rounded to 1/8)
def test_kept_unless_another_is_predicted_faster(regions, chunks):
    for best in (8, 16, 32):
        t = M.LearnedTuner([_Net(np.log2(best))])
        assert t.default == LIBRARY
        assert t.choose(_features(regions, 64)).region_chunks == (0 if best == chunks else best)


def test_autotuner_space_may_hold_the_default():
    r = T.Record(_features(24000, 64), LIBRARY, 1.0, float("nan"))
    X, _ = M.records_to_xy([r])
    assert X.shape == (1, 10) and X[0, 5] == 5.0


@pytest.mark.parametrize("error,kept", [(0.0, False), (0.1, False), (0.3, True)])
def test_a_gain_below_the_held_out_error_is_no_reason(error, kept):
    """The network predicts 0.2 (log) between two region sizes; its held-out records say +- `error`."""
    f = _features(3000, 64)
    t = M.LearnedTuner([_Net(4.0)])  # 16 chunks best, the default stands for 8
    recs = []
    for i, r in enumerate((1, 2, 4, 8, 16, 32)):
        cfg = LaunchConfig(region_chunks=r)
        p = float(t.predict(np.concatenate([f, M.config_vector(cfg, f)])[None])[0, 0])
        recs.append(T.Record(f, cfg, float(np.exp(p + (error if i % 2 else -error))), float("nan")))
    mean = np.mean([np.log(r.compress_ms) for r in recs])
    net = _Net(4.0)
    net.predict = lambda X, g=_Net(4.0).predict: g(X) - np.array([mean, 0.0])  # targets are relative to their mean
    t = M.LearnedTuner([net])
    t.hold_out(recs)
    assert abs(t.holdout_rmse - error) < 1e-6 and t.dec_margin == 0.05
    assert abs(t.margin - max(0.03, 1 - np.exp(-error))) < 1e-6
    assert t.choose(f).region_chunks == (0 if kept else 16)
