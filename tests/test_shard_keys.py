"""The order in which tracks are dealt to ranks is the batched form's queue
order: the keys of csrc/kf_batch.cu's workKey, written out by hand."""
import numpy as np


def test_work_keys_are_the_queues(kf):
    from gpukalmanfitter_gb300 import shard
    # (length, q/p, clamped length, quarter octaves above 2^-7)
    rows = [(30, 1.0, 30, 28), (30, -1.0, 30, 28), (5, 0.5, 5, 24), (5, 0.6, 5, 25), (12, -0.7071, 12, 25),
            (12, 2.0 ** -7, 12, 0), (12, 0.008, 12, 0), (0, 0.1, 1, 14), (-3, 0.1, 1, 14), (40, 0.1, 30, 14),
            (7, 100.0, 7, 31), (7, 0.0, 7, 0), (7, np.inf, 7, 0), (7, np.nan, 7, 0), (7, 3.2e38, 7, 0),
            (7, 1e300, 7, 0), (7, 1e-30, 7, 0)]
    length, qop, L, qb = map(np.array, zip(*rows))
    keys = shard.work_keys(length.astype(np.int32), qop, 30)
    assert np.array_equal(keys, (64 - L) * 32 + (31 - qb))
    assert np.array_equal(shard.work_keys(None, qop, 30), (64 - 30) * 32 + (31 - qb))
