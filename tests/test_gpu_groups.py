"""The group filter of the sweep (csrc/group.cu): joins whose windows, groups
and tiles end at odd places, and series on which it settles nothing (white
noise: every tile goes through the diagonal bound) or only part of the tiles,
against the oracle.  Tolerances of the join tests: indices exact, distance
within 1e-5 relative.  Every pair is counted once: the stage counters add up
to the pair count plus at most the seed DTWs (700 slots)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _series(synth, kind, n, seed):
    if kind == "walk":
        return synth.random_walk(n, seed)
    rng = np.random.default_rng(seed)
    if kind == "noise":
        return rng.standard_normal(n)
    if kind == "half":  # a walk, then noise: sparse and dense tiles in one join
        x = synth.random_walk(n, seed)
        x[n // 2:] = x[n // 2] + rng.standard_normal(n - n // 2)
        return x
    x = synth.random_walk(n, seed)  # "flat": stretches without any deviation
    x[n // 3:n // 3 + 200] = x[n // 3]
    x[n // 2:n // 2 + 700] = x[n // 2]
    return x


# m around the sizes where the group, the segment and the path change (8, 127,
# 128, 255, 256, 511, 512, 1024, 1025); n around one and two tiles of rows and lags
@pytest.mark.parametrize("kind,n,m,w,seed", [
    ("walk", 40, 8, 1, 1), ("walk", 1200, 8, 3, 2), ("walk", 900 + 2 * 127, 127, 6, 3),
    ("walk", 4033 + 128, 128, 7, 4), ("walk", 5003, 255, 13, 5), ("walk", 4032 + 2 * 256, 256, 3, 6),
    ("walk", 4999, 511, 26, 7), ("walk", 6001, 512, 52, 8), ("walk", 6007, 1024, 52, 9),
    ("walk", 4111, 1025, 20, 10), ("flat", 5001, 128, 7, 11), ("flat", 5001, 256, 13, 12),
    ("noise", 2500, 64, 4, 13), ("noise", 2100, 256, 3, 14), ("half", 6000, 128, 7, 15),
    ("half", 9000, 256, 3, 16)])
def test_join_with_group_filter_matches_oracle(gpu_dtwj, oracle, synth, kind, n, m, w, seed):
    x = _series(synth, kind, n, seed)
    ref = oracle.join(x, m, w)
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_NO_SEED, gpu_dtwj.F_MASKED_CASCADE, gpu_dtwj.F_NO_GRAPH):
            r = ctx.join(x, m, w, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= max(1e-5 * ref.dist, 1e-9), fl
            total = (r.pruned_fast + r.pruned_paa + r.pruned_kim + r.pruned_masked +
                     r.pruned_keogh + r.dtw_calls)
            assert 0 <= total - r.pairs <= 700, (fl, total, r.pairs)
