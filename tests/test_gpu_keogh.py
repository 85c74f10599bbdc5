"""The LB_Keogh stage's fine block means (csrc/runs.cu) at the window lengths
where their blocks change (255/256, 511/512, 1023/1024; 1025 has none), with
lengths off every multiple, on series that keep its queue empty, short and
long, against the oracle.  Tolerances of the join tests: indices exact,
distance within 1e-5 relative; every pair is counted once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n,m,w", [
    ("walk", 3000, 33, 3), ("ecg", 2500, 65, 4), ("ecg", 3000, 191, 10), ("ecg", 3000, 192, 10),
    ("walk", 4500, 255, 26), ("walk", 4500, 256, 26), ("ecg", 4000, 511, 52), ("walk", 6000, 513, 103),
    ("walk", 7000, 1023, 52), ("walk", 7000, 1024, 205), ("walk", 7000, 1025, 52)])
def test_fine_block_means_match_the_oracle(gpu_dtwj, oracle, synth, kind, n, m, w):
    # a large offset and scale: the FP32 copies are centered per block
    x = (synth.ecg_like if kind == "ecg" else synth.random_walk)(n, m + w) * 37.0 + 1e4
    ref = oracle.join(x, m, w)
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_NO_SEED, gpu_dtwj.F_MASKED_CASCADE):
            r = ctx.join(x, m, w, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= max(1e-5 * ref.dist, 1e-9), fl
            total = (r.pruned_fast + r.pruned_paa + r.pruned_kim + r.pruned_masked +
                     r.pruned_keogh + r.dtw_calls)
            assert 0 <= total - r.pairs <= 700, (fl, total, r.pairs)


def test_exact_bound_where_block_means_say_little(gpu_dtwj, oracle, synth):
    # half a walk, half noise: the fine block means stay far below LB_Keogh, which prunes
    # 72 of the 81 million pairs that reach it when it is tried on all; a third more DTWs
    # than that are allowed for the pairs that pass before the rule has seen enough
    x = synth.random_walk(30007, 7)
    x[15003:] = x[15003] + np.random.default_rng(7).standard_normal(15004)
    with gpu_dtwj.Context() as ctx:
        r = ctx.join(x, 700, 20)
        assert r.dtw_calls < (r.dtw_calls + r.pruned_keogh) * (1 - 72.0 / 81.0) * 4 / 3
        plain = ctx.join(x, 700, 20, gpu_dtwj.F_MASKED_CASCADE)
    assert (r.i, r.j) == (plain.i, plain.j) and abs(r.dist - plain.dist) <= 1e-9
