"""Windows near the longest that DTW takes (both windows of a pair lie in
shared memory): the longest give the oracle's result, longer ones are refused.
Tolerances of the pair and join tests: FP64 1e-10, FP32 2e-4, joins 1e-5."""
import numpy as np
import pytest

FP64_MAX, FP32_MAX = 12665, 25461  # w = 20: two cells per lane, one pair per warp


@pytest.mark.parametrize("m,precise", [(FP64_MAX + 1, True), (FP64_MAX + 900, True),
                                       (FP32_MAX + 1, False), (63488, False)])
def test_pair_lists_refuse_windows_that_do_not_fit(dtwj, m, precise):
    x = np.arange(2.0 * m + 10) % 97
    with pytest.raises(dtwj.DtwjError) as e:
        dtwj.pair_dtw(x, m, 20, [0], [5], precise=precise)
    assert e.value.code == dtwj.ERR_ARG


@pytest.mark.gpu
@pytest.mark.parametrize("m,precise,rtol", [(FP64_MAX, True, 1e-10), (6000, True, 1e-10),
                                            (FP32_MAX, False, 2e-4), (12000, False, 2e-4)])
def test_longest_pair_lists(gpu_dtwj, oracle, synth, m, precise, rtol):
    x = synth.random_walk(2 * m + 41, m)
    pi, pj = np.array([0, 7, 41]), np.array([m, m + 20, m + 41])
    got = gpu_dtwj.pair_dtw(x, m, 20, pi, pj, precise=precise)
    ref = [oracle.pair_dist(x, m, 20, int(i), int(j)) for i, j in zip(pi, pj)]
    np.testing.assert_allclose(got, ref, rtol=rtol)


@pytest.mark.gpu
def test_longest_join(gpu_dtwj, oracle, synth):
    m = FP64_MAX
    x = synth.random_walk(2 * m + 41, 4)
    ref = oracle.join(x, m, 20)
    with gpu_dtwj.Context() as ctx:
        for _ in range(2):
            r = ctx.join(x, m, 20)
            assert (r.i, r.j) == (ref.i, ref.j)
            assert abs(r.dist - ref.dist) <= 1e-5 * ref.dist
            with pytest.raises(gpu_dtwj.DtwjError) as e:
                ctx.join(x, m + 1, 20)
            assert e.value.code == gpu_dtwj.ERR_ARG
