"""Joins do not depend on the units of the series: z-normalisation cancels a
scale, and a power of two cancels exactly in FP64.  The FP32 copies and
reciprocal deviations of the bounds do not hold every scale (2^149 and beyond:
1 / deviation rounds to zero; 2^-127 and below: the samples lose bits, then
1 / deviation overflows), so at both ends the join must still be the unscaled
series' by the oracle: indices exact, distance within 1e-5 relative (the
tolerance of the join tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N, M, W = 20011, 256, 25


@pytest.fixture(scope="module")
def walk(oracle, synth):
    x = synth.random_walk(N, 5)
    return x, oracle.join(x, M, W)


# a scale of 1e50 as an input may have it, then powers of two around 2^127 (the
# largest FP32 value) and 2^149 (the reciprocal of the smallest)
@pytest.mark.parametrize("scale", [1e50] + [2.0 ** e for e in (126, 128, 148, 150, 152, 160, 480)])
def test_join_of_large_values(gpu_dtwj, walk, scale):
    x, ref = walk
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_NO_SEED, gpu_dtwj.F_MASKED_CASCADE):
            r = ctx.join(x * scale, M, W, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= 1e-5 * ref.dist, fl


# the smallest normal FP32 value is 2^-126, the smallest 2^-149
@pytest.mark.parametrize("e", [-100, -126, -128, -140, -145, -150, -480])
@pytest.mark.parametrize("m,w", [(256, 25), (1100, 20)])  # both copies of the block means
def test_join_of_small_values(gpu_dtwj, oracle, walk, e, m, w):
    x, ref = walk
    if m != M:
        ref = oracle.join(x, m, w)
    with gpu_dtwj.Context() as ctx:
        for fl in (0, gpu_dtwj.F_NO_SEED):
            r = ctx.join(x * 2.0 ** e, m, w, fl)
            assert (r.i, r.j) == (ref.i, ref.j), fl
            assert abs(r.dist - ref.dist) <= 1e-5 * ref.dist, fl
