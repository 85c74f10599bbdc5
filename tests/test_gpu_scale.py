"""Joins do not depend on the units of the series: z-normalisation cancels a
scale, and a power of two cancels exactly in FP64.  The FP32 copies and
reciprocal deviations of the bounds do not hold every scale (2^149 and beyond:
1 / deviation rounds to zero), so at both ends the join must still be
the unscaled series' by the oracle: indices exact, distance within 1e-5
relative (the tolerance of the join tests)."""
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
