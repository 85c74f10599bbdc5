"""The MLP's batch kernels (column sums in blocks of 64 rows, GEMM tiles of 128
rows and K stages of 64, split K from 1024 rows on) at batch sizes around their
edges, against the FP64 restatement: the FP32 path within 1e-4 per parameter
block, the BF16 path within 1e-2 of the restatement with its operands rounded
(the tolerances of the gradient tests)."""
import numpy as np
import pytest

import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 63, 64, 65, 127, 129, 1023, 1024, 1089, 8191, 8192])
def test_gradient_at_the_edges_of_the_batch_tiles(gpu_dtwj, rows):
    rng = np.random.default_rng(rows)
    x = rng.normal(0.0, 1.0, (rows, mlp_ref.IN)).astype(np.float32)
    y = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2]).astype(np.float32)
    net = gpu_dtwj.MLP(seed=11)
    p = net.params
    for precise, tol in ((True, 1e-4), (False, 1e-2)):
        ref, ref_loss = mlp_ref.grad(p, x, y, bf16_operands=not precise)
        g, loss = net.grad(x, y, precise=precise)
        gb, rb = mlp_ref.blocks(g), mlp_ref.blocks(ref)
        for k in rb:
            err = np.linalg.norm(gb[k] - rb[k]) / max(np.linalg.norm(rb[k]), 1e-30)
            assert err <= tol, (precise, k, err)
        assert loss == pytest.approx(ref_loss, rel=1e-3)
