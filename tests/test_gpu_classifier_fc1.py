"""FC1 weight gradient at batch sizes around its 64-sample stages and their
quarters, and the convolutions' data gradients behind it, against the CPU
network with the same rounding points."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu

CONV = sum(co * ci * 9 + co for ci, co in ((1, 8), (8, 16), (16, 32))) * 2
FC1 = 16 * 10240


@pytest.mark.parametrize("n", [2, 15, 33, 64, 65])
def test_fc1_gradient_matches_oracle(hdb, oracle_lib, n):
    rng = np.random.default_rng(200 + n)
    dm = rng.standard_normal((n, 64, 64)).astype(np.float32)
    ft = rng.standard_normal((n, 64, 256)).astype(np.float32)
    lab = rng.integers(0, 2, n).astype(np.int32)
    with H.Classifier(seed=9) as c:
        p = c.params()
        g, _ = c.gradients(dm, ft, lab)
    _, want, _ = oracle.cnn_run(p, dm, ft, lab)
    # rounding points agree; only FP32 summation order differs, which may move
    # single BF16 roundings of the layers before: the bound of the conv layers
    for a, b in ((0, CONV), (CONV, CONV + FC1)):
        x, y = g[a:b].astype(np.float64), want[a:b].astype(np.float64)
        assert np.linalg.norm(x - y) <= 3e-2 * np.linalg.norm(y) + 1e-7
