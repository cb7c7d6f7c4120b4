"""Gradients at the batch sizes where the backward kernels' work splits change
(a single sample, one block of bias partial sums more or less, a batch that is
no multiple of the head's 128-sample chunks), against the CPU network with the
same rounding points."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 16, 17])
def test_gradients_match_oracle(hdb, oracle_lib, n):
    rng = np.random.default_rng(100 + n)
    dm = rng.standard_normal((n, 64, 64)).astype(np.float32)
    ft = rng.standard_normal((n, 64, 256)).astype(np.float32)
    lab = rng.integers(0, 2, n).astype(np.int32)
    with H.Classifier(seed=5) as c:
        p = c.params()
        g, loss = c.gradients(dm, ft, lab)
        again, _ = c.gradients(dm, ft, lab)
    np.testing.assert_array_equal(g.view(np.uint32), again.view(np.uint32))
    _, want, want_loss = oracle.cnn_run(p, dm, ft, lab)
    assert abs(loss - want_loss) <= 2e-3 * abs(want_loss)
    at = 0
    for _ in range(2):
        for ci, co in ((1, 8), (8, 16), (16, 32)):
            for size in (co * ci * 9, co):
                a, b = g[at:at + size].astype(np.float64), want[at:at + size].astype(np.float64)
                # rounding points agree; only FP32 summation order differs
                assert np.linalg.norm(a - b) <= 3e-2 * np.linalg.norm(b) + 1e-7
                at += size


@pytest.mark.parametrize("n", [127, 128, 129, 300])
def test_head_sums_over_chunks(hdb, n):
    """The FC2 bias gradient is the sum of p - y over the batch / n, and the
    scores give p: every sample is counted once at any chunk boundary."""
    rng = np.random.default_rng(n)
    dm = rng.standard_normal((n, 64, 64)).astype(np.float32)
    ft = rng.standard_normal((n, 64, 256)).astype(np.float32)
    lab = rng.integers(0, 2, n).astype(np.int32)
    with H.Classifier(seed=6) as c:
        g, _ = c.gradients(dm, ft, lab)
        prob = c.score(dm, ft)
    want = float(np.sum(prob.astype(np.float64) - lab)) / n
    # scores of the fused kernel and of the training path agree to 2e-3 each
    assert abs(float(g[-1]) - want) <= 2e-3
    assert abs(float(g[-2]) + want) <= 2e-3
