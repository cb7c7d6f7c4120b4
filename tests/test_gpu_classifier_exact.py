"""Gradients whose sums are exact in any order, compared bit for bit: small whole
inputs and weights, and a head whose probability is exactly 1, so that every
sample of the other class carries the gradient 1 / n.  An error in one row or
column of a layer's border, in a tap or in one sample of a sum shows, which a
norm over a whole layer hides."""
import numpy as np
import pytest

import heimdall_multibeam_b200 as H
import oracle

pytestmark = pytest.mark.gpu

LAYERS = ((1, 8), (8, 16), (16, 32))


def whole_params(rng):
    """Weights of -1, 0 and 1, fewer of them the more taps there are, biases 0,
    and class 1 ahead of class 0 by 2^20."""
    p = []
    for _ in range(2):
        for ci, co in LAYERS:
            on = rng.random(co * ci * 9) < min(1.0, 9.0 / (ci * 9))
            p += [on * rng.choice([-1.0, 1.0], co * ci * 9), np.zeros(co)]
    p += [(rng.random(16 * 10240) < 1 / 64) * rng.choice([-1.0, 1.0], 16 * 10240), np.zeros(16),
          rng.choice([-1.0, 0.0, 1.0], 32), [0.0, 2.0 ** 20]]
    return np.concatenate(p).astype(np.float32)


def whole_inputs(rng, n):
    return (rng.integers(-2, 3, (n, 64, 64)).astype(np.float32),
            rng.integers(-2, 3, (n, 64, 256)).astype(np.float32))


@pytest.mark.parametrize("n", [1, 2, 4])
def test_exact_gradients(hdb, oracle_lib, n):
    rng = np.random.default_rng(n)
    p = whole_params(rng)
    dm, ft = whole_inputs(rng, n)
    lab = np.arange(n, dtype=np.int32) % 2
    with H.Classifier() as c:
        c.set_params(p)
        g, _ = c.gradients(dm, ft, lab)
    _, want, _ = oracle.cnn_run(p, dm, ft, lab)
    at = 0
    for br in range(2):
        for ci, co in LAYERS:
            for what, size in (("weights", co * ci * 9), ("biases", co)):
                np.testing.assert_array_equal(g[at:at + size], want[at:at + size],
                                              err_msg=f"branch {br} {ci}->{co} {what}")
                assert np.count_nonzero(want[at:at + size]) > size // 4
                at += size
    np.testing.assert_array_equal(g[at:], want[at:])


@pytest.mark.parametrize("n", [127, 128, 129, 300])
def test_every_sample_is_counted_once(hdb, n):
    """One sample of the other class at each end of the head's chunks of 128: the
    batch's loss and gradients are that sample's own over n."""
    rng = np.random.default_rng(n)
    p = whole_params(rng)
    dm, ft = whole_inputs(rng, n)
    head = 2 * sum(co * ci * 9 + co for ci, co in LAYERS) + 16 * 10240  # FC1's biases on
    with H.Classifier() as c:
        c.set_params(p)
        for i in sorted({0, 1, 126, 127, 128, 255, 256, n - 1} & set(range(n))):
            lab = np.ones(n, np.int32)
            lab[i] = 0
            g, loss = c.gradients(dm, ft, lab)
            one, one_loss = c.gradients(dm[i:i + 1], ft[i:i + 1], lab[i:i + 1])
            assert np.count_nonzero(one[head:]) >= 10
            # (1 / n rounds; BF16 weights' products do not enter the head's sums)
            np.testing.assert_allclose(g[head:] * n, one[head:], rtol=1e-5, atol=0)
            assert abs(loss * n - one_loss) <= 1e-5 * abs(one_loss)
