"""Noise covariances where a cluster's share of the rows and the CTAs a channel change: few
rows leave CTAs of a cluster without any, and many channels get one CTA each."""
import numpy as np
import pytest

import preprocess_ref

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# FP64 sums of n centred products: off by at most about 2 n 2^-53 of the largest products
# (n <= 129 here: 3e-14), in any order
@pytest.mark.parametrize("C", [2, 18, 19])
@pytest.mark.parametrize("rows", [2, 15, 16, 17, 33, 64, 65, 127, 128, 129])
@pytest.mark.parametrize("W", [5, 112, 113])
def test_few_rows(C, rows, W):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spikesorting_fullpursuit_b200.overlap import full_binary_pursuit as fbp
    rng = np.random.default_rng(W * 1000 + rows)
    R = [(rng.standard_normal((rows // 2, C * W)) * 3 + 5).astype(np.float32),
         (rng.standard_normal((rows - rows // 2, C * W)) - 2).astype(np.float32)]
    got = fbp.get_channel_covariance_matrix(R, C, W, 10 ** 6, False)
    want = preprocess_ref.channel_covariances(R, C, W, 10 ** 6)
    for c in range(C):
        scale = np.abs(np.vstack(R)[:, c * W:(c + 1) * W].astype(np.float64)).max() ** 2
        assert np.max(np.abs(got[c] - want[c])) <= 1e-12 * scale
        assert np.array_equal(got[c], got[c].T)
