"""The residual energy and its gradient where the launches change: a warp's share of the
channels, and the warps of a spike."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from test_gpu_adjoint import _check  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# channels: up to 8 four warps a spike, above 16 (up to 592 spikes); samples: below 606,208
# the channels are shared between 2 and 9472 / (samples / 128) warps, above by none
@pytest.mark.parametrize("C,W,N,n", [(8, 20, 900, 30), (9, 20, 900, 30), (16, 7, 400, 33), (17, 130, 700, 21),
                                     (70, 20, 300, 40), (9, 11, 4000, 592), (9, 11, 4000, 593), (5, 40, 384000, 20),
                                     (2, 40, 606208, 8), (2, 40, 606336, 8), (3, 40, 1300001, 6)])
def test_launch_shapes(C, W, N, n):
    rng = np.random.default_rng(C * 1000 + n)
    M = 3
    V = rng.standard_normal((C, N)).astype(np.float32)
    T = rng.standard_normal((M, C, W)).astype(np.float32)
    T[0, C // 2] = 0.0
    idx = np.sort(rng.integers(0, N, size=n))
    idx[0], idx[-1] = 0, N - 1
    lab = rng.integers(0, M, size=n)
    amp = rng.normal(1.0, 0.1, size=n).astype(np.float32)
    tau = rng.uniform(0.02, 0.9, size=n).astype(np.float32) * rng.choice([-1, 1], size=n).astype(np.float32)
    _check(V, T, idx.astype(np.int64), lab.astype(np.int64), amp, tau)
