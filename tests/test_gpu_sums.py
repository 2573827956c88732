"""Sums in numpy's order where the kernels split them: template energies and short clips."""
import numpy as np
import pytest

import postprocess_ref

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# below 8 values, one piece, two, many, the longest list of pieces and past it
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("C,W", [(1, 1), (1, 7), (1, 8), (1, 9), (2, 64), (3, 43), (2, 68), (5, 51), (1, 257), (16, 101),
                                 (64, 76), (64, 256), (113, 145)])
def test_template_energy(C, W, dtype):
    from spikesorting_fullpursuit_b200.overlap import neuron_separability as ns
    rng = np.random.default_rng(C * 1000 + W)
    T = (rng.standard_normal((5, C * W)) * rng.uniform(0.1, 30, (5, 1))).astype(dtype)
    A = rng.standard_normal((C, W, W)) / np.sqrt(W)
    covs = A @ A.transpose(0, 2, 1)
    ss, _ = ns.bp_thresholds(T, list(covs), C, W)
    assert ss.dtype == dtype
    assert np.array_equal(ss, np.array([np.sum(t ** 2) for t in T], dtype=dtype))
    _, _, var, *_ = ns._device_metrics(T, list(covs), C, W, 3.7, 12.0, False)
    T3 = T.astype(np.float64).reshape(5, C, W)
    want = np.einsum("mci,cij,mcj->m", T3, covs, T3)
    # C W W products summed in FP64, in any order: off by at most C W W 2^-53 of their magnitudes
    scale = np.einsum("mci,cij,mcj->m", np.abs(T3), np.abs(covs), np.abs(T3))
    assert np.all(np.abs(var - want) <= 2 * (C * W * W + 4) * 2.0 ** -53 * scale)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 3000])
@pytest.mark.parametrize("L", [1, 5, 8, 20, 121, 128])
def test_short_clips(n, L):
    """Clips that are permutations of each other: the walk's comparisons follow their sums' last bits."""
    from spikesorting_fullpursuit_b200 import postprocessing
    rng = np.random.default_rng(n + L)
    base = (rng.standard_normal(L) * 7).astype(np.float32)
    clips = np.stack([rng.permutation(base) for _ in range(n)])
    tmpl = np.zeros(L, dtype=np.float32)
    ev = np.cumsum(rng.integers(0, 5, n)).astype(np.int64)
    bp = rng.random(n) < 0.9
    want = postprocess_ref.remove_binary_pursuit_duplicates(ev, clips, tmpl, bp, 3)
    assert np.array_equal(postprocessing.remove_binary_pursuit_duplicates(ev, clips, tmpl, bp, 3), want)
