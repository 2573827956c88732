"""Residual subtraction with overlapping spikes against a sequential numpy loop: more spikes
than resident CTAs, blocks of 2048 flags with none, one and all of them set, spikes at the
recording's end and labels past the templates."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from spikesorting_fullpursuit_b200 import _native  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _subtract(V, T, idx, lab, W):
    """compute_residual (binary_pursuit.cl:57-102), spike by spike in list order."""
    C, N = V.shape
    for s, t in zip(idx, lab):
        if t < T.shape[0]:
            e = min(N, s + W)
            V[:, s:e] -= T[t].reshape(C, W)[:, :e - s]
    return V


def _run(V, T, idx, lab, W, noalloc=False):
    C, N = V.shape
    d = _native.dims(C, N, T.shape[0], W, W - 1)
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    Vd, Td = torch.from_numpy(V).cuda(), torch.from_numpy(T).cuda()
    di, dl = (torch.from_numpy(a.astype(np.int32)).cuda() for a in (idx, lab))
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    L = _native.lib()
    if noalloc:
        _native.check(L.fbp_residual_noalloc(ctypes.byref(d), p(Vd), p(Td), p(di), p(dl), idx.size, st))
    else:
        ws = torch.full((_native.workspace_bytes(d, _native.FBP_PLAIN_FP32),), 255, dtype=torch.uint8, device="cuda")
        _native.check(L.fbp_residual(ctypes.byref(d), p(Vd), p(Td), p(di), p(dl), idx.size, p(ws), ws.numel(), st))
    return Vd.cpu().numpy()


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("share", ["none", "one", "some", "all"])
@pytest.mark.parametrize("n,C,W", [(1, 1, 1), (2, 3, 7), (33, 4, 40), (2047, 2, 9), (2049, 1, 12), (2368, 5, 33),
                                   (2369, 2, 16), (6200, 3, 11), (700, 16, 101), (300, 30, 70)])
def test_overlapping_spikes_in_list_order(n, C, W, share, noalloc):
    rng = np.random.default_rng(n * 10 + W)
    idx = np.arange(n, dtype=np.int64) * (W + 1) + 1
    if share == "one" and n > 1:
        k = int(rng.integers(1, n))
        idx[k] = idx[k - 1] + W - 1
    elif share == "some":
        k = 1 + rng.permutation(n - 1)[:max(1, n // 10)] if n > 1 else np.array([], dtype=int)
        idx[k] -= rng.integers(2, W + 2, size=k.size)
        idx = np.sort(idx)
    elif share == "all":
        idx = np.sort(rng.integers(1, n * (W + 1), size=n))   # several spikes of the same sample among them
    N = n * (W + 1) + W // 2 + 1   # the last spike may reach past the end
    lab = rng.integers(0, 5, size=n)   # 4 templates: label 4 is no spike
    V = rng.standard_normal((C, N)).astype(np.float32)
    T = rng.standard_normal((4, C * W)).astype(np.float32)
    want = _subtract(V.copy(), T, idx, lab, W)
    assert np.array_equal(_run(V, T, idx, lab, W, noalloc), want)
