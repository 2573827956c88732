"""Voltage uploads whose rows lie far apart -- recordings of hours, where a row's pitch
exceeds the documented limit of a 2-D copy (2^31 - 1 bytes) -- and uploads whose source
fails on the way."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from spikesorting_fullpursuit_b200 import _native  # noqa: E402
from spikesorting_fullpursuit_b200.overlap import binary_pursuit_parallel as bpp  # noqa: E402

FAR = (1 << 29) + 3   # floats between two rows: 2^31 + 12 bytes


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def _rows(seed, n, far):
    """Two rows of n values; `far`: FAR floats apart (memory between them is never touched)."""
    rng = np.random.default_rng(seed)
    host = np.empty(FAR + n, dtype=np.float32) if far else np.empty(2 * n, dtype=np.float32)
    step = FAR if far else n
    host[:n], host[step:step + n] = rng.standard_normal(n), rng.standard_normal(n)
    return np.lib.stride_tricks.as_strided(host, (2, n), (4 * step, 4))


@pytest.mark.parametrize("far_src", [False, True])
@pytest.mark.parametrize("far_dst", [False, True])
def test_copy_rows_of_any_pitch(far_src, far_dst):
    n = 5001
    src = _rows(1, n, far_src)
    step = FAR if far_dst else n + 7
    flat = torch.empty(step + n, dtype=torch.float32, device="cuda")
    dst = flat.as_strided((2, n), (step, 1))
    dst.zero_()
    _native.check(_native.lib().fbp_copy_rows(
        ctypes.c_void_p(dst.data_ptr()), 4 * step, ctypes.c_void_p(src.ctypes.data), src.strides[0], 4 * n, 2,
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    torch.cuda.synchronize()
    assert np.array_equal(dst.cpu().numpy(), src)


@pytest.mark.parametrize("direct", [True, False])
def test_upload_of_a_part_of_a_long_recording(direct, monkeypatch):
    if not direct:
        monkeypatch.setattr(bpp._Uploader, "DIRECT_BYTES", 0)
    n = 30011
    host = _rows(2, n, True)
    dev = torch.device("cuda", torch.cuda.current_device())
    flat = torch.empty(FAR + n, dtype=torch.float32, device=dev)
    dst = flat.as_strided((2, n), (FAR, 1))   # a chunk's rows in a buffer of a longer chunk
    dst.zero_()
    up = bpp._Uploader(torch, dev)
    try:
        up.upload(host, dst)
        assert np.array_equal(dst.cpu().numpy(), host)
    finally:
        up.close()


class _FailingSource:
    """A voltage that cannot be read from sample `at` on, as a truncated file."""

    def __init__(self, data, at):
        self.data, self.at, self.shape = data, at, data.shape

    def __getitem__(self, key):
        if key[1].stop > self.at:
            raise OSError("read error")
        return self.data[key]


@pytest.mark.parametrize("at", [0, 499, 500, 30000, 30010])
def test_a_failed_upload_leaves_zeros(at, monkeypatch):
    """A pursuit that runs behind the upload must not see memory that was never written."""
    monkeypatch.setattr(bpp._Uploader, "SLAB_FLOATS", 1000)
    monkeypatch.setattr(bpp._Uploader, "LEAST_FLOATS", 1000)
    n, span = 30011, 500   # two channels: 500 samples a range
    data = np.random.default_rng(3).standard_normal((2, n))
    dev = torch.device("cuda", torch.cuda.current_device())
    dst = torch.full((2, n), float("nan"), dtype=torch.float32, device=dev)
    up = bpp._Uploader(torch, dev)
    try:
        _, upto, flags, finish = up.start_staged(_FailingSource(data, at), dst)
        with pytest.raises(OSError, match="read error"):
            finish()
        assert np.all(flags == 1) and upto[-1] == n
        done = at // span * span
        got = dst.cpu().numpy()
        assert np.array_equal(got[:, :done], data[:, :done].astype(np.float32))
        assert np.all(got[:, done:] == 0)
    finally:
        up.close()
