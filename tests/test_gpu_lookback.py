"""The ordered compaction behind every list of a pass (csrc/compact.cuh), compiled with a
plain keep-flag functor: the order and the total, and a look-back whose wait runs out --
the first tile is never started, so that nothing publishes what the others wait for."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from spikesorting_fullpursuit_b200 import build  # noqa: E402

TILE = 1024
FAILED = 3
SRC = r"""
#include "compact.cuh"
struct KeepF {
    const uint8_t* keep;
    uint32_t* out;
    __device__ bool visit(uint32_t i) const { return keep[i] != 0; }
    __device__ void emit(uint32_t i, uint32_t pos) const { out[pos] = i; }
};
extern "C" int run(const uint8_t* keep, uint32_t* out, uint32_t n, unsigned long long* state, uint32_t* total,
                   fbp::DevStatus* status, uint32_t tiles, uint32_t polls)
{
    fbp::compact_kernel<<<tiles, fbp::kCompactThreads>>>(KeepF{keep, out}, n, state, &status->ticket[0], total, status,
                                                         polls);
    return (int)cudaDeviceSynchronize();
}
extern "C" size_t ticket_offset() { return offsetof(fbp::DevStatus, ticket); }
extern "C" size_t error_offset() { return offsetof(fbp::DevStatus, error); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if not (os.path.exists(build.NVCC) or shutil.which(build.NVCC)):
        pytest.skip("no nvcc")
    d = tmp_path_factory.mktemp("lookback")
    src, so = str(d / "keep.cu"), str(d / "keep.so")
    with open(src, "w") as fp:
        fp.write(SRC)
    subprocess.check_call([build.NVCC, *build.ARCH, "-std=c++17", "-O2", "-Xcompiler", "-fPIC", "-shared", "-cudart",
                           "static", "-I", build.CSRC, "-o", so, src])
    h = ctypes.CDLL(so)
    vp, u32 = ctypes.c_void_p, ctypes.c_uint32
    h.run.argtypes = [vp, vp, u32, vp, vp, vp, u32, u32]
    h.ticket_offset.restype = h.error_offset.restype = ctypes.c_size_t
    return h


def _run(lib, keep, first_tile=0, polls=1 << 20):
    n = keep.size
    nt = -(-n // TILE)
    k = torch.from_numpy(keep).cuda()
    out = torch.full((n,), -1, dtype=torch.int32, device="cuda")
    state = torch.zeros(nt, dtype=torch.int64, device="cuda")
    total = torch.full((1,), 77, dtype=torch.int32, device="cuda")
    status = torch.zeros(64, dtype=torch.int32, device="cuda")
    status[lib.ticket_offset() // 4] = first_tile
    torch.cuda.synchronize()
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert lib.run(p(k), p(out), n, p(state), p(total), p(status), nt - first_tile, polls) == 0
    return (out.cpu().numpy(), int(total[0]), int(status[lib.error_offset() // 4]),
            state.cpu().numpy().view(np.uint64) >> np.uint64(62))


@pytest.mark.parametrize("n", [1, 1023, 1024, 1025, 33 * TILE, 200 * TILE + 17])
@pytest.mark.parametrize("share", [0.0, 0.4, 1.0])
def test_order_and_total(lib, n, share):
    keep = (np.random.default_rng(n).random(n) < share).astype(np.uint8)
    out, total, error, _ = _run(lib, keep)
    want = np.flatnonzero(keep)
    assert error == 0 and total == want.size
    assert np.array_equal(out[:total], want) and np.all(out[total:] == -1)


@pytest.mark.parametrize("tiles", [2, 3, 33, 34, 100])
def test_a_wait_that_runs_out_leaves_an_empty_list(lib, tiles):
    out, total, error, state = _run(lib, np.ones(tiles * TILE - 5, dtype=np.uint8), first_tile=1, polls=2000)
    assert error == 0x400
    assert total == 0
    assert np.all(out == -1)
    assert state[0] == 0 and np.all(state[1:] == FAILED)
