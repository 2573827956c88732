"""The kernels either side of the pursuit at the edges of their tiles and dispatch rules,
against the oracle's restatements of the reference's numpy code."""
import numpy as np
import pytest

import postprocess_ref
import preprocess_ref
import separability_ref

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# clips per register tile of a warp: 8, 16, 32, 64 keys a lane, then selection from memory
@pytest.mark.parametrize("n", [2, 31, 256, 257, 512, 513, 1024, 1025, 2048, 2049])
def test_robust_template_at_tile_edges(n):
    from spikesorting_fullpursuit_b200.processing import clip_utils
    rng = np.random.default_rng(n)
    c = (rng.standard_normal((n, 37)) * rng.uniform(0.1, 40, 37)).astype(np.float32)
    c[:, 3] = -1.5                                  # constant: empty 1-MAD set
    c[rng.integers(0, n, size=n // 2), 5] = 2.5     # ties
    c[:, 7] = np.where(rng.random(n) < 0.5, 0.0, -0.0)
    assert np.array_equal(clip_utils.calculate_robust_template(c), preprocess_ref.robust_template(c))


# FP64 sums of n centred products: off by at most about 2 n 2^-53 of the rms products
# (n <= 1000 here: 2.3e-13), in any order
@pytest.mark.parametrize("rows", [1, 7, 9, 1000])
@pytest.mark.parametrize("W", [1, 16, 111, 112, 113, 230])
def test_covariance_at_tile_edges(W, rows):
    from spikesorting_fullpursuit_b200.overlap import full_binary_pursuit as fbp
    rng = np.random.default_rng(W * 1000 + rows)
    R = [(rng.standard_normal((rows // 2, 2 * W)) * 3 + 5).astype(np.float32),
         (rng.standard_normal((rows - rows // 2, 2 * W)) - 2).astype(np.float32)]
    got = fbp.get_channel_covariance_matrix(R, 2, W, 10 ** 6, False)
    want = preprocess_ref.channel_covariances(R, 2, W, 10 ** 6)
    for c in range(2):
        w = np.atleast_2d(want[c])
        scale = np.abs(np.vstack(R)[:, c * W:(c + 1) * W].astype(np.float64)).max() ** 2
        assert np.max(np.abs(got[c] - w)) <= 1e-12 * scale
        assert np.array_equal(got[c], got[c].T)


# Against the oracle in float64 (for float32 templates too: its float32 correlations take
# the other of two nearly equal lags now and then).  A tail probability's relative error is
# about z times the error of its argument z = E_diff / sd: some 10 C W 2^-53 z in FP64 (z
# below 38: smaller probabilities underflow), and for float32 templates at shift 0, where
# E_diff and the difference are float32, 2^-23 (SS12 + SS1 / 2 + SS2 / 2) / sd + 2^-23 z.
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("W,M", [(8, 3), (64, 33), (65, 5), (80, 31), (81, 4), (104, 6), (105, 32), (128, 2), (129, 3)])
def test_pair_tiles(W, M, dtype):
    from spikesorting_fullpursuit_b200.overlap import neuron_separability as ns
    rng = np.random.default_rng(W + M)
    C = 5
    T = np.zeros((M, C, W))
    t = np.arange(W)
    for m in range(M):
        for c in rng.choice(C, size=int(rng.integers(1, C)), replace=False):
            T[m, c] = rng.uniform(-3, 3) * np.exp(-(t - 0.4 * W - rng.uniform(-3, 3)) ** 2 / (2 * rng.uniform(2, 5) ** 2))
    T[M - 1] = 0.0 if M > 2 else T[M - 1]          # a template without a channel
    T = T.reshape(M, C * W).astype(dtype)
    A = rng.standard_normal((C, W, W)) / np.sqrt(W)
    covs = [a @ a.T + 0.1 * np.eye(W) for a in A]
    ss = np.sum(T ** 2, axis=1)
    var = np.array([sum(T[m].reshape(C, W)[c] @ covs[c] @ T[m].reshape(C, W)[c] for c in range(C)) for m in range(M)])
    sm = {"templates": T, "template_SS": ss, "channel_covariance_mats": covs, "bp_n_samples_per_chan": W,
          "neuron_variances": var, "neuron_lower_thresholds": -0.5 * ss.astype(np.float64) + 3.0 * np.sqrt(var)}
    si = {"n_channels": C, "n_samples_per_chan": W}
    sm64 = dict(sm, templates=T.astype(np.float64), template_SS=ss.astype(np.float64))
    want = separability_ref.pairwise(sm64, si)
    got = ns._pair_metrics(sm, si)
    assert np.array_equal(got[3], want[3])
    rtol = np.full((M, M), 2e-9)
    if dtype == np.float32:
        for a, b in zip(*np.nonzero(want[3] == 0)):
            d = (sm64["templates"][a] - sm64["templates"][b]).reshape(C, W)
            sd = np.sqrt(sum(d[c] @ covs[c] @ d[c] for c in range(C)))
            if sd > 0:
                s12 = float(sm64["templates"][a] @ sm64["templates"][b])
                e = 0.5 * float(ss[a]) - (s12 - 0.5 * float(ss[b]))
                z = abs(e) / sd
                dz = 2.0 ** -23 * ((abs(s12) + 0.5 * float(ss[a]) + 0.5 * float(ss[b])) / sd + z)
                rtol[a, b] = np.expm1(2 * (z + 1) * dz)
    for g, w, r in zip(got[:3], want[:3], (rtol, 2e-9, 2e-9)):
        ok = (np.isnan(g) & np.isnan(w)) | (np.abs(g - w) <= 1e-290 + r * np.abs(w))
        assert np.all(ok)


# pieces of the pairwise sums: below 8, one piece, two, many, and past the warp kernel's list
@pytest.mark.parametrize("L", [1, 7, 8, 9, 64, 127, 128, 129, 136, 255, 257, 1616, 16384, 16385])
def test_sums_in_numpys_order(L):
    from spikesorting_fullpursuit_b200 import postprocessing
    rng = np.random.default_rng(L)
    n = 40
    base = (rng.standard_normal(L) * 7).astype(np.float32)
    # clips that are permutations of each other: their sums differ in the last bits only,
    # by the order of the additions, and the walk's comparisons follow them
    clips = np.stack([rng.permutation(base) for _ in range(n)])
    tmpl = np.zeros(L, dtype=np.float32)
    ev = np.arange(n, dtype=np.int64)
    bp = np.ones(n, dtype=bool)
    want = postprocess_ref.remove_binary_pursuit_duplicates(ev, clips, tmpl, bp, 2)
    got = postprocessing.remove_binary_pursuit_duplicates(ev, clips, tmpl, bp, 2)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [1, 2, 16, 17, 18, 33, 300])
@pytest.mark.parametrize("L", [2, 63, 65, 130])   # numpy sums a single column pairwise, not row by row
def test_mean_clip_row_order(n, L):
    from spikesorting_fullpursuit_b200 import postprocessing
    rng = np.random.default_rng(n * 1000 + L)
    clips = (rng.standard_normal((n, L)) * rng.uniform(0.1, 1e4, (n, 1))).astype(np.float32)
    assert np.array_equal(postprocessing.mean_clip(clips).cpu().numpy(), np.mean(clips, axis=0))


@pytest.mark.parametrize("kind", ["float32", "rows_apart", "read_only", "every_other", "int16", "float64", "reversed"])
@pytest.mark.parametrize("shape,limit", [((4, 5000), None), ((3, 1_000_003), 0), ((700, 4001), 0), ((1, 9_000_000), 0)])
def test_uploads(kind, shape, limit, monkeypatch):
    """Voltage chunks as they are and through slabs of one and of many samples a channel,
    more blocks than slabs, any dtype and row stride."""
    from spikesorting_fullpursuit_b200.overlap import binary_pursuit_parallel as bpp
    if limit is not None:
        monkeypatch.setattr(bpp._Uploader, "DIRECT_BYTES", limit)
    rng = np.random.default_rng(shape[1])
    C, N = shape
    wide = rng.integers(-3000, 3000, size=(C, 2 * N)).astype(
        {"int16": np.int16, "float64": np.float64}.get(kind, np.float32))
    host = {"every_other": wide[:, ::2], "reversed": wide[:, N - 1::-1]}.get(kind, wide[:, :N])
    if kind == "float32":
        host = np.ascontiguousarray(host)
    host.flags.writeable = kind != "read_only"
    dev = torch.device("cuda", torch.cuda.current_device())
    dst = torch.zeros((C, N), dtype=torch.float32, device=dev)
    up = bpp._Uploader(torch, dev)
    try:
        for _ in range(2):
            up.upload(host, dst)
            assert np.array_equal(dst.cpu().numpy(), host.astype(np.float32))
            dst.zero_()
    finally:
        up.close()
