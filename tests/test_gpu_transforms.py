"""Pursuits whose correlations are made by 256-point transforms, at the sizes where the
transform kernels can go wrong, against the oracle: indices, labels, order and clips equal."""
import copy

import numpy as np
import pytest

import oracle

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from spikesorting_fullpursuit_b200 import binary_pursuit, synth  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# (channels, units, sampling rate, clip window in samples before / after, shift range or None for W - 1)
CASES = {
    "one_channel_one_unit": (1, 1, 40000, 40, 60, None),
    "odd_channels_and_units": (5, 9, 30000, 30, 45, None),
    "half_shift": (7, 11, 30000, 30, 45, 37),
    "no_shift": (3, 4, 30000, 30, 45, 0),
    "shift_beyond_window": (3, 4, 20000, 10, 25, 50),
    "longest_window": (4, 5, 40000, 50, 77, None),
    "window_past_the_transform": (4, 5, 40000, 50, 78, None),
    "short_window": (4, 6, 20000, 8, 11, None),
    "seventeen_units": (16, 17, 30000, 20, 30, None),
    "many_channels": (33, 8, 30000, 20, 30, None),
    "more_channels_than_a_mask": (70, 4, 30000, 20, 30, None),
}


@pytest.mark.parametrize("recheck", [True, False])
@pytest.mark.parametrize("case", sorted(CASES))
def test_pursuit_matches_oracle(case, recheck):
    C, M, fs, before, after, S = CASES[case]
    clip = (-(before + 0.25) / fs, (after - 0.25) / fs)
    V, si, sm, _ = synth.make_recording(17 * len(case) + C, n_chans=C, fs=fs, duration_s=0.25, n_units=M,
                                        rate_model=("uniform", 20.0, 60.0), overlap_frac=0.3, clip_width=clip)
    W = si["n_samples_per_chan"]
    si["get_adjusted_clips"] = True
    si["do_overlap_recheck"] = recheck
    S = W - 1 if S is None else S
    want = oracle.binary_pursuit(V, np.float32, si, copy.deepcopy(sm), n_max_shift_inds=S,
                                 global_mem_size=183 * 1024 ** 3)
    got = binary_pursuit(V, np.float32, si, copy.deepcopy(sm), n_max_shift_inds=S, verbose=False)
    assert len(want[0]) > 0
    for g, w in zip(got, want):
        assert np.array_equal(np.asarray(g), np.asarray(w)), (case, W, S)


def _same_as_oracle(V, si, sm, S):
    want = oracle.binary_pursuit(V, np.float32, si, copy.deepcopy(sm), n_max_shift_inds=S,
                                 global_mem_size=183 * 1024 ** 3)
    got = binary_pursuit(V, np.float32, si, copy.deepcopy(sm), n_max_shift_inds=S, verbose=False)
    assert len(want[0]) > 0
    for g, w in zip(got, want):
        assert np.array_equal(np.asarray(g), np.asarray(w), equal_nan=True)


def test_samples_that_are_not_numbers_stay_in_their_windows():
    """Windows and stretches are transformed in pairs: a NaN must not reach the other one's
    spikes.  (An infinite sample's likelihood stays infinite after every subtraction: the
    reference's loop does not end on it, so there is nothing to compare with.)"""
    V, si, sm, _ = synth.make_recording(29, n_chans=4, duration_s=0.4, n_units=6,
                                        rate_model=("uniform", 30.0, 60.0), overlap_frac=0.3)
    si["get_adjusted_clips"] = True
    V = V.copy()
    V[1, 5000] = np.nan
    V[0, 9100:9104] = np.nan
    V[3, 12345] = -np.nan
    _same_as_oracle(V, si, sm, si["n_samples_per_chan"] - 1)


@pytest.mark.parametrize("amp", [(6.0, 12.0), (20.0, 60.0)])
def test_many_similar_units_on_the_same_channels(amp):
    """More rows and chunks of items reach the bounds than the screen's lists hold."""
    V, si, sm, _ = synth.make_recording(31, n_chans=3, fs=30000, duration_s=0.12, n_units=70,
                                        rate_model=("uniform", 5.0, 15.0), overlap_frac=0.5, amp=amp)
    si["get_adjusted_clips"] = True
    _same_as_oracle(V, si, sm, si["n_samples_per_chan"] - 1)


@pytest.mark.parametrize("recheck", [True, False])
@pytest.mark.parametrize("windows", [1024, 1025, 33 * 1024 + 5, 70 * 1024 - 1])
def test_window_lists_over_many_tiles(windows, recheck):
    """The passes' lists are compacted in tiles of 1024 windows, each looking back over the
    tiles before it, 32 at a time."""
    fs, W = 20000, 9
    V, si, sm, _ = synth.make_recording(windows, n_chans=1, fs=fs, duration_s=windows * W / fs, n_units=3,
                                        rate_model=("uniform", 60.0, 120.0), overlap_frac=0.2,
                                        clip_width=(-3.25 / fs, 4.75 / fs))
    assert si["n_samples_per_chan"] == W and abs(V.shape[1] - windows * W) <= W
    si["do_overlap_recheck"] = recheck
    _same_as_oracle(V, si, sm, W - 1)


@pytest.mark.parametrize("seconds", [0.05, 4.0, 13.0])
def test_few_and_many_windows(seconds):
    """Passes of fewer and of more listed windows than the recheck's screen takes 512 threads
    for, and of fewer and more queued runs than the recomputation has warps for."""
    V, si, sm, _ = synth.make_recording(61, n_chans=5, fs=30000, duration_s=seconds, n_units=8,
                                        rate_model=("uniform", 40.0, 90.0), overlap_frac=0.3)
    si["get_adjusted_clips"] = True
    _same_as_oracle(V, si, sm, si["n_samples_per_chan"] - 1)
