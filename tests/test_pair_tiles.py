"""Pairwise separability: which of its two kernels a call takes (csrc/pair_rule.cuh, on the
CPU), and the tile kernel at its edges against the oracle (on the GPU)."""
import os
import re
import subprocess

import numpy as np
import pytest

import separability_ref
from spikesorting_fullpursuit_b200 import build

OPTIN = 232448   # bytes of shared memory a CTA can ask for (B200)

# (units, channels, samples, columns a lane of the tile kernel; 0: a CTA per pair)
SIZES = [
    # around the multiples of 8 columns a lane, with one unit more or less than a tile
    (64, 5, 56, 8), (65, 5, 64, 8), (64, 5, 65, 10), (65, 5, 80, 10), (64, 4, 81, 13), (65, 2, 101, 13),
    # the largest templates that fit beside the covariances, and the next
    (64, 7, 101, 13), (64, 8, 101, 0), (64, 1, 104, 13), (64, 2, 104, 0), (64, 1, 105, 0), (64, 2, 128, 0),
    # few units: a CTA per pair
    (63, 5, 64, 0), (63, 4, 76, 0), (48, 9, 76, 10), (47, 9, 76, 0), (48, 25, 76, 0),
    # short windows: tiles for many units only
    (128, 2, 55, 8), (127, 2, 55, 0), (128, 2, 32, 8), (128, 2, 31, 0),
]


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_rule")
    src, exe = str(d / "rule.cpp"), str(d / "rule")
    with open(src, "w") as fp:
        fp.write('#include "pair_rule.cuh"\n#include <cstdio>\n#include <cstdlib>\n'
                 "int main(int, char** v) { std::printf(\"%u\", fbp::pair_tile_columns(std::atoi(v[1]), "
                 "std::atoi(v[2]), std::atoi(v[3]), std::atoi(v[4]))); }\n")
    subprocess.check_call(["g++", "-std=c++17", "-x", "c++", "-I", build.CSRC, "-o", exe, src])
    return lambda M, C, W: int(subprocess.check_output([exe, str(M), str(C), str(W), str(OPTIN)]))


@pytest.mark.parametrize("M,C,W,columns", SIZES)
def test_rule(rule, M, C, W, columns):
    assert rule(M, C, W) == columns


def test_rule_over_its_ranges(rule):
    assert rule(200, 64, 76) == 10   # the dense probe
    for M in (2, 5, 12, 40):         # few units, whatever the channels
        for C in (4, 16, 33, 64):
            for W in (20, 61, 76, 101):
                assert rule(M, C, W) == 0


@pytest.mark.parametrize("W,channels", [(64, 225), (76, 133), (80, 120), (96, 18), (101, 7), (104, 1)])
def test_largest_templates_of_the_tiles(rule, W, channels):
    assert rule(200, channels, W) > 0
    assert rule(200, channels + 1, W) == 0


def test_every_instance_of_the_tile_kernel_is_reached(rule):
    with open(os.path.join(build.CSRC, "separability.cu")) as fp:
        built = {int(n) for n in re.findall(r"^ +FBP_PAIR\((\d+)\)", fp.read(), re.M)}
    assert built == {rule(200, 1, W) for W in range(1, 130)} - {0}


# Tolerances: a tail probability's relative error is about z times the error of its argument
# z = E_diff / sd: some 10 C W 2^-53 z in FP64 (z below 38: smaller probabilities underflow),
# below 1e-10 for C W <= 1500; and for float32 templates at shift 0, where E_diff and the
# difference are float32, 2^-23 (|SS12| + SS1 / 2 + SS2 / 2) / sd + 2^-23 z.
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("M,C,W,columns", SIZES)
def test_against_the_oracle(M, C, W, columns, dtype):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    from spikesorting_fullpursuit_b200.overlap import neuron_separability as ns
    rng = np.random.default_rng(1000 * M + W)
    T = np.zeros((M, C, W))
    t = np.arange(W)
    for m in range(M):
        for c in rng.choice(C, size=int(rng.integers(1, C + 1)), replace=False):
            T[m, c] = rng.uniform(-3, 3) * np.exp(-(t - 0.4 * W - rng.uniform(-3, 3)) ** 2 / (2 * rng.uniform(2, 5) ** 2))
    T[M // 2] = 0.0
    T = T.reshape(M, C * W).astype(dtype)
    A = rng.standard_normal((C, W, W)) / np.sqrt(W)
    covs = [a @ a.T + 0.1 * np.eye(W) for a in A]
    ss = np.sum(T ** 2, axis=1)
    T64 = T.astype(np.float64)
    var = np.einsum("mci,cij,mcj->m", T64.reshape(M, C, W), np.stack(covs), T64.reshape(M, C, W))
    sm = {"templates": T, "template_SS": ss, "channel_covariance_mats": covs, "bp_n_samples_per_chan": W,
          "neuron_variances": var, "neuron_lower_thresholds": -0.5 * ss.astype(np.float64) + 3.0 * np.sqrt(var)}
    si = {"n_channels": C, "n_samples_per_chan": W}
    # the oracle in float64 for float32 templates too: its float32 correlations take the
    # other of two nearly equal lags now and then
    want = separability_ref.pairwise(dict(sm, templates=T64, template_SS=ss.astype(np.float64)), si)
    got = ns._pair_metrics(sm, si)
    assert np.array_equal(got[3], want[3])
    rtol = np.full((M, M), 2e-9)
    if dtype == np.float32:
        for a, b in zip(*np.nonzero(want[3] == 0)):
            d = (T64[a] - T64[b]).reshape(C, W)
            sd = np.sqrt(np.einsum("ci,cij,cj->", d, np.stack(covs), d))
            if sd > 0:
                s12, half = float(T64[a] @ T64[b]), 0.5 * (float(ss[a]) + float(ss[b]))
                z = abs(half - s12) / sd
                rtol[a, b] = np.expm1(2 * (z + 1) * 2.0 ** -23 * ((abs(s12) + half) / sd + z))
    for g, w, r in zip(got[:3], want[:3], (rtol, 2e-9, 2e-9)):
        ok = (np.isnan(g) & np.isnan(w)) | (np.abs(g - w) <= 1e-290 + r * np.abs(w))
        assert np.all(ok)
