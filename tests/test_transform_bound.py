"""The rounding bound of correlations made by 256-point transforms, checked on the CPU.

csrc/fft256.cuh correlates two real signals at once, z = v_A + i v_B, by complex transforms
of 16 x 16 points in float32 with template spectra computed in float64 and rounded once.
Restated here in numpy's complex64, in the same order of radix-4 steps and twiddles.  Every
output must lie within
    (64 + 3 n) 2^-24  sum_c |T_c| |z_c|          (n: non-zero template channels)
of the float64 correlation, and the padded positions must not leak between shifts."""
import numpy as np
import pytest

U = 2.0 ** -24
C64 = np.complex64


def _fft4(a, b, c, d, sign):
    s0, s1, s2, e = a + c, a - c, b + d, b - d
    s3 = (e * C64(1j * sign)).astype(C64)
    return s0 + s2, s1 + s3, s0 - s2, s1 - s3


def _fft16(x, sign):
    """x[..., 16] -> transform, two radix-4 steps in float32."""
    y = [None] * 16
    for l in range(4):
        o = _fft4(x[..., l], x[..., l + 4], x[..., l + 8], x[..., l + 12], sign)
        for r in range(4):
            w = C64(np.exp(sign * 2j * np.pi * l * r / 16))
            y[l + 4 * r] = (o[r] * w).astype(C64)
    out = [None] * 16
    for r in range(4):
        for q, v in enumerate(_fft4(*(y[4 * r + l] for l in range(4)), sign)):
            out[4 * q + r] = v
    return np.stack(out, axis=-1)


def _fft256(z, sign):
    y = _fft16(np.swapaxes(z.reshape(z.shape[:-1] + (16, 16)), -1, -2), sign)      # [l][r]
    k = np.arange(16)
    y = (y * np.exp(sign * 2j * np.pi * np.outer(k, k) / 256).astype(C64)).astype(C64)
    return np.swapaxes(_fft16(np.swapaxes(y, -1, -2), sign), -1, -2).reshape(z.shape)


def _correlate(T, z):
    """float32 correlation of T [n][W] with the complex signals z [n][256], as the kernel makes it."""
    n, W = T.shape
    pad = np.zeros((n, 256))
    pad[:, :W] = T
    spec = (np.fft.fft(pad) / 256).astype(C64)
    Z = _fft256(z.astype(C64), -1)
    P = np.zeros(256, dtype=C64)
    for c in range(n):
        P = (P + (np.conj(spec[c]) * Z[c]).astype(C64)).astype(C64)
    return _fft256(P, 1)


def _exact(T, z):
    """float64 correlation r[x] = sum_j T[j] z[(j + x) mod 256]."""
    n, W = T.shape
    r = np.zeros(256, dtype=np.complex128)
    for c in range(n):
        for j in range(W):
            r += float(T[c, j]) * np.roll(z[c].astype(np.complex128), -j)
    return r


def test_transform_pair_inverts():
    rng = np.random.default_rng(1)
    z = (rng.standard_normal((4, 256)) + 1j * rng.standard_normal((4, 256))).astype(C64)
    assert np.allclose(_fft256(z, -1), np.fft.fft(z.astype(np.complex128)), atol=2e-5)
    assert np.allclose(_fft256(_fft256(z, -1), 1) / 256, z, atol=1e-6)


@pytest.mark.parametrize("n,W", [(1, 1), (1, 128), (4, 101), (16, 76), (64, 20)])
def test_correlation_within_the_bound(n, W):
    rng = np.random.default_rng(100 * n + W)
    worst = 0.0
    for trial in range(12):
        t = np.arange(W) - 0.4 * W
        T = (rng.uniform(-12, 12, (n, 1)) * np.exp(-t ** 2 / (2 * rng.uniform(2, 9, (n, 1)) ** 2))).astype(np.float32)
        v = rng.standard_normal((2, n, 256)) * np.float32(10.0 ** rng.uniform(-3, 3))
        at = rng.integers(0, 257 - W, 2)   # a template-like event in each signal, and one of very different size
        for s in range(2):
            v[s, :, at[s]:at[s] + W] += T * (1.0 if trial % 3 else 200.0 ** s)
        v = v.astype(np.float32)
        z = v[0] + 1j * v[1]
        bound = (64 + 3 * n) * U * float((np.linalg.norm(T.astype(np.float64), axis=1)
                                          * np.linalg.norm(z, axis=1)).sum())
        err = np.abs(_correlate(T, z) - _exact(T, z)).max()
        assert err <= bound, (trial, err, bound)
        worst = max(worst, err / bound)
    assert worst > 1e-4   # the bound is not vacuous: within a few orders of the worst error


def test_window_shifts_do_not_wrap():
    """A window of W samples padded to 256 meets every shift of [-(W - 1), W - 1] apart from the others."""
    rng = np.random.default_rng(7)
    W = 128
    T = rng.standard_normal((2, W)).astype(np.float32)
    z = np.zeros((2, 256), dtype=np.complex128)
    z[:, :W] = rng.standard_normal((2, W)) + 1j * rng.standard_normal((2, W))
    got = _correlate(T, z)
    for x in range(-(W - 1), W):
        lo, hi = max(0, x), min(W, W + x)
        want = sum((T[c, lo - x:hi - x].astype(np.float64) * z[c, lo:hi]).sum() for c in range(2))
        assert abs(got[x % 256] - want) < 1e-3, x
