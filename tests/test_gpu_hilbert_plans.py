"""The Hilbert transform's plans and the STFT's frame forms at the sizes where
they change, against the oracle's numpy restatement (audio_eemd/spectra.py):
one launch or three, a row's own length or a longer convolution, even and odd
rows, radix-16 to prime factors, one row or many."""
import numpy as np
import pytest

from oracle import spectra_oracle as SP

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import spectra  # noqa: E402


def rows_of(M, N, seed):
    """Two tones and a thousandth of noise, so that |z| stays away from zero."""
    rng = np.random.default_rng(seed)
    t = np.arange(N, dtype=float)
    return np.array([np.cos(2 * np.pi * rng.uniform(0.01, 0.2) * t + rng.uniform(0, 6.3)) * 10.0 ** -m
                     + 1e-4 * 10.0 ** -m * rng.standard_normal(N) for m in range(M)])


# 4, 6: single points of the half transform; 4095 / 4096 / 4097 / 4098: one
# launch, at its own length or longer, and the first of three; 2 * 37 and 74 *
# 61: an even row whose half has no plan; 14 * 169: primes 7 and 13; 8192 and
# 9000: two-factor halves of powers of two and of 2, 3 and 5; 31 * 211 odd
@pytest.mark.parametrize("N", [4, 6, 7, 74, 2366, 2047, 4095, 4096, 4097, 4098, 4514, 6541, 8192, 9000])
@pytest.mark.parametrize("M", [1, 3])
def test_hilbert_plans(N, M):
    """Amplitudes within 1e-11 of a row's largest and frequencies within 1e-6
    of the rate (an FFT's rounding grows with log N; the smallest row is a
    hundredth of the largest, each is held to its own size)."""
    sr = 1000.0
    X = rows_of(M, N, N + M)
    f, a = (v.cpu().numpy() for v in spectra.hilbert_if_device(torch.from_numpy(X).cuda(), sr))
    for r in range(M):
        of, oa = SP.hilbert_if(X[r], sr)
        assert np.max(np.abs(a[r] - oa)) <= 1e-11 * np.max(oa), r
        ok = oa > 1e-3 * oa.max()
        ok &= np.roll(ok, 1) & np.roll(ok, -1)
        assert np.max(np.abs(f[r] - of)[ok], initial=0.0) <= 1e-6 * sr, r


def test_hilbert_many_rows_and_long_odd_rows():
    """More rows than one wave of CTAs (16 points per thread instead of 8), a
    long prime length, and the frequency's wrap at tile ends (1024 samples)."""
    sr = 1000.0
    for M, N in [(700, 1500), (40, 48000), (2, 100003)]:
        X = rows_of(2, N, N)[np.arange(M) % 2]
        f, a = (v.cpu().numpy() for v in spectra.hilbert_if_device(torch.from_numpy(X).cuda(), sr))
        for r in (0, 1):
            of, oa = SP.hilbert_if(X[r], sr)
            assert np.max(np.abs(a[r::2] - oa)) <= 1e-11 * np.max(oa)
            ok = oa > 1e-3 * oa.max()
            ok &= np.roll(ok, 1) & np.roll(ok, -1)
            assert np.max(np.abs(f[r::2] - of)[:, ok]) <= 1e-6 * sr


def test_hilbert_of_a_row_with_a_nan_leaves_the_others():
    """A row with a non-finite sample has no finite transform (not a number
    throughout); the rows beside it are untouched."""
    for N in (1000, 9000):
        X = rows_of(3, N, 5)
        Y = X.copy()
        Y[1, 17] = np.nan
        f0, a0 = (v.cpu().numpy() for v in spectra.hilbert_if_device(torch.from_numpy(X).cuda(), 1000.0))
        f, a = (v.cpu().numpy() for v in spectra.hilbert_if_device(torch.from_numpy(Y).cuda(), 1000.0))
        assert np.isnan(f[1]).all() and np.isnan(a[1]).all()
        assert np.array_equal(f[[0, 2]], f0[[0, 2]]) and np.array_equal(a[[0, 2]], a0[[0, 2]])


# odd frames (225 = 9 * 25, 3003 = 3 * 7 * 11 * 13), even ones of an odd half
# (2 * 1001), the shortest, the largest, and more frames than one wave of CTAs
@pytest.mark.parametrize("nper,N", [(2, 50), (3, 50), (16, 300), (225, 5000), (2002, 9000), (3003, 9000),
                                    (4094, 20000), (4096, 600000), (256, 200000)])
def test_stft_frame_forms(nper, N):
    """Bins within 1e-11 of the largest (the rounding of a transform of up to
    4096 points is a hundred times below that)."""
    X = rows_of(2, N, nper)
    f, t, Z = spectra.stft_device(torch.from_numpy(X).cuda(), 1000.0, nperseg=nper)
    Z = Z.cpu().numpy()
    for r in range(2):
        of, ot, oZ = SP.stft(X[r], 1000.0, nper)
        assert np.allclose(f, of) and np.allclose(t, ot)
        assert np.max(np.abs(Z[r] - oZ)) <= 1e-11 * np.max(np.abs(oZ))
