"""The Hilbert frequency and amplitude where a row is zero or not finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import spectra  # noqa: E402


def hilbert(X):
    return [v.cpu().numpy() for v in spectra.hilbert_if_device(torch.from_numpy(X).cuda(), 1000.0)]


# one launch and three, at the row's own length and as a convolution
@pytest.mark.parametrize("N", [2, 3, 5, 8, 97, 4096, 4097, 4098, 5000, 7001])
def test_zero_rows_of_either_sign(N):
    """A zero row has no phase to move, whichever of its zeros are negative."""
    X = np.zeros((4, N))
    X[1] = -0.0
    X[2, ::3] = -0.0
    X[3, 1::2] = -0.0
    f, a = hilbert(X)
    assert not f.any() and not a.any()


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("N", [2, 3, 4, 5, 4098])
def test_rows_with_a_non_finite_sample(N, bad):
    """Such a row has no finite transform; the row beside it keeps its own."""
    X = np.random.default_rng(N).standard_normal((3, N))
    f0, a0 = hilbert(X)
    X[0, 0] = X[1, N - 1] = bad
    f, a = hilbert(X)
    assert not np.isfinite(f[:2]).any() and not np.isfinite(a[:2]).any()
    assert np.array_equal(f[2], f0[2]) and np.array_equal(a[2], a0[2])
