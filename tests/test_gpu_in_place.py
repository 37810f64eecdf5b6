"""Spectra calls whose output shares memory with the input rows, through the C
entry points: the results are those of separate buffers."""
import numpy as np
import pytest

from oracle import spectra_oracle as SP

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import _sp  # noqa: E402


def rows_of(M, N, seed):
    """Two tones and a ten-thousandth of noise, so that |z| stays away from zero."""
    rng = np.random.default_rng(seed)
    t = np.arange(N, dtype=float)
    return np.array([np.cos(2 * np.pi * rng.uniform(0.01, 0.2) * t + rng.uniform(0, 6.3))
                     + 1e-4 * rng.standard_normal(N) for _ in range(M)])


# one launch (4096) and three (9000, 48000) at the row's own length, convolutions
# (4095; 7001; 6561 alone, whose workspace does not hold the copy as well)
@pytest.mark.parametrize("M,N", [(3, 4096), (3, 4095), (1, 6561), (2, 7001), (2, 9000), (4, 48000)])
@pytest.mark.parametrize("where", ["freq", "amp", "freq one sample on", "amp one row on"])
def test_hilbert_in_place(M, N, where):
    """Bounds as for separate buffers: amplitudes within 1e-11 of a row's
    largest, frequencies within 1e-6 of the rate."""
    sr = 1000.0
    X = rows_of(M, N, N + M)
    pool = torch.empty((M * N + N,), dtype=torch.float64, device="cuda")
    shift = {"freq one sample on": 1, "amp one row on": N}.get(where, 0)
    x, shared = pool[:M * N], pool[shift:shift + M * N]
    x.copy_(torch.from_numpy(X).reshape(-1))
    other = torch.empty_like(shared)
    freq, amp = (shared, other) if where.startswith("freq") else (other, shared)
    ws = torch.empty((_sp.hilbert_workspace(M, N),), dtype=torch.uint8, device="cuda")
    _sp.hilbert_if(x, M, N, sr, freq, amp, ws)
    f, a = freq.cpu().numpy().reshape(M, N), amp.cpu().numpy().reshape(M, N)
    for r in range(M):
        of, oa = SP.hilbert_if(X[r], sr)
        assert np.max(np.abs(a[r] - oa)) <= 1e-11 * np.max(oa), r
        ok = oa > 1e-3 * oa.max()
        ok &= np.roll(ok, 1) & np.roll(ok, -1)
        assert np.max(np.abs(f[r] - of)[ok], initial=0.0) <= 1e-6 * sr, r
