"""Results through the pinned staging buffer against the direct pinned copies."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from eemd4cuda_b200 import emd_par as M  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.fixture
def small_stage(monkeypatch):
    """A staging buffer of 512 doubles (two halves of 256) and a result limit of 4096 bytes."""
    monkeypatch.setattr(M, "PINNED_RESULT_BYTES", 4096)
    monkeypatch.setattr(M, "_STAGE", {})


def test_staged_copies_of_every_slice_count(small_stage):
    pairs = []
    for i, n in enumerate((0, 1, 255, 256, 257, 512, 513, 2048, 2051)):
        src = torch.arange(n, dtype=torch.float64, device="cuda") + 10000 * i
        pairs.append((np.full((n,), -1.0), src))
    M._staged_copies(torch, pairs)
    for dst, src in pairs:
        assert np.array_equal(dst, src.cpu().numpy())


def _calls(x):
    trials = np.stack([x, x[::-1] * 1.5, np.zeros_like(x)])
    for kw in (dict(max_imf=-1), dict(max_imf=3), dict(max_imf=4, dtype="float32")):
        r = M.decompose(x, E=6, eps=0.2, seed=3, max_sifts=20, **kw)
        yield r.imfs, r.residual, r.stats["per_mode_sifts"] if "per_mode_sifts" in r.stats else ()
    for t in (trials, trials[2:]):
        yield M.gpu_eemd_full(t, E=len(t), max_imf=5, max_sifts=20)


@pytest.mark.parametrize("n", [64, 1501])
def test_staged_results_equal_direct_ones(n, request):
    x = np.cumsum(np.random.default_rng(n).standard_normal(n))
    direct = list(_calls(x))
    request.getfixturevalue("small_stage")
    for a, b in zip(direct, _calls(x)):
        for u, v in zip(a, b):
            u, v = np.asarray(u), np.asarray(v)
            assert u.dtype == v.dtype and np.array_equal(u, v)
