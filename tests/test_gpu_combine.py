"""The served decomposition and its gate metrics over batches and chunk counts
around the kernels' edges, against the numpy restatement."""
import numpy as np
import pytest

from oracle import surrogate_oracle as SO

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import _sg  # noqa: E402


@pytest.mark.parametrize("S,N,chunks,P", [(1, 100, 1, 6), (1, 127, 200, 3), (3, 4099, 9, 0), (130, 257, 32, 6)])
def test_combine_and_gate(S, N, chunks, P):
    """Float64 sums of at most N terms in another order: 1e-12 of the largest
    value, and of the metrics' O(1) cross terms."""
    rng = np.random.default_rng(S + N)
    K, C = 10, 16
    sums = rng.standard_normal((S, K, N))
    count = rng.integers(0, 9, (S, K)).astype(np.int32)  # powers of two, others, and none
    sums[count == 0] = 0.0
    x = rng.standard_normal((S, N)).astype(np.float32)
    scale = (0.5 + rng.random(S)).astype(np.float32)
    net = torch.from_numpy(rng.standard_normal((S, N, C)).astype(np.float32)).to(torch.bfloat16)
    dev = [torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (sums, count, x, scale)]
    imfs = torch.empty((S, K, N), dtype=torch.float64, device="cuda")
    resid = torch.empty((S, N), dtype=torch.float64, device="cuda")
    partial = torch.empty((S * chunks * _sg.stat_count(),), dtype=torch.float64, device="cuda")
    metrics = torch.empty((S, 4), dtype=torch.float64, device="cuda")
    fallback = torch.empty((S,), dtype=torch.int32, device="cuda")
    _sg.combine(*dev, net.cuda(), imfs, resid, partial, chunks, S, N, K, C, P, 1e-6, 0.0, metrics, fallback)
    oi, orr, recon, io_p, io, io_ref = SO.combine(sums, count, x, scale.astype(np.float64), net.double().numpy(), P)
    top = np.abs(oi).max()
    assert np.max(np.abs(imfs.cpu().numpy() - oi)) <= 1e-12 * top
    assert np.max(np.abs(resid.cpu().numpy() - orr)) <= 1e-12 * max(top, np.abs(orr).max())
    m = metrics.cpu().numpy()
    for got, want in ((m[:, 1], io_p), (m[:, 2], io), (m[:, 3], io_ref)):
        assert np.max(np.abs(got - want)) <= 1e-12 * max(1.0, np.abs(want).max()) * K * K
    assert np.all(m[:, 0] <= 1e-12) and np.all(recon <= 1e-12)
    want = np.abs(io_p) - np.abs(io_ref) > 0.0
    sure = np.abs(np.abs(io_p) - np.abs(io_ref)) > 1e-9
    assert np.array_equal(fallback.cpu().numpy().astype(bool)[sure], want[sure])
