"""Device and host memory that calls and their results hold."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import emd_par, surrogate  # noqa: E402


def test_backward_holds_two_input_gradients():
    """Whatever the number of layers: the gradient a layer reads and the one it
    writes, each [B][T][HIDDEN] in bf16."""
    B, T = 8, 8192
    net = surrogate.Net(seed=0)
    g = torch.Generator(device="cuda").manual_seed(1)
    inp = torch.randn((B, T, surrogate.CH), generator=g, device="cuda").bfloat16()
    dout = torch.randn((B, T, surrogate.CH), generator=g, device="cuda").bfloat16()
    acts = net.forward(inp, B, T)
    net.backward(acts, dout, B, T)
    torch.cuda.synchronize()
    base = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    net.backward(acts, dout, B, T)
    torch.cuda.synchronize()
    net.check()
    one = B * T * surrogate.HIDDEN * 2
    assert torch.cuda.max_memory_allocated() - base <= 2 * one + (1 << 20)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
def test_a_kept_residual_keeps_no_imf_rows(dtype):
    x = np.random.default_rng(2).standard_normal(4096)
    r = emd_par.decompose(x, E=1, max_imf=5, dtype=dtype)
    assert r.residual.base.untyped_storage().nbytes() == r.residual.nbytes
    tol = 1e-12 if dtype is np.float64 else 1e-5  # rounding of the stored rows
    assert np.max(np.abs(r.imfs.sum(axis=0) + r.residual - x)) <= tol * np.max(np.abs(x))


@pytest.mark.parametrize("max_imf", [-1, 12])
def test_a_large_ensemble_keeps_its_modes_only(max_imf):
    """More than 64 MB of IMF slots: the rows past the mode count are given back."""
    n = 1 << 20
    x = np.sin(0.05 * np.arange(n))
    r = emd_par.decompose(x, E=2, eps=1e-3, max_imf=max_imf, seed=1, max_sifts=5)
    assert r.imfs.shape == (r.n_modes, n) and r.n_modes > 0
    assert r.imfs.base is None and r.imfs.flags.owndata and r.imfs.flags.writeable
    assert np.max(np.abs(r.imfs.sum(axis=0) + r.residual - x)) <= 1e-12
