"""What eemd_workspace_size asks for against what the engine's arrays hold (host only)."""
import pytest

from eemd4cuda_b200 import _lib as L


def size(dtype, n, trials, external, **kw):
    p = L.default_params()
    p.dtype = L.EEMD_F64 if dtype == "f64" else L.EEMD_F32
    p.max_imf = 8
    p.cluster_size = 8
    for k, v in kw.items():
        setattr(p, k, v)
    return L.workspace_size(p, [n], trials, external)


@pytest.mark.parametrize("dtype,b", [("f64", 8), ("f32", 4)])
@pytest.mark.parametrize("external", [False, True])
def test_bytes_per_sample(dtype, b, external):
    """Of a long signal on the 32-byte grid, per sample: the residual (and the
    IMF rows), a scratch row and a second residual; knots, two lists of half a
    sample each of either kind, an index and a value; half a record of either
    kind, four coefficients and an index; two run records of 4 bytes per 32
    bytes of samples.  Lists and tables are rounded up: 1 %."""
    n = 1 << 22
    per = b * (3 + (0 if external else 8)) + 2 * (4 + b) + (4 * b + 4) + 2 * 4 * b / 32
    got = size(dtype, n, 1, external) / n
    assert per <= got <= 1.01 * per
