"""A workspace at any address: a slice of a pool at 16 bytes past a 32-byte
boundary, where the engine's 32-byte accesses would not be aligned, or at an
odd byte, of exactly the size asked for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import _lib as L  # noqa: E402
from eemd4cuda_b200 import emd_par as M  # noqa: E402


@pytest.mark.parametrize("dtype,exact", [(np.float64, False), (np.float64, True), (np.float32, False)])
@pytest.mark.parametrize("external", [False, True])
def test_workspace_address(dtype, exact, external):
    """The same bits as in a workspace at the start of an allocation, with the
    caller's IMF rows and without, on rows off the 32-byte grid and on it."""
    E, M_, lengths = 3, 4, [1001, 4096]
    total = sum(lengths)
    x = torch.from_numpy(np.random.default_rng(3).standard_normal(total).astype(dtype)).cuda()
    p = M.make_params(dtype=dtype, noise_mode=L.EEMD_NOISE_PHILOX, seed=4, eps=0.2, tau=0.25, max_sifts=9, max_imf=M_,
                      exact=exact)
    need = L.workspace_size(p, lengths, E, external)
    got = []
    for at in (0, 16, 8, 1, 31):
        pool = torch.empty((need + at,), dtype=torch.uint8, device="cuda")
        ws = pool[at:]
        assert ws.data_ptr() % 32 == at
        imfs = torch.zeros((E * M_ * total,), dtype=x.dtype, device="cuda") if external else None
        s = torch.zeros((M_ * total,), dtype=torch.float64, device="cuda")
        c = torch.zeros((2 * M_,), dtype=torch.int32, device="cuda")
        r = torch.zeros((E * total,), dtype=x.dtype, device="cuda")
        n = torch.zeros((2 * E,), dtype=torch.int32, device="cuda")
        L.run(p, x, lengths, 0, E, ws, imfs=imfs, resid_out=r, imf_sum=s, mode_count=c, nsift=n)
        got.append((s, c, r, n) + ((imfs,) if external else ()))
    assert int(got[0][3].sum()) > 0 and bool(got[0][0].any())
    for other in got[1:]:
        assert all(torch.equal(a, b) for a, b in zip(got[0], other))
