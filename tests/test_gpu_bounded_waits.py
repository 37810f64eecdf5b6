"""The warp-specialised kernels under a poll limit of one: a call either gives
the right result or says that a wait gave up, and leaves the device as it was."""
import numpy as np
import pytest

from oracle import surrogate_oracle as SO

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import _sg  # noqa: E402


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(torch.bfloat16)


@pytest.mark.parametrize("limit", [1, 0])
@pytest.mark.parametrize("N,C", [(64, 64), (16, 64), (64, 16)])
def test_weight_gradient(N, C, limit):
    """Within 4e-5 sqrt(B T) of the float64 sums, as at the tiles' edges."""
    B, T, dil = 4, 20000, 3  # several tiles per CTA
    rng = np.random.default_rng(N + C)
    dy, x = bf16(rng.standard_normal((B, T, N))), bf16(rng.standard_normal((B, T, C)))
    dw = torch.zeros((N, 3, C), dtype=torch.float32, device="cuda")
    db = torch.zeros((N,), dtype=torch.float32, device="cuda")
    err = torch.zeros((1,), dtype=torch.int32, device="cuda")
    _sg.wgrad(dy.cuda(), x.cuda(), dw, db, B, T, N, C, N, C, dil, err=err, spin_limit=limit)
    status = int(err.item())
    assert status == 0 or (limit == 1 and status == _sg.SG_E_TIMEOUT)
    if status == 0:
        ow, ob = SO.conv_weight_grad(dy.double().numpy(), x.double().numpy(), dil)
        tol = 4e-5 * np.sqrt(B * T)
        assert np.max(np.abs(dw.cpu().numpy() - ow)) <= tol and np.max(np.abs(db.cpu().numpy() - ob)) <= tol


@pytest.mark.parametrize("limit", [1, 0])
@pytest.mark.parametrize("cin,cout", [(64, 64), (16, 64), (64, 16)])
def test_convolution(cin, cout, limit):
    """The same bits as the tensor-core form without warp roles."""
    B, T, dil = 4, 20000, 3
    rng = np.random.default_rng(cin + cout)
    x = bf16(rng.standard_normal((B, T, cin))).cuda()
    wp = torch.empty((cout * 3 * cin,), dtype=torch.bfloat16, device="cuda")
    _sg.pack(torch.from_numpy(rng.standard_normal((cout, 3, cin)).astype(np.float32)).cuda(), wp, cout, cin, cout, cin)
    y, ref = (torch.empty((B, T, cout), dtype=torch.bfloat16, device="cuda") for _ in range(2))
    err = torch.zeros((1,), dtype=torch.int32, device="cuda")
    _sg.conv(x, wp, None, ref, B, T, cin, cout, dil, tensor_cores=1, err=err)
    _sg.conv(x, wp, None, y, B, T, cin, cout, dil, tensor_cores=4, err=err, spin_limit=limit)
    status = int(err.item())
    assert status == 0 or (limit == 1 and status == _sg.SG_E_TIMEOUT)
    if status == 0:
        assert torch.equal(y, ref)
