"""The warp-specialised convolution's two epilogue groups (even and odd tiles of
a CTA) and its first copies, from one tile on the device to four per CTA,
against the single-buffered kernel bit for bit; and the closing reductions of a
training step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import _sg  # noqa: E402


def conv(mode, x, wp, b, B, T, cin, cout, **kw):
    err = torch.zeros((1,), dtype=torch.int32, device="cuda")
    y = torch.full((B, T, cout), 7.0, dtype=torch.bfloat16, device="cuda")
    _sg.conv(x, wp, b, y, B, T, cin, cout, 3, tensor_cores=mode, err=err, **kw)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    return y


@pytest.mark.parametrize("cin,cout", [(16, 64), (64, 64), (64, 16)])
@pytest.mark.parametrize("tiles,ragged", [(1, 127), (2, 0), (147, 1), (149, 5), (297, 0), (445, 64), (593, 3)])
def test_tiles_per_cta(cin, cout, tiles, ragged):
    T = tiles * 128 - ragged
    g = torch.Generator().manual_seed(tiles + cin + cout)
    x = torch.randn((1, T, cin), generator=g).to(torch.bfloat16).cuda()
    w = (torch.randn((cout, 3, cin), generator=g) / np.sqrt(3 * cin)).cuda()
    wp = torch.empty((cout * 3 * cin,), dtype=torch.bfloat16, device="cuda")
    _sg.pack(w, wp, cout, cin, cout, cin)
    b = torch.randn((cout,), generator=g).cuda()
    # a mask's zeros of both signs, negatives and numbers that are none let nothing through
    mask = torch.randn((1, T, cout), generator=g).to(torch.bfloat16)
    mask.view(-1)[::7], mask.view(-1)[3::11], mask.view(-1)[5::13] = 0.0, -0.0, float("nan")
    for kw in (dict(relu=True), dict(relu=False), dict(relu=False, direction=-1, mask=mask.cuda())):
        bias = None if "mask" in kw else b
        one, ws = (conv(m, x, wp, bias, 1, T, cin, cout, **kw) for m in (1, 4))
        assert torch.equal(one.view(torch.int16), ws.view(torch.int16))


@pytest.mark.parametrize("B,T,project", [(1, 41, False), (2, 9000, True), (32, 4096, True), (33, 4100, False)])
@pytest.mark.parametrize("delta", [0.0, 0.7])
def test_loss_turns(B, T, project, delta):
    """Fewer elements than one turn of the grid to nine turns (of four at a
    time), squared and Huber loss, with and without the zero-sum projection:
    float32 sums within 1e-5 of the loss, the gradient within bf16's 2^-8."""
    C, cv, margin = 16, 10, 20
    g = torch.Generator().manual_seed(B)
    out, tgt = (torch.randn((B, T, C), generator=g).to(torch.bfloat16) for _ in range(2))
    dout = torch.full((B, T, C), 7.0, dtype=torch.bfloat16, device="cuda")
    acc = torch.zeros((1,), dtype=torch.float32, device="cuda")
    _sg.loss(out.cuda(), None, tgt.cuda(), dout, acc, B, T, C, cv, margin, project=project, delta=delta)
    d = (out.double() - tgt.double()).numpy()
    d[:, :margin] = d[:, T - margin:] = 0.0
    d[..., cv:] = 0.0
    count = B * (T - 2 * margin) * cv
    big = np.abs(d) > delta if delta > 0 else np.zeros(d.shape, bool)
    loss = np.where(big, 2 * delta * np.abs(d) - delta ** 2, d * d).sum() / count
    grad = 2.0 * np.where(big, delta * np.sign(d), d) / count
    if project:
        grad[..., :cv] -= grad.sum(-1, keepdims=True) / cv
    assert abs(float(acc.item()) - loss) <= 1e-5 * loss
    assert np.max(np.abs(dout.double().cpu().numpy() - grad)) <= 2 ** -8 * np.max(np.abs(grad))
