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


@pytest.mark.parametrize("tensor_cores", [True, False])
def test_passes_in_one_call_equal_layer_by_layer(tensor_cores):
    """A network's forward and backward pass against the same kernels called
    one by one: the same activations, and gradients within the float32 rounding
    of sums added in another order (B T products, as the weight-gradient tests)."""
    from eemd4cuda_b200 import surrogate as SU

    B, T = 2, 300
    net = SU.Net(seed=3)
    g = torch.Generator().manual_seed(1)
    x = torch.randn((B, T, SU.CH), generator=g).to(torch.bfloat16).cuda()
    dout = torch.randn((B, T, SU.CH), generator=g).to(torch.bfloat16).cuda()
    acts = net.forward(x, B, T, tensor_cores)
    net.backward(acts, dout, B, T, tensor_cores)
    mode = net.conv_kernel if tensor_cores else 0
    got, src, dy = net.grads.clone(), x, dout
    for i, lay in enumerate(net.layers):
        y = torch.empty_like(acts[i + 1])
        _sg.conv(src, lay["wp"], lay["bias"], y, B, T, lay["cin_p"], lay["cout_p"], lay["dil"], relu=lay["relu"],
                 tensor_cores=mode, err=net.err)
        assert torch.equal(y, acts[i + 1])
        src = y
    net.grads.zero_()
    for i in range(len(net.layers) - 1, -1, -1):
        lay = net.layers[i]
        _sg.wgrad(dy, acts[i], lay["dw"], lay["db"], B, T, lay["cout_p"], lay["cin_p"], lay["cout_v"], lay["cin_v"],
                  lay["dil"], tensor_cores=tensor_cores)
        dx = torch.empty((B, T, lay["cin_p"]), dtype=torch.bfloat16, device="cuda")
        _sg.conv(dy, lay["wt"], None, dx, B, T, lay["cout_p"], lay["cin_p"], lay["dil"], direction=-1, mask=acts[i],
                 tensor_cores=mode, err=net.err)
        dy = dx
    net.check()
    scale = float(net.grads.abs().max())
    assert scale > 0 and float((got - net.grads).abs().max()) <= 4e-5 * np.sqrt(B * T) * scale


def test_a_refused_layer_ends_the_pass():
    x = torch.zeros((1, 64, 16), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(_sg.SurrogateError) as e:
        _sg.forward_layers([(x, x, None, x, None, 16, 48, 1, 1, False)], 1, 64, tensor_cores=4)
    assert e.value.status == _sg.SG_E_BADARG
