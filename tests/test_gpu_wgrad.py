"""The warp-specialised weight gradient (operands read MN-major through tensor
maps) at the edges of its tiles, against the float64 oracle on the same bf16
operands, and the loss kernel's block sums."""
import numpy as np
import pytest

from oracle import surrogate_oracle as SO

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import _sg  # noqa: E402


def bf16(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(torch.bfloat16)


# one sample, a tile of 128 and one to either side, dilations of up to a tile,
# more tiles than one wave of CTAs; the padded and the whole channel counts
@pytest.mark.parametrize("N,C,nv,cv", [(64, 64, 64, 64), (16, 64, 6, 64), (64, 16, 64, 11), (16, 16, 10, 16)])
@pytest.mark.parametrize("B,T,dil", [(1, 1, 1), (2, 127, 1), (3, 128, 128), (2, 129, 64), (2, 1000, 37), (5, 8197, 2)])
def test_weight_gradient_tiles(N, C, nv, cv, B, T, dil):
    """A sum of B T products of bf16 values in float32 (rounded or truncated
    at 2^-23 of the running sum per addition, a random walk of B T of them):
    within 1e-5 sqrt(B T) of the products' unit variance."""
    rng = np.random.default_rng(T + dil)
    dy, x = bf16(rng.standard_normal((B, T, N))), bf16(rng.standard_normal((B, T, C)))
    dw = torch.zeros((nv, 3, cv), dtype=torch.float32, device="cuda")
    db = torch.zeros((nv,), dtype=torch.float32, device="cuda")
    err = torch.zeros((1,), dtype=torch.int32, device="cuda")
    _sg.wgrad(dy.cuda(), x.cuda(), dw, db, B, T, N, C, nv, cv, dil, err=err)
    torch.cuda.synchronize()
    assert int(err.item()) == 0
    ow, ob = SO.conv_weight_grad(dy.double().numpy(), x.double().numpy(), dil)
    tol = 1e-5 * max(1.0, np.sqrt(B * T)) * 4
    assert np.max(np.abs(dw.cpu().numpy() - ow[:nv, :, :cv])) <= tol
    assert np.max(np.abs(db.cpu().numpy() - ob[:nv])) <= tol


@pytest.mark.parametrize("B,T", [(1, 41), (3, 300), (16, 4096)])
def test_loss_sums(B, T):
    """The mean squared loss and its gradient from fewer than one CTA's
    elements to several turns of every CTA (float32 sums: 1e-5 of the loss;
    the gradient in bf16: 2^-8)."""
    rng = np.random.default_rng(B)
    C, cv, margin = 16, 6, 20
    out, tgt = bf16(rng.standard_normal((B, T, C))), bf16(rng.standard_normal((B, T, C)))
    dout = torch.empty((B, T, C), dtype=torch.bfloat16, device="cuda")
    acc = torch.zeros((1,), dtype=torch.float32, device="cuda")
    _sg.loss(out.cuda(), None, tgt.cuda(), dout, acc, B, T, C, cv, margin)
    d = (out.double() - tgt.double()).numpy()
    d[:, :margin] = d[:, T - margin:] = 0.0
    d[..., cv:] = 0.0
    count = B * (T - 2 * margin) * cv
    assert abs(float(acc.item()) - np.sum(d * d) / count) <= 1e-5 * np.sum(d * d) / count
    g = 2.0 * d / count
    assert np.max(np.abs(dout.double().cpu().numpy() - g)) <= 2 ** -8 * np.max(np.abs(g))


@pytest.mark.parametrize("project", [False, True])
def test_pack_layers_equals_pack_and_bias(project):
    """One launch for every layer gives each layer's own eemd_sg_pack (both
    operands) and eemd_sg_bias, bit for bit, padded channel counts included."""
    g = torch.Generator().manual_seed(1)
    layers, want = [], []
    for N, C, nv, cv in [(64, 16, 64, 11), (64, 64, 64, 64), (16, 64, 6, 64), (16, 16, 10, 16)]:
        w, b = torch.randn((nv, 3, cv), generator=g).cuda(), torch.randn((nv,), generator=g).cuda()
        outs = [[torch.full((N * 3 * C,), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2)]
                + [torch.full((N,), 7.0, device="cuda")] for _ in range(2)]
        layers.append((w, b, *outs[0], N, C, nv, cv, project))
        _sg.pack(w, outs[1][0], N, C, nv, cv, project=project)
        _sg.pack(w, outs[1][1], C, N, cv, nv, transpose=True, project=project)
        _sg.bias(b, outs[1][2], N, nv, project=project)
        want.append(outs)
    _sg.pack_layers(layers)
    torch.cuda.synchronize()
    for got, ref in want:
        assert all(torch.equal(u, v) for u, v in zip(got, ref))
