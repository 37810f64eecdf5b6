"""One layer of the surrogate network at a time against the pass that launches them all."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

from eemd4cuda_b200 import surrogate  # noqa: E402


@pytest.mark.parametrize("tensor_cores", [True, False])
def test_layers_one_by_one_equal_the_pass(tensor_cores):
    B, T = 2, 300
    net = surrogate.Net(seed=3)
    g = torch.Generator(device="cuda").manual_seed(1)
    x = torch.randn((B, T, surrogate.CH), generator=g, device="cuda").bfloat16()
    acts = net.forward(x, B, T, tensor_cores)
    src = x
    for i in range(len(net.layers)):
        dst = torch.empty_like(acts[i + 1])
        net.layer(i, src, dst, B, T, tensor_cores)
        assert torch.equal(dst, acts[i + 1]), i
        src = dst
    net.check()
