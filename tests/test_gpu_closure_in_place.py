"""cb2_mlp_forward with an output that overlaps its input gives the values of the
call with buffers of their own, for the fused kernels (64 units) and the general
ones (40 units): more rows than one tile a CTA, so that some are read after
others have been written."""
import pytest

torch = pytest.importorskip("torch")

from calypso_b200 import closure  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nhid", [40, 64])
@pytest.mark.parametrize("shift", [-3, 0, 1000])
def test_output_over_the_input(nhid, shift):
    rows = 148 * 128 * 2 + 77
    net = closure.MLP(16, nhid, 5, seed=2)
    x = torch.randn((rows, 16), generator=torch.Generator().manual_seed(1)).cuda()
    ref = net.forward(x)
    buf = torch.zeros(4 + rows * 16, device="cuda")
    buf[4:] = x.reshape(-1)
    torch.cuda.synchronize()
    xp = buf.data_ptr() + 16
    closure._check(closure._lib().cb2_mlp_forward(net._h, xp, rows, xp + 4 * shift), "cb2_mlp_forward")
    y = buf[4 + shift:4 + shift + rows * 5].view(rows, 5)
    assert torch.equal(y, ref)
    net.close()
