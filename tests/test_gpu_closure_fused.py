"""The closure network's one-kernel passes (forward, data gradient, weight
gradients) against the float64 oracle at the edges of their row tiles and of
the sizes they take, and the general kernels beyond those sizes.

Tolerance 1e-4 relative L2: an activation enters a product as bfloat16 hi +
lo, 2^-17 of its value off, in two (forward) to four (gradient) products in a
row, and a sum over up to 256 units may be about ten times smaller than its
terms: 4 x 10 x 2^-17 = 3e-4 in the worst case, a third of that in the L2
norm."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from calypso_b200 import closure  # noqa: E402
from oracle import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


# (nin, nhid, nout): the closure's own, a vector-load remainder, every limit
# of the fused passes, one beyond each (33 inputs, 288 and 40 units, 9 outputs)
SIZES = [(16, 256, 5), (7, 64, 3), (32, 160, 8), (33, 64, 4), (8, 288, 5), (16, 40, 5), (16, 64, 9)]


@pytest.mark.parametrize("nin,nhid,nout", SIZES)
@pytest.mark.parametrize("rows", [1, 127, 128, 129, 2500])
def test_passes_match_oracle(nin, nhid, nout, rows):
    net = closure.MLP(nin, nhid, nout, seed=3)
    rng = np.random.default_rng(rows)
    x = rng.standard_normal((rows, nin)).astype(np.float32)
    t = rng.standard_normal((rows, nout)).astype(np.float32)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    p = net.params()
    p[nin * nhid:nin * nhid + nhid] = rng.standard_normal(nhid) * 0.1      # biases
    net.set_params(p)
    y, _ = mlp_oracle.forward(p, x, nin, nhid, nout)
    assert rel(net.forward(xd).cpu().numpy(), y) < 1e-4
    loss, g = net.loss_grad(xd, td, want_grad=True)
    loss_o, g_o = mlp_oracle.loss_grad(p, x, t, nin, nhid, nout)
    assert abs(loss - loss_o) < 1e-4 * loss_o
    o = 0
    for s in [nhid * nin, nhid, nhid * nhid, nhid, nout * nhid, nout]:
        assert rel(g[o:o + s], g_o[o:o + s]) < 1e-4, (o, s)
        o += s
    net.close()


def test_rows_beyond_one_tile_a_cta():
    """more tiles than SMs: every CTA walks several, the last one partial"""
    rows = 148 * 128 * 2 + 77
    net = closure.MLP(16, 256, 5, seed=4)
    x = torch.randn((rows, 16), generator=torch.Generator().manual_seed(1))
    t = torch.randn((rows, 5), generator=torch.Generator().manual_seed(2))
    p = net.params()
    y, _ = mlp_oracle.forward(p, x.numpy(), 16, 256, 5)
    assert rel(net.forward(x.cuda()).cpu().numpy(), y) < 1e-4
    # rows that start off a 16-byte boundary
    flat = torch.zeros(rows * 16 + 1, device="cuda")
    flat[1:] = x.cuda().reshape(-1)
    assert rel(net.forward(flat[1:].view(rows, 16)).cpu().numpy(), y) < 1e-4
    loss, g = net.loss_grad(x.cuda(), t.cuda(), want_grad=True)
    loss_o, g_o = mlp_oracle.loss_grad(p, x.numpy(), t.numpy(), 16, 256, 5)
    assert abs(loss - loss_o) < 1e-4 * loss_o and rel(g, g_o) < 1e-4
    net.close()
