"""The fused training pass computes what the layer-by-layer kernels do.

A network of 16 inputs takes the fused kernels; the same network with 17 more
inputs of zero weight and zero value takes the general ones, and every product
then has the same terms in the same order.  Batches of at most 256 rows are one
chunk of each sum over the rows, so their weight gradients are equal bit for
bit.  Larger batches add nz chunks in an order that is not fixed: each side is
within nz 2^-24 of the sum of the terms' magnitudes.  The loss is a float64 sum
of n O equal terms in another order."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from calypso_b200 import closure  # noqa: E402

pytestmark = pytest.mark.gpu

WIDE = 33


def networks(nhid, nout, rows, seed):
    """(network, x, t) on 16 and on 33 inputs, the parameters by block"""
    rng = np.random.default_rng(seed)
    W1 = rng.uniform(-0.43, 0.43, (nhid, 16)).astype(np.float32)
    rest = [rng.uniform(-a, a, s).astype(np.float32) for a, s in
            ((0.1, nhid), (0.11, (nhid, nhid)), (0.1, nhid), (0.11, (nout, nhid)), (0.1, nout))]
    x = rng.standard_normal((rows, 16)).astype(np.float32)
    t = torch.from_numpy(rng.standard_normal((rows, nout)).astype(np.float32)).cuda()
    out = []
    for nin in (16, WIDE):
        w = np.zeros((nhid, nin), np.float32)
        w[:, :16] = W1
        net = closure.MLP(nin, nhid, nout)
        net.set_params(np.concatenate([w.ravel()] + [b.ravel() for b in rest]))
        xd = torch.zeros((rows, nin), device="cuda")
        xd[:, :16] = torch.from_numpy(x).cuda()
        out.append((net, xd, t))
    return out


def blocks(g, nin, nhid, nout):
    s = [(nhid, nin), (nhid,), (nhid, nhid), (nhid,), (nout, nhid), (nout,)]
    b = [v.reshape(sh) for v, sh in zip(np.split(g, np.cumsum([int(np.prod(q)) for q in s])[:-1]), s)]
    b[0] = b[0][:, :16]
    return b


def gradients(nhid, nout, rows, seed):
    got = []
    for nin, (net, x, t) in zip((16, WIDE), networks(nhid, nout, rows, seed)):
        loss, g = net.loss_grad(x, t, want_grad=True)
        got.append((loss, blocks(g, nin, nhid, nout)))
        net.close()
    return got


@pytest.mark.parametrize("nhid,nout", [(64, 3), (160, 8), (256, 5)])
@pytest.mark.parametrize("rows", [1, 129, 256])
def test_one_chunk_is_equal(nhid, nout, rows):
    (l0, g0), (l1, g1) = gradients(nhid, nout, rows, rows)
    assert abs(l0 - l1) <= rows * nout * 2.0 ** -53 * l1
    for q in (0, 2, 4):
        assert np.array_equal(g0[q], g1[q]), q


@pytest.mark.parametrize("nhid,nout,rows", [(256, 5, 16384), (160, 8, 40001)])
def test_many_chunks_agree(nhid, nout, rows):
    (l0, g0), (l1, g1) = gradients(nhid, nout, rows, 7)
    assert abs(l0 - l1) <= rows * nout * 2.0 ** -53 * l1
    # sums of the terms' magnitudes, float64
    (net, x, t) = networks(nhid, nout, rows, 7)[0]
    W1, b1, W2, b2, W3, b3 = (torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in blocks(net.params(), 16, nhid, nout))
    W1, W2, W3 = (w.bfloat16().double() for w in (W1, W2, W3))
    act = torch.nn.functional.silu
    z1 = (x.double() @ W1.T + b1).requires_grad_()
    h1 = act(z1)
    z2 = (h1 @ W2.T + b2)
    z2.retain_grad()
    h2 = act(z2)
    y = h2 @ W3.T + b3
    y.retain_grad()
    ((y - t) ** 2).mean().backward()
    S = [z1.grad.abs().T @ x.double().abs(), z2.grad.abs().T @ h1.abs(), y.grad.abs().T @ h2.abs()]
    nz = rows // 256 + 1
    for q, s in zip((0, 2, 4), S):
        assert np.all(np.abs(g0[q] - g1[q]) <= 2 * nz * 2.0 ** -24 * s.detach().cpu().numpy()), q
    net.close()
