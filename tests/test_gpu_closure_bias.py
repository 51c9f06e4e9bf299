"""Bias gradients of the fused training pass: float64 sums over the rows, in a
fixed order, rounded to float32 once.

The network is chosen so that every summand is known exactly: zero W1, b1 and b2
make both hidden layers zero, where SiLU' is 1/2; W3 has one power of two a unit
and W2 one a column.  Then dY = 2 (b3 - t) / (n O) in float32, a unit's gradient
is that of one output, split into two bfloat16 terms as every operand of a
product is, times powers of two.  Tolerance: the last rounding, 2^-24 of the
sum, and n float64 additions, n 2^-53 of the summands' magnitudes.  A float32
sum of 65613 rows is off by about 1e-6 of the summands' magnitudes' root sum of
squares."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from calypso_b200 import closure  # noqa: E402
from oracle.mlp_oracle import bf16_round  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nhid,nout", [(64, 3), (160, 8), (256, 5)])
@pytest.mark.parametrize("rows", [1, 300, 65613])
def test_bias_gradients_are_float64_sums(nhid, nout, rows):
    rng = np.random.default_rng(rows + nhid)
    u = np.arange(nhid)
    W3, W2 = np.zeros((nout, nhid), np.float32), np.zeros((nhid, nhid), np.float32)
    s3 = (2.0 ** -(1 + u % 4) * np.where(u % 3, 1, -1)).astype(np.float32)
    W3[u % nout, u] = s3
    v = (3 * u + 1) % nhid          # W2[v][u]: unit v of the second layer feeds from unit u of the first
    s2 = (2.0 ** -(u % 3)).astype(np.float32)
    W2[v, u] = s2
    b3 = rng.standard_normal(nout).astype(np.float32)
    p = np.concatenate([np.zeros(16 * nhid + nhid, np.float32), W2.ravel(), np.zeros(nhid, np.float32), W3.ravel(), b3])
    net = closure.MLP(16, nhid, nout)
    net.set_params(p)
    x = torch.randn((rows, 16), generator=torch.Generator().manual_seed(1)).cuda()
    t = (b3 + rng.standard_normal((rows, nout))).astype(np.float32)
    td = torch.from_numpy(t).cuda()
    got = [net.loss_grad(x, td, want_grad=True)[1] for _ in range(2)]
    net.close()

    d = b3 - t
    dy = (np.float32(2.0) * d) / np.float32(rows * nout)
    hi = bf16_round(dy)
    split = hi + bf16_round((dy - hi.astype(np.float32)).astype(np.float32))
    dz2 = 0.5 * split[:, u % nout] * s3
    dz1 = 0.5 * dz2[:, v] * s2
    o1, o2 = 16 * nhid, 16 * nhid + nhid + nhid * nhid
    o3 = o2 + nhid + nout * nhid
    for at, n, terms in ((o1, nhid, dz1), (o2, nhid, dz2), (o3, nout, dy.astype(np.float64))):
        ref = terms.sum(0, dtype=np.float64)
        tol = 2.0 ** -24 * np.abs(ref) + rows * 2.0 ** -53 * np.abs(terms).sum(0)
        for g in got:
            assert np.all(np.abs(g[at:at + n] - ref) <= tol), (at, np.max(np.abs(g[at:at + n] - ref) / tol))
        assert np.array_equal(got[0][at:at + n], got[1][at:at + n])
