"""A closure network whose products' waits have a budget of zero (one try,
CB2_PIPE_WAIT_NS=0 at its creation) gives up at its first wait that is not
complete: the kernels drain their products, free their tensor memory and return,
and the call reports CB2_ERR_TIMEOUT.  Another network then runs as ever.  Many
tiles a CTA.  (The general kernels' products are complete whenever the threads
that stage the next operands get to look.)"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from calypso_b200 import CalypsoError, closure  # noqa: E402
from calypso_b200.sph_mhd import ERR_TIMEOUT  # noqa: E402
from oracle import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nhid", [64, 256])
def test_wait_that_runs_out_is_reported(nhid, monkeypatch):
    rows = 128 * 148 * 3 + 5
    x = torch.randn((rows, 16), generator=torch.Generator().manual_seed(1)).cuda()
    t = torch.randn((rows, 5), generator=torch.Generator().manual_seed(2)).cuda()
    monkeypatch.setenv("CB2_PIPE_WAIT_NS", "0")
    net = closure.MLP(16, nhid, 5, seed=2)
    monkeypatch.delenv("CB2_PIPE_WAIT_NS")
    for call in (lambda: net.forward(x), lambda: net.loss_grad(x, t)):
        with pytest.raises(CalypsoError) as e:
            call()
        assert e.value.code == ERR_TIMEOUT
    net.close()
    net = closure.MLP(16, nhid, 5, seed=2)
    y, _ = mlp_oracle.forward(net.params(), x.cpu().numpy(), 16, nhid, 5)
    got = net.forward(x).cpu().numpy()
    assert np.linalg.norm(got - y) < 1e-4 * np.linalg.norm(y)
    assert np.isfinite(net.loss_grad(x, t))
    net.close()
