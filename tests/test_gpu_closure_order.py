"""The closure network's parameters are read and written in the order of the
calls, whichever stream a call works on: the network's own, or that of a
context the network is attached to.  Networks of 2048 units make each update
long enough (4 million parameters) for a queue of them to build up."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from calypso_b200 import PREC_MIXED, SphMHD, closure, configs  # noqa: E402
from oracle import mlp_oracle  # noqa: E402

pytestmark = pytest.mark.gpu

WIDE = 2048
FORCES = 48     # d_rj slot the closure adds to


def batch(rows, seed=0):
    g = torch.Generator().manual_seed(seed)
    return torch.randn((rows, 16), generator=g).cuda(), torch.randn((rows, 5), generator=g).cuda()


def test_parameters_read_behind_queued_updates():
    net = closure.MLP(16, WIDE, 5, seed=1)
    start = net.params()
    net.loss_grad(*batch(64))
    for _ in range(100):
        net.adam_step(1e-3)
    p = net.params()
    net.sync()
    assert np.array_equal(p, net.params())
    # set behind the queue, too
    for _ in range(100):
        net.adam_step(1e-3)
    net.set_params(start)
    net.sync()
    assert np.array_equal(start, net.params())
    net.close()


def test_set_parameters_are_the_ones_used():
    net = closure.MLP(16, 256, 5, seed=1)
    x, _ = batch(64)
    p0 = net.params()
    for i in range(60):
        p = np.roll(p0, 7 * i)
        net.set_params(p)
        y = net.forward(x).cpu().numpy()
        ref, _ = mlp_oracle.forward(p, x.cpu().numpy(), 16, 256, 5)
        assert np.linalg.norm(y - ref) < 1e-4 * np.linalg.norm(ref), i
    net.close()


def shell_with(net):
    p = configs.shell_params(15, 9, 24, 48, E=1e-3, Ra=100.0, dt=5e-5)
    g = SphMHD(p, PREC_MIXED)
    n = p["nr"]
    norm = np.concatenate([np.zeros(16 * n), np.ones(16 * n), 1e-2 * np.ones(5 * n)]).astype(np.float32)
    closure._check(closure._lib().cb2_closure_attach(g._h, net._h, closure._fptr(norm)), "cb2_closure_attach")
    g.init_fields(2, 3)
    g.step(2)
    return g


@pytest.mark.parametrize("graph", [False, True])
def test_step_reads_behind_queued_updates(graph):
    got = []
    for drained in (True, False):
        net = closure.MLP(16, WIDE, 5, seed=1)
        g = shell_with(net)
        g.step(1, graph=graph)
        g.sync()
        net.loss_grad(*batch(64))
        for _ in range(100):
            net.adam_step(1e-3)
        if drained:
            net.sync()
        g.step(1, graph=graph)
        got.append(g.get_field(FORCES))
        g.close()
        net.close()
    assert np.array_equal(*got)


@pytest.mark.parametrize("graph", [False, True])
def test_update_waits_for_queued_steps(graph):
    got = []
    for drained in (True, False):
        net = closure.MLP(16, WIDE, 5, seed=1)
        g = shell_with(net)
        net.loss_grad(*batch(64))
        net.sync()
        g.step(6, graph=graph)
        if drained:
            g.sync()
        net.adam_step(0.1)
        got.append(g.get_field(FORCES))
        g.close()
        net.close()
    assert np.array_equal(*got)


@pytest.mark.parametrize("graph", [False, True])
def test_passes_wait_for_queued_steps(graph):
    # a network of these widths has one set of work buffers for all its passes
    got = []
    x, t = batch(1000)
    for drained in (True, False):
        net = closure.MLP(16, WIDE, 5, seed=1)
        g = shell_with(net)
        net.loss_grad(x, t)          # buffers of their largest size
        out = []
        for call in (lambda: net.forward(x).cpu().numpy(), lambda: np.array(net.loss_grad(x, t))):
            g.step(6, graph=graph)
            if drained:
                g.sync()
            out.append(call())
        got.append(out + [g.get_field(FORCES)])
        g.close()
        net.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def test_network_closed_before_its_context():
    net = closure.MLP(16, 64, 5, seed=1)
    g = shell_with(net)
    net.close()
    g.step(2)                       # the plain step from here on
    assert np.all(np.isfinite(g.energies()))
    g.close()
