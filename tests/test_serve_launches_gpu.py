"""The server's count of step kernels is the backend's own, and the batch's is
what its runs enqueued: one launch per step, or per two where the members'
records exceed what the L2 holds."""
import pytest

from pfa_gb300 import ic
from pfa_gb300.serve import GpuBackend, Request, Server
from test_serve_cpu import Clock, FakeBackend, _req, _server


class CountingBackend(FakeBackend):
    def advance(self, steps_2d, handles_2d, items_3d):
        super().advance(steps_2d, handles_2d, items_3d)
        return 7


def test_counts_are_the_backends():
    reqs = [_req(0, (12, 12), 250), _req(1, (6, 6, 6), 130)]
    srv = Server(CountingBackend(10 ** 6, 10 ** 6), tick_steps=100, clock=Clock())
    srv.run_trace(list(reqs), realtime=False)
    assert srv.step_launches == 7 * srv.ticks
    srv, be = _server(10 ** 6, 10 ** 6)  # one that does not count: every step
    srv.run_trace(list(reqs), realtime=False)
    assert srv.step_launches == sum(n + sum(m) for n, m in be.calls) == 380


@pytest.mark.gpu
@pytest.mark.parametrize("side,per", [(200, 1), (1600, 2)])
def test_batch_counts_its_launches(pfa, side, per):
    f = ic.grid2d(side, side, seed=side, stripe_width=20, n_particles=2, radius=4.0)
    be = GpuBackend(pfa, pfa.model_params(), pfa.model_params(dim=3), pfa.Batch.footprint(f[0].shape), 0)
    srv = Server(be, tick_steps=50)
    srv.run_trace([Request(0, f, 105)], realtime=False)
    # 50, 50 and 5 steps
    assert srv.step_launches == (105 if per == 1 else 25 + 25 + 3) == be.batch.step_launches()
    be.close()
