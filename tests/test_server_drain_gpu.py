"""drain() returns when every submitted request is done, failed or cancelled, those too
that are with the thread that makes members at that moment."""
import pytest

from acoustics_b200 import scene as S
from acoustics_b200.server import SolveServer
from tests.test_failures_gpu import P32, scenes

pytestmark = pytest.mark.gpu


def test_drain_waits_for_requests_being_made(fdtd_lib):
    reqs = scenes(51, 4, steps_lo=20, steps_hi=40)
    with SolveServer(precision=P32, graph_steps=8, chunk_steps=16) as srv:
        for n in range(1, 41):
            ids = [srv.submit(sc) for sc in reqs]
            if n % 4 == 0:
                try:
                    srv.cancel(ids[-1])
                except Exception:  # finished already
                    pass
            srv.drain(timeout_s=60)
            for i in ids:
                assert srv.poll(i)[0] in (S.REQ_DONE, S.REQ_CANCELLED)
            st = srv.stats()
            assert st["completed"] + st["cancelled"] == 4 * n and st["queued"] == st["running"] == 0
