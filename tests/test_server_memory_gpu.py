"""The device memory a finished request gives back is held by the requests admitted on it
before the result is out: a client that answers a result by allocating at once takes
neither their memory nor (here, where it can be told apart) their allocation."""
import ctypes as C

import numpy as np
import pytest

from acoustics_b200 import scene as S
from acoustics_b200._lib import FDTDError, load
from acoustics_b200.scene import Options
from acoustics_b200.server import SolveServer
from tests.test_failures_gpu import INJ_DEVICE, INJ_NONE, OOM, P32, _wait_running, scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def disarm():
    yield
    load().fdtd_debug_inject_failure(INJ_NONE, 0)


def test_the_next_admission_allocates_before_the_client(fdtd_lib):
    L = load()
    first, second = scenes(41, 2, steps_lo=400, steps_hi=400)
    desc, keep = scenes(42, 1)[0].to_c()
    opt = Options(precision=P32, kernel=S.KERNEL_FUSED)
    with SolveServer(precision=P32, graph_steps=8, chunk_steps=16, max_members=1) as srv:
        for _ in range(25):
            a = srv.submit(first)
            _wait_running(srv, a)
            L.fdtd_debug_inject_failure(INJ_DEVICE, 0)  # the next device allocation fails: the second request's
            b = srv.submit(second)
            h = C.c_void_p()
            srv.wait(a)
            assert L.fdtd_solver_create(C.byref(desc), C.byref(opt), C.byref(h)) == 0
            L.fdtd_solver_destroy(h)
            with pytest.raises(FDTDError) as e:
                srv.result(b)
            assert e.value.status == OOM
            assert np.isfinite(srv.result(a)[0]).all()
        del keep
        # requests behind a finished one still run, and drain waits for results that are still to come out
        ids = [srv.submit(sc) for sc in (second, first, second)]
        ys = [srv.result(i)[0] for i in ids]
        assert np.array_equal(ys[0], ys[2])
        srv.submit(second)
        st = srv.stats()
        assert st["failed"] == 25 and st["device_bytes_in_use"] >= 0
