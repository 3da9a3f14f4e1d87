"""A request that arrives at an idle server is admitted at once, also when the
Krylov solves of concurrent requests share launches: the clock of this server
stands still, so a request held back for any time would never start."""
import threading

import numpy as np
import pytest

from pdesolver_gb300 import eulergpu, serve


@pytest.mark.parametrize("slots", [1, 4])
@pytest.mark.parametrize("batch_gmres", [False, True])
def test_a_lone_request_is_admitted_at_once(monkeypatch, slots, batch_gmres):
    started = threading.Event()

    class Server(serve.SteadySolveServer):
        def _gpu_run_request(self, req, meshes, stream, res):
            started.set()

        _gpu_make_meshes = staticmethod(lambda req: [])
        _gpu_close_meshes = staticmethod(lambda meshes: None)
        _gpu_make_stream = staticmethod(lambda: None)

    monkeypatch.setattr(eulergpu, "set_gmres_batching", lambda enable=True, window_us=50.0: None)
    srv = Server(100, slots=slots, batch_gmres=batch_gmres, clock=lambda: 0.0)
    srv.start()
    srv.submit(serve.SolveRequest(rid=0, levels=[], q0=np.zeros(1), opts={}, footprint=1))
    at_once = started.wait(5.0)
    srv.finish()
    assert at_once
