"""A caller's CUDA graph of an asynchronous residual sets the status word at
every replay, so a synchronous residual of a good state clears the word even
when the call before it left it clear: nothing is left for eg_sync to report.
A replay on its own is reported by eg_sync, once."""
import numpy as np
import pytest

from pdesolver_gb300 import abi, eulergpu, problems

pytestmark = pytest.mark.gpu


def _sync(g):
    try:
        g.sync()
    except eulergpu.EulerGPUError as e:
        return e.status
    return abi.EG_OK


@pytest.mark.parametrize("n", [6, 40])   # one launch, two kernels
def test_flags_of_replays(gpu_lib, n):
    import torch
    ms, opts, q = problems.config1(n=n, p=2, family="omega", seed=4)
    g = eulergpu.GPUMesh(ms, opts)
    s = torch.cuda.Stream()
    g.set_stream(s.cuda_stream)
    good = torch.from_numpy(q).cuda()
    x, r = good.clone(), torch.zeros_like(good)
    bad = good.clone()
    bad[0, 0, 0] = -1.0
    torch.cuda.synchronize()
    g.eval_residual(good, r)
    g.eval_residual_async(x, r)
    assert _sync(g) == abi.EG_OK
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        g.eval_residual_async(x, r)

    def replay(state):
        with torch.cuda.stream(s):
            x.copy_(state)
            graph.replay()
        s.synchronize()

    for _ in range(2):
        g.eval_residual(good, r)
        replay(bad)
        g.eval_residual(good, r)
        assert _sync(g) == abi.EG_OK
        g.eval_residual(good, r)
        replay(bad)
        assert _sync(g) == abi.EG_ERR_NEG_DENSITY
        assert _sync(g) == abi.EG_OK
        replay(good)
        assert _sync(g) == abi.EG_OK
    del graph
    g.close()
