"""A step asked for while the handle's stream is being captured is refused, and
the caller's capture goes on: nothing of the step is in its graph, and the
handle steps as before afterwards."""
import numpy as np
import pytest

from exadglm_b200 import capi
from exadglm_b200 import problem as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("phys,steps_before", [("euler", 0), ("euler", 2), ("advection", 0),
                                               ("advection", 1)])
def test_step_under_capture_is_refused(phys, steps_before):
    torch = pytest.importorskip("torch")
    prob = (P.euler_sine(n=3, N=3, noise=1e-3, seed=1) if phys == "euler"
            else P.advection_gaussian(n=3, N=3, width2=0.05))
    ref = capi.Solver(prob)
    ref.step(steps_before + 1)
    want = ref.get_state()
    ref.close()
    s = capi.Solver(prob)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    s.step(steps_before)
    s.sync()
    x = torch.zeros(8, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin(capture_error_mode="thread_local")
        for ask in (lambda: s.step(1), lambda: s.step(1, dt=1e-3)):
            with pytest.raises(capi.DglmError, match="captured"):
                ask()
        x.add_(1)
        graph.capture_end()
    torch.cuda.synchronize()
    graph.replay()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(x.cpu(), torch.full((8,), 2.0))
    s.step(1)
    assert np.array_equal(s.get_state(), want)
    s.close()
