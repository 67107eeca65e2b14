"""zj_adjoint_run under stream capture: it waits for its stream, so it refuses, and
the refusal leaves the capture, the handle's kept block and its results as they were."""
import numpy as np
import pytest

from zhijian_b200 import meshgen as M
from zhijian_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu


def test_adjoint_run_refuses_a_capturing_stream(zjlib):
    import torch
    s = FRSolver(M.tgv_mesh(40, seed=2), make_params(poly_order=3, rho_inf=1.0, p_inf=1 / (1.4 * 0.09), Mach=0.3,
                                                     Re=500.0, compat=False, viscous=True, riemann="Roe",
                                                     bcs=[(1, "slipwall")]))
    s.setInitialCondition(M.taylor_green)
    stream = torch.cuda.Stream()
    s.set_stream(stream.cuda_stream)
    G0 = torch.randn(s.shape, device="cuda", dtype=torch.float64)
    x = torch.zeros(4, device="cuda")

    def run():
        G = G0.clone()
        torch.cuda.synchronize()
        s.adjoint_run(1e-3, 6, 3, G.data_ptr())
        return G.cpu().numpy()

    first = run()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        x += 1.0
        with pytest.raises(RuntimeError, match="capture"):
            s.adjoint_run(1e-3, 6, 3, G0.data_ptr())
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4
    assert np.array_equal(run(), first)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] < 8 << 20       # the block is 40 MB
    s.close()
