"""zj_adjoint_run keeps its checkpoint block on the handle between calls: runs
of changing length and interval (the block grows, is reused at a smaller size,
is reused on another stream) give what a fresh handle gives, bit for bit."""
import numpy as np
import pytest

from zhijian_b200 import meshgen as M
from zhijian_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu


def _solver(mesh, viscous):
    s = FRSolver(mesh, make_params(poly_order=2, rho_inf=1.0, p_inf=1 / (1.4 * 0.09), Mach=0.3, Re=500.0,
                                   compat=False, viscous=viscous, riemann="Roe", bcs=[(1, "slipwall")]))
    s.setInitialCondition(M.taylor_green)
    return s


def _run(s, n, k, seed):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    G = torch.randn(s.shape, generator=g, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    d = s.adjoint_run(1e-3, n, k, G.data_ptr())
    return G.cpu().numpy(), d["dRe"]


@pytest.mark.parametrize("viscous", [True, False])
def test_adjoint_runs_on_one_handle_equal_fresh_handles(zjlib, viscous):
    import torch
    mesh = M.tgv_mesh(9, seed=2)
    kept = _solver(mesh, viscous)
    for i, (n, k) in enumerate([(2, 1), (7, 3), (3, 2), (1, 5), (7, 3)]):
        stream = torch.cuda.Stream()
        if i % 2:
            kept.set_stream(stream.cuda_stream)
        fresh = _solver(mesh, viscous)
        (Ga, ra), (Gb, rb) = _run(kept, n, k, i), _run(fresh, n, k, i)
        assert np.array_equal(Ga, Gb) and ra == rb
        fresh.close()
    kept.close()
