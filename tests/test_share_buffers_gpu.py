"""Device memory of the faces' viscous shares: 4 values a flux point in the
arithmetic type.  Only FP64 handles hold gradient traces (8 values, for the
adjoint); the precision form and the Jacobian-vector product do not.

A Navier-Stokes handle of the precision form differs from the inviscid one by that
buffer alone, 4 bytes times trace_n = (4 E + boundary edges) (P+1) 4 values; the first
Jacobian-vector product allocates two dual-number trace buffers, metrics, three
face and nine state arrays.  cudaMalloc hands out multiples of 2 MiB, so each array
may add up to that; doubled share buffers would be 34 and 134 MB more."""
import numpy as np
import pytest

from zhijian_b200 import meshgen as M
from zhijian_b200.solver import FRSolver, make_params

pytestmark = pytest.mark.gpu
N, P, MIB = 362, 3, 1 << 20
TRACE_N = (4 * N * N + 4 * N) * (P + 1) * 4


def used():
    import torch
    torch.cuda.synchronize()
    free, total = torch.cuda.mem_get_info()
    return total - free


def solver(mesh, viscous, precision):
    return FRSolver(mesh, make_params(poly_order=P, rho_inf=1.0, p_inf=1 / (1.4 * 0.09), Mach=0.3, Re=500.0,
                                      compat=False, viscous=viscous, riemann="Roe", bcs=[(1, "slipwall")],
                                      precision=precision))


def test_precision_form_holds_one_share_buffer(zjlib):
    mesh = M.tgv_mesh(N, seed=3)
    solver(mesh, True, "mixed").close()          # context and modules
    grown = []
    for viscous in (False, True):
        before = used()
        s = solver(mesh, viscous, "mixed")
        grown.append(used() - before)
        s.close()
    assert abs(grown[1] - grown[0] - 4 * TRACE_N) <= 4 * MIB, (grown, 4 * TRACE_N)


def test_jacobian_product_holds_one_share_buffer(zjlib):
    import torch
    mesh = M.tgv_mesh(N, seed=3)
    s = solver(mesh, True, "fp64")
    s.setInitialCondition(M.taylor_green)
    U = torch.from_numpy(s.copyToHost()).cuda()
    V, JV = torch.ones_like(U), torch.empty_like(U)
    w = solver(M.tgv_mesh(5, seed=3), True, "fp64")      # the kernels' module, loaded before the count
    z = torch.ones(w.shape, dtype=torch.float64, device="cuda")
    w.rhs_jvp(z.data_ptr(), z.data_ptr(), torch.empty_like(z).data_ptr())
    before = used()
    s.rhs_jvp(U.data_ptr(), V.data_ptr(), JV.data_ptr())
    grown = used() - before
    sp = N * N * (P + 1) ** 2
    need = 16 * (5 * sp + 2 * TRACE_N) + 8 * (3 * N * N * 4 * (P + 1) * 4 + 9 * sp * 4)
    assert need <= grown <= need + 30 * 2 * MIB, (grown, need)
    w.close()
    s.close()
