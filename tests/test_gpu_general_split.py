"""Cell matrices from stored geometry on both sides of the mesh size (84 cells per SM, 12768 on 152) up to which several threads share
a quadrilateral's matrix, against the oracle.

FP64: the suite's 1e-12 bound.  FP32 Jacobian: 5e-5 on the same scale, the bound of the other tests of this form.
"""
import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, oracle_problem, perturbed_vertices
from tests.test_gpu_assembly_parity import TOL64, scaled_err


@pytest.mark.gpu
@pytest.mark.parametrize("dim,order,kind,n", [
    (2, 1, "diffusion_1pu2", (112, 113)), (2, 1, "diffusion_1pu2", (113, 114)),
    (2, 2, "thermal", (112, 113)), (2, 2, "diffusion_1pu2", (113, 114))])
@pytest.mark.parametrize("fp32", [False, True])
def test_shared_and_whole_cell_matrices_match_oracle(cuda, dim, order, kind, n, fp32):
    from mrhyde_gb300 import AssemblyManager

    rng = np.random.default_rng(91)
    cfg = dict(dim=dim, order=order, n=n, kind=kind, source=("const", 3.0, 0.0), dirichlet_faces=1 | 8,
               kappa=np.exp(0.5 * rng.standard_normal(int(np.prod(n)))),
               vertex_coords=perturbed_vertices(dim, n, (0, 0, 0), (1, 1, 1), 0.25, 92))
    O = oracle_problem(cfg)
    u = rng.uniform(0.0, 0.5, O.ndof)
    ro, Jo = O.assemble(u)
    G = gpu_problem(cfg)
    A = AssemblyManager(G)
    ud = torch.tensor(u, device="cuda")
    r, J = torch.full_like(ud, 7.0), torch.full_like(G.new_matrix_values(fp32=fp32), 3.0)
    A.assembleJacRes(ud, r, J, fp32_jacobian=fp32, overwrite=True)
    assert scaled_err(r.cpu().numpy(), ro) <= TOL64
    assert scaled_err(J.cpu().numpy(), Jo) <= (5e-5 if fp32 else TOL64)
    r2, J2 = torch.full_like(r, 7.0), torch.full_like(J, 3.0)
    A.assembleRes(ud, r2, overwrite=True)
    A.assembleJac(ud, J2, fp32_jacobian=fp32, overwrite=True)
    assert scaled_err(r2.cpu().numpy(), ro) <= TOL64
    assert scaled_err(J2.cpu().numpy(), Jo) <= (5e-5 if fp32 else TOL64)
