"""1 + u^2 on Q1 hexahedra (54 numbers a cell, gathered row by row) against the oracle, at cell counts that fill less
than, exactly and more than a workspace block and a CTA.

FP64: the suite's 1e-12 bound.  FP32 Jacobian: 5e-5 on the same scale, the bound of the other tests of this form
(at most 8 * 8 * 4 products an entry, whose terms cancel down to the scale's floor).
"""
import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, oracle_problem
from tests.test_gpu_assembly_parity import TOL64, scaled_err


@pytest.mark.gpu
@pytest.mark.parametrize("n,faces", [((1, 1, 1), 0), ((1, 2, 16), 3), ((33, 5, 4), 1 | 8 | 32), ((8, 4, 4), 63), ((2, 130, 1), 0)])
@pytest.mark.parametrize("fp32", [False, True])
def test_nonlinear_q1_matches_oracle(cuda, n, faces, fp32):
    from mrhyde_gb300 import AssemblyManager

    cfg = dict(dim=3, order=1, n=n, kind="diffusion_1pu2", source=("const", 10.0, 0.0), dirichlet_faces=faces,
               lo=(0.0, -0.5, 0.0), hi=(1.0, 0.5, 2.0))
    O = oracle_problem(cfg)
    u = np.random.default_rng(61).uniform(-0.5, 0.5, O.ndof)
    ro, Jo = O.assemble(u)
    G = gpu_problem(cfg)
    A = AssemblyManager(G)
    ud = torch.tensor(u, device="cuda")
    r, J = torch.full_like(ud, 7.0), torch.full_like(G.new_matrix_values(fp32=fp32), 3.0)
    A.assembleJacRes(ud, r, J, fp32_jacobian=fp32, overwrite=True)
    assert scaled_err(r.cpu().numpy(), ro) <= TOL64
    assert scaled_err(J.cpu().numpy(), Jo) <= (5e-5 if fp32 else TOL64)
    # the residual alone has the same bits; so does the FP64 Jacobian alone (the FP32 one forms its
    # fields in FP32 when no residual is asked for)
    r2, J2 = torch.full_like(r, 7.0), torch.full_like(J, 3.0)
    A.assembleRes(ud, r2, overwrite=True)
    A.assembleJac(ud, J2, fp32_jacobian=fp32, overwrite=True)
    assert torch.equal(r2, r)
    if fp32:
        assert scaled_err(J2.cpu().numpy(), Jo) <= 5e-5
    else:
        assert torch.equal(J2, J)
    # sum-into: the residual adds cell by cell in the same order from r; the fixed rows' diagonal stays 1
    r3, J3 = r.clone(), J.clone()
    A.assembleJacRes(ud, r3, J3, fp32_jacobian=fp32)
    r4 = r.clone()
    A.assembleRes(ud, r4)
    assert torch.equal(r3, r4)
    assert scaled_err(r3.cpu().numpy(), 2 * ro) <= TOL64
    expect = 2 * J
    rp, ci = G.graph()
    row = torch.repeat_interleave(torch.arange(G.info.n_dofs, device="cuda"), rp.diff())
    fixed = torch.zeros(G.info.n_dofs, dtype=torch.bool, device="cuda")
    fixed[G.fixed_dofs()[0].long()] = True
    expect[fixed[row] & (row == ci)] = 1.0
    assert torch.equal(J3, expect)
