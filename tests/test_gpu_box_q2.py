"""Thermal Q2 on identical affine cells (one thread per row, kappa sums times class coefficients) against the oracle.

FP64: the suite's 1e-12 bound.  FP32 Jacobian: an entry is K32 * S32 with S32 a sum of at most eight positive
rounded kappa by three additions, so at most six roundings of 2^-24 each: 4e-7 of the entry.  Sizes: single
cells, rows of a kind that fill less than, exactly and more than a warp, and more than one CTA of a kind.
"""
import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, oracle_problem
from tests.test_gpu_assembly_parity import TOL64, scaled_err

CASES = [((1, 1, 1), 0, "const"), ((2, 1, 3), 63, "sinprod"), ((33, 2, 2), 3, "const"), ((5, 6, 7), 1 | 8 | 32, "sinprod"),
         ((1, 1), 0, "sinprod"), ((31, 2), 15, "const"), ((13, 20), 1 | 8, "sinprod")]


@pytest.mark.gpu
@pytest.mark.parametrize("n,faces,source", CASES)
@pytest.mark.parametrize("fp32", [False, True])
def test_box_q2_matches_oracle(cuda, n, faces, source, fp32):
    from mrhyde_gb300 import AssemblyManager

    rng = np.random.default_rng(90)
    cfg = dict(dim=len(n), order=2, n=n, lo=(0.0, -1.0, 0.5)[:len(n)], hi=(2.0, 0.5, 1.0)[:len(n)], kind="thermal",
               source=(source, 1.5, 2.0), kappa=np.exp(0.5 * rng.standard_normal(int(np.prod(n)))),
               dirichlet_faces=faces, dirichlet=("const", 0.3))
    O = oracle_problem(cfg)
    u = rng.uniform(-1.0, 1.0, O.ndof)
    ro, Jo = O.assemble(u)
    G = gpu_problem(cfg)
    A = AssemblyManager(G)
    ud = torch.tensor(u, device="cuda")
    r, J = torch.full_like(ud, 7.0), torch.full_like(G.new_matrix_values(fp32=fp32), 3.0)
    A.assembleJacRes(ud, r, J, fp32_jacobian=fp32, overwrite=True)
    assert scaled_err(r.cpu().numpy(), ro) <= TOL64
    assert scaled_err(J.cpu().numpy(), Jo) <= (4e-7 if fp32 else TOL64)
    # the separate calls give the same bits; sum-into adds them, the fixed rows' diagonal stays 1
    r2, J2 = torch.full_like(r, 7.0), torch.full_like(J, 3.0)
    A.assembleRes(ud, r2, overwrite=True)
    A.assembleJac(ud, J2, fp32_jacobian=fp32, overwrite=True)
    assert torch.equal(r2, r) and torch.equal(J2, J)
    A.assembleJacRes(ud, r2, J2, fp32_jacobian=fp32)
    expect = 2 * J
    rp, ci = G.graph()
    row = torch.repeat_interleave(torch.arange(G.info.n_dofs, device="cuda"), rp.diff())
    fixed = torch.zeros(G.info.n_dofs, dtype=torch.bool, device="cuda")
    fixed[G.fixed_dofs()[0].long()] = True
    expect[fixed[row] & (row == ci)] = 1.0
    assert torch.equal(r2, 2 * r) and torch.equal(J2, expect)
