"""Multigrid on meshes of at most 32 nodes, whose hierarchy is the coarsest level alone: the cycle is the dense inverse
applied to the residual.

Reference: the oracle's matrix and residual solved densely on the host.  Bounds as in the other multigrid tests: 1e-9
of the solution's largest value in FP64, 3e-4 with an FP32 matrix."""
import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, oracle_problem

CFGS = [dict(dim=3, order=1, n=(1, 1, 1), dirichlet_faces=1), dict(dim=3, order=1, n=(2, 2, 2), dirichlet_faces=3),
        dict(dim=3, order=1, n=(1, 2, 3), dirichlet_faces=32), dict(dim=2, order=1, n=(3, 3), dirichlet_faces=4)]
IDS = ["x".join(map(str, c["n"])) for c in CFGS]


def _dense(O, vals):
    rp, ci = O.graph()
    M = np.zeros((O.ndof, O.ndof))
    for i in range(O.ndof):
        M[i, ci[rp[i]:rp[i + 1]]] = vals[rp[i]:rp[i + 1]]
    return M


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", CFGS, ids=IDS)
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("krylov", ["cg", "bicgstab"])
@pytest.mark.parametrize("prec", ["gmg", "gmg_split"])
def test_one_level_solve(cuda, cfg, fp32, krylov, prec):
    from mrhyde_gb300 import AssemblyManager, SolverManager

    rng = np.random.default_rng(11)
    c = dict(cfg, source=("const", 1.0, 0.0), kappa=np.exp(0.5 * rng.standard_normal(int(np.prod(cfg["n"])))))
    G, O = gpu_problem(c), oracle_problem(c)
    A, S = AssemblyManager(G), SolverManager(G, preconditioner=prec)
    r, J = G.new_vector(), G.new_matrix_values(fp32=fp32)
    A.assembleJacRes(G.new_vector(), r, J, fp32_jacobian=fp32, overwrite=True)
    ro, Jo = O.assemble(np.zeros(O.ndof))
    xo = np.linalg.solve(_dense(O, Jo), ro)
    tol = 1e-5 if fp32 else 1e-11
    for _ in range(2):  # the second solve runs on buffers that hold the first one's values
        x = G.new_vector()
        res = (S.PCG if krylov == "cg" else S.BiCGStab)(J, r, x, tol=tol, maxiter=50)
        assert res.rel_residual <= tol and res.iterations <= 3, res
        np.testing.assert_allclose(x.cpu().numpy(), xo, rtol=0, atol=(3e-4 if fp32 else 1e-9) * np.abs(xo).max())


@pytest.mark.gpu
@pytest.mark.parametrize("cfg", CFGS, ids=IDS)
@pytest.mark.parametrize("kind", ["thermal", "diffusion_1pu2"])
@pytest.mark.parametrize("mixed", [False, True])
def test_one_level_newton(cuda, cfg, kind, mixed):
    from mrhyde_gb300 import SolverManager

    c = dict(cfg, kind=kind, source=("const", 10.0, 0.0))
    G, O = gpu_problem(c), oracle_problem(c)
    S = SolverManager(G, nonlinear_tol=1e-10, max_nonlinear_iters=20, linear_tol=1e-4 if mixed else 1e-11,
                      mixed_precision=mixed, preconditioner="gmg")
    u = G.new_vector()
    res = S.nonlinearSolver(u)
    assert res.rel_residual < 1e-10
    r0, _ = O.assemble(O.set_dirichlet(np.zeros(O.ndof)), jac=False)
    r, _ = O.assemble(u.cpu().numpy(), jac=False)
    assert np.abs(r).max() <= 1e-9 * np.abs(r0).max()
