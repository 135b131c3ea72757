"""y = J x on Q1 graphs against 64-bit sums on the host: |y - y_ref| <= 27 * 2^-53 * sum |J x| (at most 27 terms a row).
FP32 values are widened on the integer pipes: zeros, subnormals and the largest and smallest normal values are among
them; rows with an infinite value or a NaN give what the host gives.  Sizes: tiles of 32 rows with whole, cut and
single rows, one and several planes."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("n", [(1, 1, 1), (2, 1, 3), (9, 5, 4), (40, 3, 2), (31, 7, 1), (1, 1), (17, 9), (100, 3)])
@pytest.mark.parametrize("fp32", [False, True])
def test_q1_apply(cuda, n, fp32):
    from mrhyde_gb300 import Problem, SolverManager

    P = Problem(dim=len(n), order=1, n=n)
    rng = np.random.default_rng(7)
    J = rng.standard_normal(P.info.nnz)
    J[rng.integers(0, J.size, J.size // 4)] = 0.0
    J[::17] = -0.0
    if fp32:
        J = J.astype(np.float32)
        J[::7] = np.float32(1e-42)
        J[3::11] = np.finfo(np.float32).tiny
        J[5::13] = -np.finfo(np.float32).max
    J[J.size // 2] = np.inf
    J[J.size // 3] = np.nan
    x = rng.standard_normal(P.info.n_dofs)
    y = torch.full((P.info.n_dofs,), 7.0, dtype=torch.float64, device="cuda")
    SolverManager(P).apply(torch.tensor(J, device="cuda"), torch.tensor(x, device="cuda"), y)
    rp, ci = (a.cpu().numpy() for a in P.graph())
    terms = J.astype(np.float64) * x[ci]
    ref, size = np.add.reduceat(terms, rp[:-1]), np.add.reduceat(np.abs(terms), rp[:-1])
    y, fin = y.cpu().numpy(), np.isfinite(size)
    assert np.array_equal(np.isfinite(y), fin) and np.array_equal(np.isnan(y), np.isnan(ref))
    assert np.all(np.abs(y[fin] - ref[fin]) <= 27 * 2.0 ** -53 * size[fin])
