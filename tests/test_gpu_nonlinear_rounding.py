"""Rounding of the FP64 matrices of 1 + u^2 on Q1 hexahedra, against extended precision on the host: 2-norm of the error
over that of the matrix, mean over 20 fields, in units of 2^-53.

The sums over pairs of nodes share their terms; done with differences they lost bits where the coefficient changes
strongly over a cell.  Cells of any shape: no further off than the per-cell forward differentiation, which uses
no such sums.  Boxes: at most 5 units, where a contraction row by row measured 4.6, 4.0 and 4.3."""
import numpy as np
import pytest
import torch

LD = np.longdouble
N = (3, 3, 3)
HI = (1.0, 0.7, 0.45)
NODE = np.stack(np.meshgrid(*[np.arange(m + 1) for m in N], indexing="ij")[::-1], -1).reshape(-1, 3)


def _matrix(pts, u):
    """Dense matrix of the mesh, no Dirichlet rows."""
    g = LD(1) / np.sqrt(LD(3))
    M = np.zeros((len(u), len(u)), LD)
    bits = np.array([[v & 1, (v >> 1) & 1, v >> 2] for v in range(8)])
    for c in np.ndindex(*N[::-1]):
        corner = np.array(c[::-1]) + bits
        at = corner @ np.array([1, N[0] + 1, (N[0] + 1) * (N[1] + 1)])
        for q in bits:
            x = np.where(q, g, -g)
            val, der = (1 + np.where(bits, 1, -1) * x) / 2, np.where(bits, LD(0.5), LD(-0.5))
            phi = val.prod(1)
            dphi = np.stack([np.where(np.arange(3) == k, der, val).prod(1) for k in range(3)], 1)
            A = pts[at].T @ dphi
            cof = np.array([[A[(k + 1) % 3, (m + 1) % 3] * A[(k + 2) % 3, (m + 2) % 3]
                             - A[(k + 1) % 3, (m + 2) % 3] * A[(k + 2) % 3, (m + 1) % 3] for m in range(3)] for k in range(3)])
            det = (A[0] * cof[0]).sum()
            grad = dphi @ (cof / det).T
            uq, gu = phi @ u[at], grad.T @ u[at]
            M[np.ix_(at, at)] += abs(det) * ((1 + uq * uq) * (grad @ grad.T) + 2 * uq * np.outer(grad @ gu, phi))
    return M


@pytest.mark.gpu
@pytest.mark.parametrize("mapped", [False, True])
@pytest.mark.parametrize("scale", [0.1, 10.0, 1e4])
def test_matrix_is_as_near_as_the_plain_sums(cuda, mapped, scale):
    from mrhyde_gb300 import AssemblyManager, Problem

    err, plain = [], []
    for seed in range(20):
        rng = np.random.default_rng(seed)
        h = np.array(HI) / np.array(N)
        pts = NODE * h
        if mapped:
            pts = pts + 0.2 * h * rng.uniform(-1, 1, pts.shape)
        u = scale * rng.uniform(-1, 1, len(pts))
        P = Problem(dim=3, order=1, n=N, hi=HI, kind="diffusion_1pu2", dirichlet_faces=0, source=("const", 1.0, 0.0),
                    vertex_coords=pts if mapped else None)
        A, ud = AssemblyManager(P), torch.tensor(u, device="cuda")
        rp, ci = (t.cpu().numpy() for t in P.graph())
        rows = np.repeat(np.arange(len(u)), np.diff(rp))
        x = pts.astype(LD) if mapped else NODE.astype(LD) * np.array(HI).astype(LD) / 3
        want = _matrix(x, u.astype(LD))[rows, ci]
        for out, force in ((err, False), (plain, True)):
            J = P.new_matrix_values()
            A.assembleJac(ud, J, overwrite=True, force_cell=force)
            d = J.cpu().numpy().astype(LD) - want
            out.append(float(np.sqrt((d * d).sum() / (want * want).sum()) * 2.0 ** 53))
    assert np.mean(err) <= (np.mean(plain) if mapped else 5.0), (np.mean(err), np.mean(plain))
