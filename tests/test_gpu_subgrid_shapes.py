"""The batched subgrid solver at the shapes where its column mapping changes: one interior node, one column, one
plane, columns cut into segments, the largest problem (15 x 15 columns of 15 rows), for each thread count.

Bound on the solution: the refinement stops at a relative residual of 1e-10 in the inf-norm, so 1e-9 of the largest
value, as in the other subgrid test; the FP32 Jacobian within the suite's 2e-6."""
import numpy as np
import pytest

from tests.cases import oracle_problem
from tests.test_gpu_assembly_parity import TOL32, scaled_err

SIZES = [(2, 2, 2), (16, 16, 16), (16, 2, 3), (2, 16, 16), (3, 2, 16), (16, 15, 2), (9, 16, 16), (4, 5, 16)]


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512, 1024])
def test_batch_shapes(cuda, threads):
    from mrhyde_gb300.subgrid import SubgridBatch

    rng = np.random.default_rng(33)
    sizes = np.array(SIZES)
    kaps = [np.exp(rng.standard_normal(int(np.prod(s)))) for s in sizes]
    dbcs = [rng.uniform(-1.0, 1.0, int(np.prod(s + 1))) for s in sizes]
    B = SubgridBatch(sizes, kaps, dbcs, source=2.0)
    B.set_config(threads, 1)
    B.u.fill_(7.0)
    B.J.fill_(7.0)
    st = B.solve()
    assert np.all(st[:, 3] == 0) and np.all(st[:, 2] <= 1e-10)
    for k, s in enumerate(SIZES):
        cfg = dict(dim=3, order=1, n=s, kappa=kaps[k], source=("const", 2.0, 0.0), dirichlet_faces=63,
                   dirichlet=("node", dbcs[k]))
        O = oracle_problem(cfg)
        uo, rc, _ = O.newton(O.set_dirichlet(np.zeros(O.ndof)), nltol=1e-12, maxiter=4, lintol=1e-14)
        assert np.abs(B.solution(k).cpu().numpy() - uo).max() <= 1e-9 * np.abs(uo).max(), s
        _, Jo = O.assemble(uo)
        o = int(B.nnz_off[k])
        assert scaled_err(B.J[o:o + O.nnz].cpu().numpy(), Jo) <= TOL32, s
