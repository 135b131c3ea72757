"""1+u^2 on Q2 hexahedra, a mesh of several slabs: rows beside the next slab's cells on a second stream give the bits of
the one-stream order that a captured call takes, also when two threads assemble on one problem at a time."""
import threading

import numpy as np
import pytest
import torch

from tests.cases import gpu_problem


@pytest.mark.gpu
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("overwrite", [False, True])
def test_slabs_give_the_bits_of_one_stream(cuda, fp32, overwrite):
    from mrhyde_gb300 import AssemblyManager

    n = (47, 41, 37)
    cfg = dict(dim=3, order=2, n=n, kind="diffusion_1pu2", source=("const", 10.0, 0.0), dirichlet_faces=3)
    G = gpu_problem(cfg)
    A = AssemblyManager(G)
    rng = np.random.default_rng(17)
    us = [torch.tensor(rng.uniform(0.0, 0.3, G.info.n_dofs), device="cuda") for _ in range(2)]

    def outputs():
        return torch.full_like(us[0], 0.5), torch.full_like(G.new_matrix_values(fp32=fp32), 0.25)

    def run(u, r, J):
        A.assembleJacRes(u, r, J, fp32_jacobian=fp32, overwrite=overwrite, tensor_cores=False)

    want = []
    for u in us:
        r, J = outputs()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            run(u, r, J)
        g.replay()
        torch.cuda.synchronize()
        want.append((r, J))
    got = [outputs() for _ in us]
    torch.cuda.synchronize()

    def worker(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            run(us[k], *got[k])
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=worker, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    alone = outputs()
    run(us[0], *alone)
    for (r, J), (rw, Jw) in zip(got + [alone], want + want[:1]):
        assert torch.equal(r, rw)
        assert torch.equal(J, Jw)
