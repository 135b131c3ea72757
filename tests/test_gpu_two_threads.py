"""Two threads assemble on one handle at a time, each on a stream and with inputs of its own: every call has the bits of
a call alone (the header's contract for mrg_assemble and mrg_spmv)."""
import threading

import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, perturbed_vertices


def _mapped(dim, n):
    return perturbed_vertices(dim, n, (0, 0, 0), (1, 1, 1), 0.2, 3)


CFGS = {
    "thermal_cubes": dict(dim=3, order=1, n=(12, 12, 12), kind="thermal"),
    "thermal_mapped": dict(dim=3, order=1, n=(12, 11, 10), kind="thermal", vertex_coords=_mapped(3, (12, 11, 10))),
    "nonlinear_q1": dict(dim=3, order=1, n=(15, 14, 13), kind="diffusion_1pu2"),
    "general_q1": dict(dim=3, order=1, n=(11, 10, 9), kind="diffusion_1pu2", vertex_coords=_mapped(3, (11, 10, 9))),
    "quad_q1": dict(dim=2, order=1, n=(40, 30), kind="diffusion_1pu2"),
    "quad_q2": dict(dim=2, order=2, n=(40, 30), kind="diffusion_1pu2", vertex_coords=_mapped(2, (40, 30))),
    "box_q2": dict(dim=3, order=2, n=(8, 7, 6), kind="thermal"),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CFGS))
@pytest.mark.parametrize("fp32", [False, True])
def test_two_threads_on_one_handle(cuda, name, fp32):
    from mrhyde_gb300 import AssemblyManager, SolverManager

    G = gpu_problem(CFGS[name])
    A, S = AssemblyManager(G), SolverManager(G)
    rng = np.random.default_rng(17)
    us = [torch.tensor(rng.uniform(0.0, 0.5, G.info.n_dofs), device="cuda") for _ in range(2)]

    def call(u):
        r, J, y = torch.full_like(u, 0.5), torch.full_like(G.new_matrix_values(fp32=fp32), 0.25), torch.empty_like(u)
        A.assembleJacRes(u, r, J, fp32_jacobian=fp32, overwrite=True)
        S.apply(J, u, y)
        return r, J, y

    want = [call(u) for u in us]
    torch.cuda.synchronize()
    got = [[], []]

    def worker(k):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(8):
                got[k].append(call(us[k]))
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=worker, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(2):
        assert len(got[k]) == 8
        for outs in got[k]:
            for a, b in zip(outs, want[k]):
                assert torch.equal(a, b)
