"""A handle is destroyed while work of its calls is still waiting on other streams: destroying waits for it, whichever of
the streams it is on, so nothing it reads is freed.  The outputs have the bits of a call on the current stream."""
import numpy as np
import pytest
import torch

from tests.cases import gpu_problem, perturbed_vertices

DELAY = 200_000_000  # SM cycles, about a tenth of a second
N = (9, 8, 7)
CFGS = {
    "general": dict(dim=3, order=1, n=N, kind="diffusion_1pu2", vertex_coords=perturbed_vertices(3, N, (0, 0, 0), (1, 1, 1), 0.2, 5)),
    "box_q2": dict(dim=3, order=2, n=N, kind="thermal", kappa=np.linspace(1.0, 2.0, 504)),
    "nonlinear_q2": dict(dim=3, order=2, n=N, kind="diffusion_1pu2"),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CFGS))
@pytest.mark.parametrize("streams", [3, 20])  # 20: more than the handle keeps marks for at first
def test_destroy_waits_for_every_stream(cuda, name, streams):
    from mrhyde_gb300 import AssemblyManager

    G = gpu_problem(CFGS[name])
    A = AssemblyManager(G)
    u = torch.rand(G.info.n_dofs, dtype=torch.float64, device="cuda")
    want_r, want_J = G.new_vector(), G.new_matrix_values()
    A.assembleJacRes(u, want_r, want_J, overwrite=True)
    out = [(torch.full_like(want_r, 7.0), torch.full_like(want_J, 7.0)) for _ in range(streams)]
    side = [torch.cuda.Stream() for _ in range(streams)]
    torch.cuda.synchronize()
    with torch.cuda.stream(side[0]):
        torch.cuda._sleep(DELAY)
    for s, (r, J) in zip(side, out):
        with torch.cuda.stream(s):
            A.assembleJacRes(u, r, J, overwrite=True)
    A.assembleJacRes(u, want_r, want_J, overwrite=True)
    G.close()
    assert all(s.query() for s in side)
    for r, J in out:
        assert torch.equal(r, want_r) and torch.equal(J, want_J)


@pytest.mark.gpu
def test_destroy_waits_for_an_apply_and_a_new_kappa(cuda):
    from mrhyde_gb300 import SolverManager

    G = gpu_problem(CFGS["box_q2"])
    J = torch.rand(G.info.nnz, dtype=torch.float64, device="cuda")
    x, y, want = torch.rand(G.info.n_dofs, dtype=torch.float64, device="cuda"), G.new_vector(), G.new_vector()
    S = SolverManager(G)
    S.apply(J, x, want)
    side = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    for s in side[:2]:
        with torch.cuda.stream(s):
            torch.cuda._sleep(DELAY)
    with torch.cuda.stream(side[0]):
        S.apply(J, x, y)
    with torch.cuda.stream(side[1]):
        G.set_kappa(torch.ones(G.info.n_cells, dtype=torch.float64, device="cuda"))
    with torch.cuda.stream(side[2]):
        S.apply(J, x, torch.empty_like(y))
    G.close()
    assert all(s.query() for s in side)
    assert torch.equal(y, want)
