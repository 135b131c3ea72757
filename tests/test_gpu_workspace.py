"""Assembly with less memory for its workspace than it asks for (a fake of the allocating call says so): in ever smaller
pieces of cell layers with the bits of one piece, and in the end, with no workspace at all, by the per-cell kernels."""
import numpy as np
import pytest
import torch

from mrhyde_gb300 import _lib as L
from tests.cases import gpu_problem, perturbed_vertices
from tests.fakecuda import Fake, library


@pytest.fixture(scope="module")
def fake_lib(cuda, tmp_path_factory):
    return library(str(tmp_path_factory.mktemp("fake")))


def _mapped(n):
    return perturbed_vertices(len(n), n, (0, 0, 0), (1, 1, 1), 0.2, 3)


def _cfg(dim, order, n, kind, mapped):
    c = dict(dim=dim, order=order, n=n, kind=kind, source=("const", 3.0, 0.0), dirichlet_faces=1 | 8,
             hi=(1.0, 0.7, 0.45)[:dim])
    if kind == "thermal":
        c["kappa"] = np.exp(0.5 * np.random.default_rng(4).standard_normal(int(np.prod(n))))
    if mapped:
        c["vertex_coords"] = _mapped(n)
    return c


CFGS = {
    "nonlinear_q1": _cfg(3, 1, (7, 5, 13), "diffusion_1pu2", False),
    "nonlinear_q1_flat": _cfg(3, 1, (40, 9, 1), "diffusion_1pu2", False),
    "general_q1": _cfg(3, 1, (9, 4, 8), "diffusion_1pu2", True),
    "quad_q1": _cfg(2, 1, (23, 17), "diffusion_1pu2", True),
    "quad_q2": _cfg(2, 2, (150, 101), "diffusion_1pu2", True),
    "quad_q2_thermal": _cfg(2, 2, (19, 15), "thermal", True),
    "nonlinear_q2": _cfg(3, 2, (5, 7, 9), "diffusion_1pu2", False),
    "nonlinear_q2_slabs": _cfg(3, 2, (43, 41, 40), "diffusion_1pu2", False),
}


@pytest.mark.gpu
@pytest.mark.parametrize("name", list(CFGS))
@pytest.mark.parametrize("call,fp32", [("jacres", False), ("jacres", True), ("jac", False), ("jac", True), ("res", False)])
@pytest.mark.parametrize("overwrite", [False, True])
def test_pieces_give_the_bits_of_the_whole(fake_lib, monkeypatch, name, call, fp32, overwrite):
    from mrhyde_gb300 import AssemblyManager

    monkeypatch.setattr(L, "_lib", fake_lib)
    fake = Fake(fake_lib)
    fake.pool_most.value = 2 ** 60
    G = gpu_problem(CFGS[name])
    A = AssemblyManager(G)
    u = torch.tensor(np.random.default_rng(8).uniform(0.0, 0.5, G.info.n_dofs), device="cuda")

    def run(**kw):
        r, J = torch.full_like(u, 0.5), torch.full_like(G.new_matrix_values(fp32=fp32), 0.25)
        if call == "jacres":
            A.assembleJacRes(u, r, J, fp32_jacobian=fp32, overwrite=overwrite, **kw)
        elif call == "jac":
            A.assembleJac(u, J, fp32_jacobian=fp32, overwrite=overwrite, **kw)
        else:
            A.assembleRes(u, r, overwrite=overwrite, **kw)
        return r, J

    fake.pool_largest.value = 0
    want = run()
    whole, sizes = fake.pool_largest.value, []
    assert whole > 0
    while True:
        fake.pool_most.value = (sizes[-1] if sizes else whole) - 1
        fake.pool_taken.value = fake.pool_largest.value = 0
        got = run()
        if not fake.pool_taken.value:
            break
        sizes.append(fake.pool_largest.value)
        for a, b in zip(got, want):
            assert torch.equal(a, b), sizes
    layers = CFGS[name]["n"][-1]
    assert len(sizes) >= (2 if layers > 3 else 0)
    # no memory at all: what the per-cell kernels give
    for a, b in zip(got, run(force_cell=True)):
        assert torch.equal(a, b)
    fake.pool_most.value = 2 ** 60
    for a, b in zip(run(), want):  # and the next call has its workspace again
        assert torch.equal(a, b)
    G.close()


@pytest.mark.gpu
def test_idle_workspace_is_given_back(cuda):
    """Calls overlapping on six streams take six workspaces; a synchronisation leaves the handle's own request and 1 GiB."""
    from mrhyde_gb300 import AssemblyManager, Problem

    G = Problem(dim=3, order=1, n=(120, 120, 120), kind="diffusion_1pu2")
    need = 120 ** 3 * (54 + 8) * 8  # 857 MB
    A = AssemblyManager(G)
    u = G.new_vector()
    out = [(G.new_vector(), G.new_matrix_values()) for _ in range(6)]
    side = [torch.cuda.Stream() for _ in out]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for s, (r, J) in zip(side, out):
        with torch.cuda.stream(s):
            torch.cuda._sleep(50_000_000)
            A.assembleJacRes(u, r, J, overwrite=True)
    torch.cuda.synchronize()
    assert free - torch.cuda.mem_get_info()[0] <= need + 2 ** 30 + 2 ** 27  # and what mapping rounds up
    for r, J in out[1:]:
        assert torch.equal(J, out[0][1]) and torch.equal(r, out[0][0])
    G.close()
