"""Launches that the CUDA runtime refuses (a fake of the call returns the error) end the solve with an error, whichever
launch of the multigrid iteration it is, and leave nothing behind: the next solve on the handle gives the same bits as
one without the refusal."""
import pytest
import torch

from mrhyde_gb300 import _lib as L
from tests.fakecuda import Fake, library


@pytest.fixture(scope="module")
def fake_lib(cuda, tmp_path_factory):
    return library(str(tmp_path_factory.mktemp("fake")))


@pytest.mark.gpu
@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("krylov", ["cg", "bicgstab"])
def test_refused_launch_is_reported(fake_lib, monkeypatch, fp32, krylov):
    from mrhyde_gb300 import AssemblyManager, Problem, SolverManager

    monkeypatch.setattr(L, "_lib", fake_lib)
    fake = Fake(fake_lib)

    def handle():
        P = Problem(dim=3, order=1, n=(14, 13, 12), dirichlet_faces=3)
        r, J = P.new_vector(), P.new_matrix_values(fp32=fp32)
        AssemblyManager(P).assembleJacRes(P.new_vector(), r, J, fp32_jacobian=fp32, overwrite=True)
        return P, SolverManager(P, preconditioner="gmg"), r, J

    def solve(P, S, r, J):
        x = P.new_vector()
        (S.PCG if krylov == "cg" else S.BiCGStab)(J, r, x, tol=1e-5 if fp32 else 1e-10, maxiter=50)
        return x

    P, S, r, J = handle()
    fake.launches.value, fake.launch_at.value = 0, 0
    want = solve(P, S, r, J)
    count = fake.launches.value
    assert count >= 20
    P.close()
    for at in range(1, count + 1):
        P, S, r, J = handle()
        fake.launches.value, fake.launch_at.value = 0, at
        with pytest.raises(L.MrgError) as e:
            solve(P, S, r, J)
        assert e.value.status == L.MRG_ECUDA
        fake.launch_at.value = 0
        assert torch.equal(solve(P, S, r, J), want)
        P.close()
