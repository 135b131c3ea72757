"""The serving loop's estimate of a request's device memory counts the workspace of its assembly calls."""
import pytest

from mrhyde_gb300 import _lib as L
from mrhyde_gb300 import serving


def _workspace(n, mixed):
    nonlinear, thermal = (serving.estimate_bytes(serving.Request(0, k, n, 1, mixed)) for k in ("nonlinear", "thermal"))
    return nonlinear - thermal


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("n", [16, 45, 96, 300])
def test_nonlinear_requests_count_their_workspace(n, mixed):
    want = min(n ** 3 * 54 * (4 if mixed else 8), 4 << 30)
    assert want <= _workspace(n, mixed) <= want + 64 * 54 * 8


@pytest.mark.gpu
@pytest.mark.parametrize("mixed", [False, True])
def test_the_estimate_covers_what_a_request_takes(cuda, tmp_path, monkeypatch, mixed):
    import torch

    from tests.fakecuda import Fake, library

    lib = library(str(tmp_path))
    monkeypatch.setattr(L, "_lib", lib)
    serving.solve_request(serving.Request(0, "nonlinear", 21, 3, mixed), torch.cuda.Stream())
    taken = Fake(lib).pool_largest.value
    assert 0 < taken <= _workspace(21, mixed)
