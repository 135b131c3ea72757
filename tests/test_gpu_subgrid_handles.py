"""Two subgrid batches of unlike sizes alive at a time: making the second must not take from the first the shared
memory that its problems need.  The solution has the bits of the batch solved before the other one existed."""
import numpy as np
import pytest
import torch


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [256, 512, 1024])
def test_a_second_batch_leaves_the_first_its_shared_memory(cuda, threads):
    from mrhyde_gb300.subgrid import SubgridBatch

    def batch(n, seed):
        rng = np.random.default_rng(seed)
        B = SubgridBatch([(n, n, n)] * 2, [np.exp(rng.standard_normal(n ** 3)) for _ in range(2)],
                         [rng.uniform(-1.0, 1.0, (n + 1) ** 3) for _ in range(2)], source=1.0)
        B.set_config(threads, 1)
        return B

    first = batch(16, 1)
    first.solve()
    want = first.u.clone()
    first = batch(16, 1)
    second = batch(4, 2)
    first.u.fill_(7.0)
    assert np.all(first.solve()[:, 3] == 0)
    assert torch.equal(first.u, want)
    assert np.all(second.solve()[:, 3] == 0)
