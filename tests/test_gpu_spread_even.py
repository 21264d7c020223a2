"""GPU: which plans split tiles over work items combined with atomics (their adjoint launches
the zeroing pass): those with a crowded tile, and those whose tiles are all fuller than twice
an item; evenly filled tiles up to that stay whole."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, M, width, crowded, split", [
    ((48, 48, 48), 51200, 4, False, False), ((48, 48, 48), 51200, 6, False, False), ((48, 48, 48), 51200, 4, True, True),
    ((48, 48, 48), 400000, 6, False, True), ((128, 128), 8000, 4, False, False), ((128, 128), 8000, 4, True, True),
    ((128, 128), 25600, 4, False, True)])
def test_split_tiles(N, M, width, crowded, split):
    import pyfourier_b200 as P
    from torch.profiler import ProfilerActivity, profile

    rng = np.random.default_rng(M)
    coord = rng.uniform(-0.49, 0.49, (M, len(N))) * np.array(N[::-1])
    if crowded:
        coord[: M // 2] *= 0.02
    plan = P.plan_nufft(torch.as_tensor(coord.astype(np.float32)), N, width=width, oversamp=1.25, device="cuda:0")
    y = torch.ones((3, M), dtype=torch.complex64, device="cuda")
    P.nufft_adj(y, nufft_plan=plan)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        P.nufft_adj(y, nufft_plan=plan)
        torch.cuda.synchronize()
    names = [e.name for e in prof.events()]
    assert any("spread" in n for n in names)
    assert any("zero_tiles" in n for n in names) == split
