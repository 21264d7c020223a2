"""GPU: the adjoint on crowded tiles at the item sizes that the plan picks by the number
of samples (a tile above it is zeroed and split over items combined with atomics).

Sample counts below, at and above one item of the smallest size (128 visits), one sample
more, and many items; channel counts around the zeroing kernel's group of 8; an extent
whose tiles are narrower than the full one.  Tolerance as the other operators' (rel-L2
1e-5 against the oracle: float summation order differs)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import nufft_oracle as orc  # noqa: E402


@pytest.mark.parametrize("shape, width, osf", [((300,), 4, 1.25), ((26, 37), 4, 1.25), ((40, 24), 6, 1.5),
                                               ((11, 12, 14), 4, 2.0)])
@pytest.mark.parametrize("M, B", [(1, 1), (127, 7), (128, 8), (129, 9), (5000, 17), (40001, 3)])
def test_split_tiles_by_sample_count(shape, width, osf, M, B):
    import pyfourier_b200 as P

    rng = np.random.default_rng(M)
    ext = np.asarray(shape[::-1], np.float32)
    # three quarters of the samples within two pixels of the centre, the rest anywhere
    r = np.where(np.arange(M)[:, None] % 4 > 0, 2.0 / ext, 0.49)
    coord = (rng.uniform(-1, 1, (M, len(shape))) * r * ext).astype(np.float32)
    y = (rng.standard_normal((B, M)) + 1j * rng.standard_normal((B, M))).astype(np.complex64)
    op = orc.plan_nufft(coord, shape, width=width, oversamp=osf)
    gp = P.plan_nufft(torch.as_tensor(coord), shape, width=width, oversamp=osf, device="cuda:0")
    got = P.nufft_adj(torch.as_tensor(y).cuda(), nufft_plan=gp).cpu().numpy()
    assert orc.rel_l2(got, orc.nufft_adj(y, op)) < 1e-5
