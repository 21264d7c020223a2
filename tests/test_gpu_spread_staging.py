"""GPU: the register spreads on work items whose batches are full or one or two samples short of
it, so that the last copy round of a batch is partial in every record length (the lanes past
its last piece must copy nothing: a zero-size asynchronous copy still writes its destination,
and once zeroed neighbour entries of the batch, by up to 7e-3 of the adjoint).

An item of a crowded tile takes at most `chunk` visits, here a whole number of batches: 80
(3D, groups of 8 channels), 128 (16), 224 (32), 96 (2D).  Two applies agree to 1e-6 (split
tiles are combined by atomics), the first channel with the float64 adjoint to 2e-5, as
test_gpu_configs.py's."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import nufft_oracle as orc  # noqa: E402


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("N, B, batch", [((32, 32, 32), 5, 80), ((32, 32, 32), 16, 128), ((32, 32, 32), 31, 224),
                                         ((64, 64), 11, 96), ((64, 64), 16, 96), ((64, 64), 33, 96)])
@pytest.mark.parametrize("width, osf", [(4, 1.25), (6, 1.5), (7, 1.5), (8, 2.0)])
def test_partial_copy_rounds(N, B, batch, width, osf):
    import pyfourier_b200 as P

    rng = np.random.default_rng(B + width)
    M = 60000
    # density falling with the radius: tiles of every fullness, the centre ones split
    coord = rng.standard_normal((M, len(N))) * 0.12 * np.array(N[::-1])
    coord = np.clip(coord, -0.49 * N[0], 0.49 * N[0]).astype(np.float32)
    y = (rng.standard_normal((B, M)) + 1j * rng.standard_normal((B, M))).astype(np.complex64)
    plan = P.plan_nufft(torch.as_tensor(coord), N, width=width, oversamp=osf, device="cuda:0")
    oplan = orc.plan_nufft(coord, N, width=width, oversamp=osf)
    x64 = orc.nufft_adj_f64(y[:1].reshape(1, -1), oplan)
    yt = torch.as_tensor(y).cuda()
    for chunk in (batch, 5 * batch, 10 * batch):
        plan.interpolator.set_tuning(chunk=chunk)
        x1 = P.nufft_adj(yt, nufft_plan=plan).cpu().numpy()
        x2 = P.nufft_adj(yt, nufft_plan=plan).cpu().numpy()
        assert _rel(x2, x1) < 1e-6
        assert _rel(x1[0], x64.reshape(x1[0].shape)) < 2e-5
