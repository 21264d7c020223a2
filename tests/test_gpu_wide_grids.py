"""GPU: interleaved grids of 2^31 channel values and more, where the gather kernels take 64-bit
offsets (channel pairs, single channels, a channel per lane; interpolation and trajectory
gradient), against the same call in two smaller batches, which take 32-bit ones.

Tolerance: rel-L2 1e-5, as the other comparisons of two forms of the same sums."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N, osf, B", [((64, 64), 16.0, 2049), ((48, 48, 48), 11.0, 15), ((54, 54, 54), 12.0, 16),
                                       ((64, 64, 64), 8.0, 17)])
def test_against_two_batches(N, osf, B):
    import pyfourier_b200 as P
    from pyfourier_b200._nufft import _Ctx, fwd_core, traj_grad_core

    rng = np.random.default_rng(B)
    M = 2000
    coord = ((rng.random((M, len(N))) - 0.5) * np.array(N[::-1])).astype(np.float32)
    coord[: M // 4] *= 0.02  # taps across the periodic seam
    plan = P.plan_nufft(torch.as_tensor(coord), N, width=4, oversamp=osf, device="cuda:0")
    values = int(np.prod([int(s) for s in plan.os_shape])) * B
    assert values >= 2 ** 31
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 2 * values * 8 + (8 << 30):
        pytest.skip("the two grids do not fit the free device memory")
    g = torch.Generator("cuda").manual_seed(B)
    x = torch.complex(*torch.randn((2, B, 1, *N), generator=g, device="cuda"))
    v = torch.complex(*torch.randn((2, B, M), generator=g, device="cuda"))
    ctx = _Ctx(plan, None, None, 0)
    y, t = fwd_core(ctx, x), traj_grad_core(ctx, x, v, 1.0)
    h = B // 2
    yr = torch.cat([fwd_core(ctx, x[:h].contiguous()), fwd_core(ctx, x[h:].contiguous())])
    tr = sum(traj_grad_core(ctx, x[s].contiguous(), v[s].contiguous(), 1.0) for s in (slice(0, h), slice(h, B)))
    rel = lambda a, b: float(torch.linalg.norm(a - b) / torch.linalg.norm(b))  # noqa: E731
    assert rel(y, yr) < 1e-5
    assert rel(t, tr) < 1e-5
    torch.cuda.empty_cache()
