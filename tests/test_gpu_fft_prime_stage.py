"""GPU: lengths that run a prime stage in the fused passes (every case asserts that the
grid takes them): alone, with a last stage, in the row and in both column layouts, with the
doubled and with the single coefficient table, and in the pruned, B0 and Gram passes.

Tolerances as test_gpu_fft_lengths.py (full transforms against complex128: 10 x 6e-8 for the
stages and sqrt(r) 6e-8 <= 13 x 6e-8 for the r <= 167 terms summed one by one, below 2e-6),
1e-5 against the planar path, test_gpu_gram_rows.py's for the Gram."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from test_fft_route import fused  # noqa: E402


@pytest.mark.parametrize("shape", [(37, 10), (9, 37), (61, 61), (122, 12), (12, 122), (37 * 11, 10), (10, 37 * 13), (488, 6),
                                   (127, 10), (9, 127), (254, 20), (20, 254), (53, 10, 12), (10, 53, 12), (10, 12, 53),
                                   (106, 10, 59), (134, 6, 8), (8, 134, 6), (6, 8, 134), (89, 96, 96), (96, 89, 96),
                                   (96, 96, 89)])
@pytest.mark.parametrize("B", [1, 5, 16])
def test_transform(shape, B):
    from test_gpu_fft_lengths import _check

    assert fused(shape)
    _check(shape, B)


@pytest.mark.parametrize("N", [(111, 64, 64), (64, 111, 64), (87, 64, 64), (64, 92, 64)])
@pytest.mark.parametrize("B, L", [(1, 0), (5, 0), (2, 3)])
def test_large_primes(N, B, L):
    import pyfourier_b200 as P
    import test_gpu_kernels as K

    rng = np.random.default_rng(B + L)
    crn = lambda *s: torch.as_tensor((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()  # noqa: E731
    coord = torch.as_tensor(((rng.random((20, 30, 3)) - 0.5) * np.array(N[::-1])).astype(np.float32))
    kw = {}
    if L:
        kw = dict(zmap=torch.as_tensor(rng.uniform(-100, 100, N).astype(np.float32)), L=L, nbins=20, dt=1e-5)
    plan = P.plan_nufft(coord, N, width=4, oversamp=1.5, device="cuda:0", **kw)
    assert max(plan.os_shape) > 127 and fused(plan.os_shape, N)
    K._pipeline_both(plan, crn(B, 1, *N), crn(B, 600), None, plan.zmap_s_kernel, plan.zmap_t_kernel, max(L, 1))


@pytest.mark.parametrize("n, os", [((16, 53), (32, 106)), ((53, 16), (106, 32)), ((9, 127), (18, 254)), ((6, 7, 37), (12, 14, 74))])
@pytest.mark.parametrize("K, L", [(0, 0), (3, 0), (0, 2)])
def test_gram(n, os, K, L):
    from test_gpu_gram_rows import _check

    assert fused(os, n, gram=True, lowrank=K, nseg=max(L, 1))
    _check(n, os, 3, K=K, L=L)
