"""GPU: the fused transform over lengths of every kind of stage plan: two stages, three
and more, a radix above 16, primes above 13 (alone, with one and with several other
factors, two of them), the lengths that run on tensor-memory-accelerator tiles, the
longest one taken, and one past it (library transform).

A sparse FFT whose samples are all grid points is the transform itself (no kernel, no
oversampling).  Tolerance: float32 rounding of a length-n transform is about
6e-8 log2 n, and 6e-8 sqrt(r) more for a stage that sums r terms one by one (r <= 251
here): (10 + 16) x 6e-8 < 2e-6 rel-L2 in each direction, against complex128."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 13, 16, 17, 18, 22, 26, 31, 34, 51, 77, 96, 121, 125, 128, 143, 160, 167, 169, 180, 208, 220, 225,
           240, 250, 251, 256, 275, 289, 290, 323, 334, 343, 375, 440, 500, 512, 575, 600, 667, 720, 768, 875, 961,
           1000, 1024, 1025]


def _check(shape, B):
    import pyfourier_b200 as P

    g = torch.Generator("cuda").manual_seed(sum(shape) + B)
    x = torch.complex(*torch.randn((2, B, *shape), generator=g, device="cuda"))
    ax = tuple(range(-len(shape), 0))
    idx = torch.stack(torch.meshgrid(*[torch.arange(n) for n in shape], indexing="ij")[::-1], -1)
    idx = idx.reshape(1, -1, len(shape)).float()
    plan = P.plan_spfft(idx.cuda(), shape, device="cuda:0")
    k = P.sparse_fftn(x, plan=plan).reshape(x.shape)
    ref = torch.fft.fftshift(torch.fft.fftn(torch.fft.ifftshift(x.to(torch.complex128), ax), dim=ax), ax)
    assert float(torch.linalg.norm(k - ref) / torch.linalg.norm(ref)) < 2e-6
    y = P.sparse_ifftn(x.reshape(B, *idx.shape[:-1]), plan=plan)
    ref = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(x.to(torch.complex128), ax), dim=ax), ax)
    assert float(torch.linalg.norm(y - ref) / torch.linalg.norm(ref)) < 2e-6


@pytest.mark.parametrize("shape", [(47, 53, 10), (53, 10, 53), (10, 53, 59), (53, 53, 53), (53, 106, 10)])
def test_several_prime_axes(shape):
    _check(shape, 3)


@pytest.mark.parametrize("n", LENGTHS)
def test_each_axis(n):
    _check((n, 10), 3)
    _check((9, n), 3)


@pytest.mark.parametrize("B", [1, 2, 5, 8, 12, 16, 17, 24, 33])
@pytest.mark.parametrize("shape", [(6, 7, 40), (33, 18, 20), (10, 250, 8), (12, 160, 160)])
def test_3d_channels(shape, B):
    _check(shape, B)


@pytest.mark.parametrize("N, osf", [((13, 17), 2.0), ((57, 88), 1.25), ((100, 45), 1.25), ((200, 30), 1.25),
                                    ((167, 20), 2.0), ((9, 300), 2.0), ((11, 13, 17), 2.0), ((20, 36, 50), 1.25)])
@pytest.mark.parametrize("B, L", [(1, 0), (5, 0), (16, 0), (4, 3)])
def test_pruned_passes_against_the_planar_path(N, osf, B, L):
    """Pad, crop, deapodisation, B0 factors and segment sums of the first and last passes,
    against the library transform with separate pad and crop kernels (rel-L2 1e-5, as the
    other comparisons of the two paths)."""
    import test_gpu_kernels as K
    import pyfourier_b200 as P

    rng = np.random.default_rng(B + L)
    crn = lambda *s: torch.as_tensor((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()  # noqa: E731
    coord = torch.as_tensor(((rng.random((20, 30, len(N))) - 0.5) * np.array(N[::-1])).astype(np.float32))
    kw = {}
    if L:
        kw = dict(zmap=torch.as_tensor(rng.uniform(-100, 100, N).astype(np.float32)), L=L, nbins=20, dt=1e-5)
    plan = P.plan_nufft(coord, N, width=4, oversamp=osf, device="cuda:0", **kw)
    K._pipeline_both(plan, crn(B, 1, *N), crn(B, 600), None, plan.zmap_s_kernel, plan.zmap_t_kernel, max(L, 1))
