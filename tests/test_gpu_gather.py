"""GPU: the row forms of the interpolation and of the trajectory gradient against the
planar kernels, over channel counts on both sides of every lane layout (one unit per tap,
several samples per warp, channel pairs, several chunks, a channel per lane), kernel
widths inside and at the compiled ones, sample counts around a warp's and a CTA's turn,
taps across the periodic seam, frames, a subspace basis and B0 segments.

The interpolation is compared on one grid (the INTERP and OUT stages against pfb_interp),
so that the transforms' rounding, which deapodisation amplifies on small grids of wide
kernels, is not part of the comparison; the gradient through pfb_nufft_traj_grad with a
workspace that only the planar path fits and with the full one.

Tolerance: rel-L2 1e-5, as the other comparisons of the two paths (summation order; sums
of at most 8^3 float32 products)."""

import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _both(plan, image, values, basis=None):
    from pyfourier_b200 import _lib
    from pyfourier_b200._nufft import _Ctx, _ptr, _stream

    L = _lib.load()
    ctx = _Ctx(plan, basis, None, 0)
    (seg,) = list(ctx.segments())
    o = ctx.opts(image.shape[0], seg)
    P = int(o.nseg) * image.shape[0] * ctx.C
    small, big = ctypes.c_size_t(), ctypes.c_size_t()
    _lib.check(L.pfb_workspace_size(ctx.interp.handle, P, ctypes.byref(small)))
    _lib.check(L.pfb_apply_workspace_size(ctx.interp.handle, ctypes.byref(o), ctypes.byref(big)))
    assert big.value > small.value
    rel = lambda a, b: float(torch.linalg.norm((a - b).to(torch.complex128)) / torch.linalg.norm(b.to(torch.complex128)))  # noqa: E731
    h, st, M = ctx.interp.handle, _stream(ctx.dev), ctx.interp.total_samples
    # interpolation: a random planar grid, and the same grid with the channels interleaved
    # at the workspace's interleaved region (after the planar one, 256-byte rounded)
    gvol = int(np.prod(plan.os_shape))
    ngrp = 1 if basis is not None else ctx.nframes
    grid = torch.complex(*torch.randn((2, ngrp, P // ngrp, gvol), generator=torch.Generator("cuda").manual_seed(1), device="cuda"))
    ws = torch.empty(big.value, dtype=torch.uint8, device="cuda")
    off = (P * gvol * 8 + 255) // 256 * 256
    ws[off:off + P * gvol * 8].view(torch.complex64).copy_(grid.transpose(1, 2).reshape(-1))
    k0 = torch.full((image.shape[0], M), float("nan"), dtype=torch.complex64, device="cuda")
    k1 = torch.full_like(k0, float("nan"))
    # the planar kernels number the planes (segment, batch, frame or coefficient)
    planes = grid.reshape(P, gvol) if ngrp == 1 else grid.transpose(0, 1).contiguous()
    _lib.check(L.pfb_interp(h, ctypes.byref(o), _ptr(planes), _ptr(k0), 1, st))
    for stage, dst in (("interp", None), ("out", _ptr(k1))):
        _lib.check(L.pfb_nufft_stage(h, ctypes.byref(o), _lib.STAGES[stage], None, dst, ctypes.c_float(1.0), _ptr(ws),
                                     big.value, st))
    assert rel(k1, k0) < 1e-5
    grads = []
    for n in (small.value, big.value):
        g = torch.full((M, ctx.interp.ndim), 0.25, device="cuda")
        o.flags = _lib.PFB_FLAG_ACCUMULATE
        _lib.check(L.pfb_nufft_traj_grad(h, ctypes.byref(o), _ptr(image), _ptr(values), ctypes.c_void_p(g.data_ptr()),
                                         ctypes.c_float(0.5), _ptr(ws), n, st))
        grads.append(g - 0.25)
    assert rel(grads[1], grads[0]) < 1e-5


def _crn(rng, *s):
    return torch.as_tensor((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)).cuda()


def _coord(rng, M, N):
    c = ((rng.random((M, len(N))) - 0.5) * np.array(N[::-1])).astype(np.float32)
    c[: M // 3] *= 0.05  # first taps around the seam of the FFT layout
    return torch.as_tensor(c)


@pytest.mark.parametrize("N, osf", [((70,), 1.25), ((22, 31), 1.5), ((11, 14, 12), 1.25)])
@pytest.mark.parametrize("width", [2, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("B", [1, 2, 3, 5, 8, 9, 16, 17, 33, 64])
def test_channels_and_widths(N, osf, width, B):
    import pyfourier_b200 as P

    rng = np.random.default_rng(B * 10 + width)
    M = 261
    plan = P.plan_nufft(_coord(rng, M, N), N, width=width, oversamp=osf, device="cuda:0")
    _both(plan, _crn(rng, B, 1, *N), _crn(rng, B, M))


@pytest.mark.parametrize("M", [1, 7, 8, 9, 63, 64, 65, 5000])
@pytest.mark.parametrize("B", [1, 4, 32])
def test_sample_counts(M, B):
    import pyfourier_b200 as P

    rng = np.random.default_rng(M)
    N = (18, 20)
    plan = P.plan_nufft(_coord(rng, M, N), N, width=4, oversamp=2.0, device="cuda:0")
    _both(plan, _crn(rng, B, 1, *N), _crn(rng, B, M))


@pytest.mark.parametrize("B, K, L", [(2, 0, 0), (3, 2, 0), (6, 3, 0), (2, 0, 3), (5, 0, 4)])
def test_frames_basis_and_segments(B, K, L):
    import pyfourier_b200 as P

    rng = np.random.default_rng(B + K + L)
    N, F, M = (20, 18), 3, 120
    coord = torch.stack([_coord(rng, M, N).reshape(4, 30, 2) for _ in range(F)])
    kw = {}
    if L:
        kw = dict(zmap=torch.as_tensor(rng.uniform(-100, 100, N).astype(np.float32)), L=L, nbins=20, dt=1e-5)
    plan = P.plan_nufft(coord, N, width=4, oversamp=1.25, device="cuda:0", **kw)
    basis = _crn(rng, F, K).contiguous() if K else None
    _both(plan, _crn(rng, B, K or F, *N), _crn(rng, B, F * M), basis)
