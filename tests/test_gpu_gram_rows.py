"""GPU: the Gram apply on the fused passes (outer axes, then rows with the kernel product
between the two transforms) against complex128 torch, on random kernels: subspace sizes
1 to 8, elementwise planes with and without frames, batch counts around the items of a
CTA, embedded, dense and partly dense grids in 2D and 3D, B0 segments, and grid lengths of
two stages, of radices above 16, of three stages, with a prime factor, and past the fused
lengths (library transform).

Tolerance: 6e-8 log2 n rel-L2 for each of the 2 transforms of at most 3 axes (n <= 440),
2 x 3 x 9 x 6e-8 = 3.2e-6, and the product's rounding: 5e-6."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def _crn(g, *s):
    return torch.complex(torch.randn(s, generator=g, device="cuda"), torch.randn(s, generator=g, device="cuda"))


def _check(n, os, B, K=0, F=1, L=0):
    import pyfourier_b200 as P

    g = torch.Generator("cuda").manual_seed(B + K + sum(n))
    nd, vol = len(n), 1
    for v in os:
        vol *= v
    lead = (L,) if L else ()
    if K:
        value = _crn(g, *lead, vol, K, K)
    else:
        value = _crn(g, *lead, *((F,) if F > 1 else ()), *os)
    zs = _crn(g, L, *n) if L else None
    x = _crn(g, B, *((K or F,) if K or F > 1 else ()), *n)
    gm = P.GramMatrix(value, tuple(os), nd, bool(K), zs, L or None, torch.device("cuda:0"), image_shape=tuple(n))
    got = P.sparse_gram(x, gm)
    ax = tuple(range(-nd, 0))
    off = [max(b // 2 - a // 2, 0) for a, b in zip(n, os)]
    cut = (Ellipsis, *(slice(o, o + a) for o, a in zip(off, n)))
    ref = 0
    for q in range(max(L, 1)):
        t = (value[q] if L else value).to(torch.complex128)
        c = zs[q].to(torch.complex128) if L else 1.0
        e = torch.zeros((*x.shape[: x.ndim - nd], *os), dtype=torch.complex128, device="cuda")
        e[cut] = c * x
        f = torch.fft.fftn(e, dim=ax)
        if K:
            f = torch.einsum("vij,bjv->biv", t, f.reshape(B, K, vol)).reshape(f.shape)
        else:
            f = f * t
        y = torch.fft.ifftn(f, dim=ax)[cut]
        ref = ref + (c.conj() * y if L else y)
    assert float(torch.linalg.norm(got - ref) / torch.linalg.norm(ref)) < 5e-6


@pytest.mark.parametrize("K", [1, 2, 3, 4, 5, 8])
@pytest.mark.parametrize("B", [1, 2, 3, 7])
def test_subspace_sizes(K, B):
    _check((18, 20), (36, 40), B, K=K)
    _check((10, 220), (20, 440), B, K=K)


@pytest.mark.parametrize("B, F", [(1, 1), (5, 1), (17, 1), (33, 1), (2, 3), (9, 2)])
def test_elementwise_planes(B, F):
    _check((21, 17), (42, 34), B, F=F)
    _check((7, 12, 16), (14, 24, 32), B, F=F)


@pytest.mark.parametrize("n", [(31, 37), (29, 31), (97, 20), (12, 194), (20, 178), (10, 41, 12)])
@pytest.mark.parametrize("K, L", [(0, 0), (3, 0), (0, 2)])
def test_dense_grids_with_prime_factors(n, K, L):
    _check(n, n, 3, K=K, L=L)


@pytest.mark.parametrize("n, os", [((16, 30), (16, 30)), ((16, 30), (32, 30)), ((9, 125), (9, 250)), ((1, 40), (1, 80)),
                                   ((62, 31), (124, 62)), ((27, 216), (54, 432)), ((8, 9, 10), (8, 9, 10)),
                                   ((6, 14, 22), (12, 14, 44)), ((10, 11, 53), (20, 22, 106)), ((6, 520), (12, 1040)),
                                   ((64,), (128,))])
@pytest.mark.parametrize("K, L", [(0, 0), (3, 0), (0, 2), (4, 3)])
def test_grids_and_segments(n, os, K, L):
    _check(n, os, 3, K=K, L=L)


# (n, embedded length) of the rows: two stages with constants, alike and unlike, with radices
# to 16 and above, odd, dense and single-point images
@pytest.mark.parametrize("n, os", [(48, 96), (97, 160), (128, 256), (1, 240), (100, 200), (125, 250), (176, 352),
                                   (256, 512), (150, 150), (144, 144)])
@pytest.mark.parametrize("B, F", [(1, 1), (9, 1), (2, 3)])
def test_elementwise_rows_of_two_stages(n, os, B, F):
    _check((5, n), (10, os), B, F=F)
    _check((2, 3, n), (4, 6, os), B, F=F)
