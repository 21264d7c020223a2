"""GPU: a Gram whose grid is the image, with a field map of one segment: conj(C) G(C x) on
the fused passes and on the library's transform (1D, 3D, lengths that are primes), against
complex128 torch at test_gpu_gram_rows.py's tolerance."""

import pytest

from test_gpu_gram_rows import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(64,), (97, 97), (12, 194), (96, 128), (16, 30), (8, 9, 10), (53, 10, 53)])
@pytest.mark.parametrize("K, F", [(0, 1), (0, 3), (3, 1), (8, 1)])
def test_one_segment(n, K, F):
    _check(n, n, 3, K=K, F=F, L=1)
