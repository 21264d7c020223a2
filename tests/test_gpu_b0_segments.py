"""GPU: the B0 segments of an adjoint summed within one call against one segment a call, for
transform lengths on both sides of the tensor-map passes (250, 240 and 256 points take them,
160 and 225 do not), an odd and an even row length and the whole, a part and one of the
segments per call.

Tolerance: the same products are summed in another order and scaled before or after the sum,
at most 6 segments x 2 roundings of 6e-8 each way: 2e-6 rel-L2."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny, osf", [(200, 1.25), (192, 1.25), (128, 2.0), (128, 1.25), (180, 1.25)])
@pytest.mark.parametrize("nx", [18, 21])
def test_segments_in_one_call(ny, osf, nx):
    import pyfourier_b200 as P

    g = torch.Generator("cuda").manual_seed(ny + nx)
    B, views, samples, L = 3, 7, 64, 6
    lim = torch.tensor([nx / 2, ny / 2], device="cuda")
    coord = (torch.rand((views, samples, 2), generator=g, device="cuda") * 2 - 1) * 0.999 * lim
    k = torch.complex(torch.randn((B, views, samples), generator=g, device="cuda"),
                      torch.randn((B, views, samples), generator=g, device="cuda"))
    zmap = torch.rand((ny, nx), generator=g, device="cuda") * 50.0
    T = 1e-5 * np.arange(samples, dtype=np.float32)
    got = [P.nufft_adj(k, coord, (ny, nx), zmap=zmap, L=L, T=T, L_batch_size=s, oversamp=osf) for s in (1, 4, 6)]
    ref = torch.linalg.norm(got[0])
    assert float(ref) > 0
    for y in got[1:]:
        assert float(torch.linalg.norm(y - got[0]) / ref) < 2e-6
