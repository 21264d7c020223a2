"""GPU: tensors whose conjugation or negation torch has only noted (``x.conj()``, and the
gradients that pass through one) give what the same values in memory give: images,
k-space, bases, weights, Gram and gridding inputs, and the gradients of both directions.

Tolerance: rel-L2 1e-6, the order of the adjoint's atomic sums."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N, M, B, F, K = (18, 20), 300, 3, 4, 2


def _crn(seed, *s):
    g = torch.Generator("cuda").manual_seed(seed)
    return torch.complex(*torch.randn((2, *s), generator=g, device="cuda"))


def _same(a, b):
    assert float(torch.linalg.norm(a - b) / torch.linalg.norm(b)) < 1e-6


def _plan(frames=1):
    import pyfourier_b200 as P

    rng = np.random.default_rng(0)
    c = ((rng.random((frames, 10, M // 10, 2)) - 0.5) * np.array(N[::-1])).astype(np.float32)
    c = torch.as_tensor(c if frames > 1 else c[0])
    return P.plan_nufft(c, N, device="cuda:0"), c


def test_nufft_inputs():
    import pyfourier_b200 as P

    plan, _ = _plan()
    x, y = _crn(1, B, *N), _crn(2, B, 10, M // 10)
    z = _crn(3, 10, M // 10)
    w = z.conj().imag  # a negated view
    assert x.conj().is_conj() and w.is_neg()
    _same(P.nufft(x.conj(), nufft_plan=plan, weight=w), P.nufft(x.conj().resolve_conj(), nufft_plan=plan, weight=-z.imag))
    _same(P.nufft_adj(y.conj(), nufft_plan=plan, weight=w),
          P.nufft_adj(y.conj().resolve_conj(), nufft_plan=plan, weight=-z.imag))


def test_single_sample_weight():
    """One weight: its negated view counts as contiguous."""
    import pyfourier_b200 as P

    plan = P.plan_nufft(torch.zeros(1, 1, 2), N, device="cuda:0")
    z, x = _crn(3, 1, 1), _crn(1, B, *N)
    assert z.conj().imag.is_contiguous()
    _same(P.nufft(x, nufft_plan=plan, weight=z.conj().imag), P.nufft(x, nufft_plan=plan, weight=-z.imag))


def test_basis():
    import pyfourier_b200 as P

    plan, _ = _plan(F)
    basis, x, y = _crn(4, F, K).conj(), _crn(5, B, K, *N), _crn(6, B, F, 10, M // 10)
    _same(P.nufft(x, nufft_plan=plan, basis=basis), P.nufft(x, nufft_plan=plan, basis=basis.resolve_conj()))
    _same(P.nufft_adj(y, nufft_plan=plan, basis=basis), P.nufft_adj(y, nufft_plan=plan, basis=basis.resolve_conj()))


def test_gradients():
    import pyfourier_b200 as P

    plan, c = _plan()
    x, y = _crn(1, B, *N), _crn(2, B, 10, M // 10)
    for f, v, t in ((P.nufft, x, y), (P.nufft_adj, y, x)):
        grads = []
        for lazy in (True, False):
            a, k = v.clone().requires_grad_(True), c.cuda().requires_grad_(True)
            r = f(a, coord=k, shape=N, nufft_plan=plan).conj()
            r = r if lazy else r.resolve_conj()
            if lazy:
                r.backward(t)  # the gradient that arrives is t.conj(), noted but not carried out
            else:
                r.backward(t.clone())
            grads.append((a.grad, k.grad))
        a, k = v.clone().requires_grad_(True), c.cuda().requires_grad_(True)
        f(a, coord=k, shape=N, nufft_plan=plan).backward(t.conj().resolve_conj())
        for g in grads:
            _same(g[0], a.grad)
            _same(g[1], k.grad)


def test_gram_and_gridding():
    import pyfourier_b200 as P
    from pyfourier_b200._preinterp import GrogPlan

    _, c = _plan(F)
    gm = P.plan_spgram(c, N, basis=_crn(4, F, K), device="cuda:0")
    x = _crn(5, B, K, *N).conj()
    _same(P.sparse_gram(x, gm), P.sparse_gram(x.resolve_conj(), gm))
    value = _crn(7, *N).conj()
    mk = lambda v: P.GramMatrix(v, N, 2, False, None, None, torch.device("cuda:0"), image_shape=N)  # noqa: E731
    x = _crn(8, B, *N)
    _same(P.sparse_gram(x, mk(value)), P.sparse_gram(x, mk(value.resolve_conj())))
    g = GrogPlan(_crn(9, B, 8, 8), c[0], N, device="cuda:0")
    s = _crn(10, 2, B, M).conj()
    _same(g.apply(s), g.apply(s.resolve_conj()))
