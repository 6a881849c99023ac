"""The FP64 real-times-complex products (force bias, VHS and their complex-Cholesky forms) at the edges
of their tiles, copy widths and K splits, against torch in complex128.

Sums of K products in FP64: relative errors stay below K eps of the absolute sums, 1e-12 here."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _data(seed):
    rng = np.random.default_rng(seed)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    return real, lambda *s: torch.complex(real(*s), real(*s))


@pytest.mark.parametrize("W,X,M,na,nb", [(1, 1, 1, 1, 0), (64, 120, 26, 5, 5), (37, 131, 15, 3, 1), (5, 129, 33, 7, 7),
                                         (33, 64, 16, 1, 1), (640, 600, 31, 4, 3), (2048, 33, 9, 2, 2)])
def test_force_bias(W, X, M, na, nb):
    from ipie_b200._lib import call, ptr, stream

    real, cplx = _data(W + X)
    ra, rb, ga, gb = real(X, na * M), real(X, max(nb, 1) * M), cplx(W, na * M), cplx(W, max(nb, 1) * M)
    out = torch.full((W, X), float("nan"), dtype=torch.complex128, device="cuda")
    call("ipie_b200_construct_force_bias_batch_single_det", ptr(ra), ptr(rb), ptr(ga), ptr(gb), W, X, M, na, nb,
         ptr(out), stream())
    want = ga @ ra.T.to(ga.dtype)
    if nb:
        want = want + gb @ rb.T.to(gb.dtype)
    assert _rel(out, want) < 1e-12
    out2 = torch.empty_like(out)  # one tensor for both spins counts twice
    call("ipie_b200_construct_force_bias_batch_single_det", ptr(ra), ptr(ra), ptr(ga), ptr(ga), W, X, M, na, na,
         ptr(out2), stream())
    assert _rel(out2, 2 * (ga @ ra.T.to(ga.dtype))) < 1e-12


@pytest.mark.parametrize("W,X,M", [(1, 1, 1), (64, 120, 26), (37, 131, 15), (640, 100, 40), (9, 17, 65)])
def test_construct_vhs(W, X, M):
    from ipie_b200._lib import call, ptr, stream

    real, cplx = _data(W + X)
    i, j = torch.triu_indices(M, M)
    ii, jj = i.int().cuda(), j.int().cuda()
    L, xs = real(len(i), X), cplx(X, W)
    out = torch.full((W, M, M), float("nan"), dtype=torch.complex128, device="cuda")
    call("ipie_b200_construct_vhs", ptr(L), ptr(ii), ptr(jj), M, X, ptr(xs), W, 0.3, ptr(out),
         stream())
    v = 0.3j * (L.to(xs.dtype) @ xs).T
    want = torch.zeros_like(out)
    want[:, i, j] = v
    want[:, j, i] = v
    assert _rel(out, want) < 1e-12


@pytest.mark.parametrize("W,X,M,N", [(1, 1, 1, 1), (256, 160, 12, 6), (37, 131, 15, 3), (300, 9, 33, 2)])
def test_complex_forms(W, X, M, N):
    from ipie_b200._lib import call, ptr, stream

    real, cplx = _data(W + X)
    r, g = cplx(X, N * M), cplx(W, N * M)
    re, im = r.real.contiguous(), r.imag.contiguous()
    out = cplx(W, X + 3)
    want = out.clone()
    call("ipie_b200_force_bias_complex", ptr(re), ptr(im), ptr(g), W, X, N * M,
         ptr(out), X + 3, 2, 1, stream())
    want[:, 2:2 + X] += g @ r.T
    assert _rel(out, want) < 1e-12
    c, xs = cplx(M * M, X), cplx(X, W)
    re, im = c.real.contiguous(), c.imag.contiguous()
    v = torch.full((W, M, M), float("nan"), dtype=torch.complex128, device="cuda")
    call("ipie_b200_construct_vhs_complex", ptr(re), ptr(im), M, X, ptr(xs), W, 0.3,
         ptr(v), stream())
    assert _rel(v, 0.3j * (c @ xs).T.reshape(W, M, M)) < 1e-12
