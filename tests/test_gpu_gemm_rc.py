"""The FP64 real-times-complex products (force bias, VHS and their complex-Cholesky forms) at the edges
of their tiles, copy widths and K splits, against torch in complex128.  ``PLAN`` names the (tile, K split) that
a size takes: tiles of 128 x 32, 64 x 32 and 32 x 16 complex entries, splits over 1 to 8 CTAs.

Sums of K products in FP64: relative errors stay below K eps of the absolute sums, 1e-12 here."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _chunks(*k):
    return sum((n + 15) // 16 for n in k)  # of 16 K, per segment


def _plan(M, N, chunks):
    import ctypes

    from ipie_b200._lib import lib

    tile, split = ctypes.c_int(), ctypes.c_int()
    assert lib().ipie_b200_rc_plan_test(M, N, chunks, ctypes.byref(tile), ctypes.byref(split)) == 0
    return tile.value, split.value


def _rel(a, b):
    return float((a - b).norm() / b.norm())


def _data(seed):
    rng = np.random.default_rng(seed)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    return real, lambda *s: torch.complex(real(*s), real(*s))


@pytest.mark.parametrize("W,X,M,na,nb,PLAN", [
    (1, 1, 1, 1, 0, (2, 1)), (64, 120, 26, 5, 5, (2, 8)), (37, 131, 15, 3, 1, (2, 1)), (5, 129, 33, 7, 7, (2, 8)),
    (33, 64, 16, 1, 1, (2, 1)), (640, 600, 31, 4, 3, (2, 1)), (2048, 33, 9, 2, 2, (2, 1)), (260, 257, 27, 5, 5, (2, 2)),
    (333, 65, 27, 5, 5, (2, 4)), (515, 600, 15, 2, 1, (0, 1)), (1030, 200, 400, 4, 0, (0, 2)),
    (515, 200, 60, 8, 7, (0, 4)), (260, 200, 65, 4, 3, (0, 8)), (1030, 200, 45, 1, 0, (1, 1)),
    (700, 600, 91, 3, 2, (1, 2)), (130, 385, 27, 5, 5, (1, 4)), (333, 257, 81, 11, 9, (1, 8))])
def test_force_bias(W, X, M, na, nb, PLAN):
    from ipie_b200._lib import call, ptr, stream

    assert _plan(X, W, _chunks(na * M, nb * M)) == PLAN

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


@pytest.mark.parametrize("W,X,M,PLAN", [
    (1, 1, 1, (2, 1)), (64, 120, 26, (2, 4)), (37, 131, 15, (2, 4)), (640, 100, 40, (0, 1)), (9, 17, 65, (2, 1)),
    (9, 257, 13, (2, 8)), (33, 385, 51, (2, 2)), (101, 600, 31, (0, 8)), (515, 17, 31, (1, 1)), (515, 600, 20, (1, 2)),
    (101, 257, 31, (1, 4))])
def test_construct_vhs(W, X, M, PLAN):
    from ipie_b200._lib import call, ptr, stream

    assert _plan(M * (M + 1) // 2, W, _chunks(X)) == PLAN

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


@pytest.mark.parametrize("W,X,M,N,BIAS,VHS", [
    (1, 1, 1, 1, (2, 1), (2, 1)), (256, 160, 12, 6, (2, 1), (2, 4)), (37, 131, 15, 3, (2, 1), (2, 8)),
    (300, 9, 33, 2, (2, 4), (0, 1)), (130, 385, 13, 7, (1, 4), None), (260, 257, 20, 7, (2, 2), None),
    (9, 17, 20, 7, (2, 8), None), (130, 385, 40, 3, None, (0, 2)), (130, 17, 40, 3, None, (1, 1)),
    (130, 131, 20, 3, None, (1, 4)), (17, 257, 31, 3, None, (1, 8)), (33, 131, 40, 3, None, (2, 2))])
def test_complex_forms(W, X, M, N, BIAS, VHS):
    from ipie_b200._lib import call, ptr, stream

    assert BIAS is None or _plan(X, W, _chunks(N * M, N * M)) == BIAS
    assert VHS is None or _plan(M * M, W, _chunks(X, X)) == VHS

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
