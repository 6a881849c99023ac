"""The field shift (with its transposed copy, and as binary16 rows) at the edges of its walker groups, field
steps and X splits, on a force bias that meets the bound, against torch in FP64 (cmf and cfb: sums of X
terms, 1e-12 of their absolute sums; the binary16 head and remainder: 2^-21 of the largest field)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
SDT = 0.005 ** 0.5


def _inputs(W, X):
    rng = np.random.default_rng(W + X)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    return torch.complex(real(W, X), real(W, X)) * 12, real(W, X), torch.complex(real(X), real(X))


def _expected(vb, xi, mf):
    xbar = -SDT * (1j * vb - mf)
    a = xbar.abs()
    xbar = torch.where(a > 1.0, xbar / a, xbar)
    want = xi - xbar
    return want, (-SDT * (want * mf), xi * xbar - 0.5 * xbar * xbar)


def _shift(vb, xi, mf, form, offset=0):
    """(xs (X, W) or None, planes hi, lo (W, 2, ldx) or None, cmf, cfb); form: "rows" (planes alone), "both"
    or "copy".  Planes start ``offset`` halves into their allocations and hold -7 where nothing is written."""
    from ipie_b200._lib import call, ptr, stream

    (W, X), ldx = vb.shape, (vb.shape[1] + 7) // 8 * 8
    c128 = dict(dtype=torch.complex128, device="cuda")
    cmf, cfb, xs = torch.zeros(W, **c128), torch.zeros(W, **c128), torch.zeros(X, W, **c128)
    hi, lo = (torch.full((W * 2 * ldx + 8,), -7.0, dtype=torch.float16, device="cuda")[offset:offset + W * 2 * ldx]
              for _ in range(2))
    if form == "copy":
        call("ipie_b200_field_shift", ptr(vb), ptr(xi), ptr(mf), W, X, SDT, 1.0, ptr(xs), ptr(cmf), ptr(cfb), stream())
        return xs, None, cmf, cfb
    call("ipie_b200_field_shift_mixed", ptr(vb), ptr(xi), ptr(mf), W, X, SDT, 1.0, ptr(xs) if form == "both" else None,
         ptr(hi), ptr(lo), ptr(cmf), ptr(cfb), stream())
    return (xs if form == "both" else None), (hi.reshape(W, 2, ldx), lo.reshape(W, 2, ldx)), cmf, cfb


@pytest.mark.parametrize("W,X", [(1, 1), (8, 64), (9, 65), (64, 120), (640, 600), (33, 129), (3, 2000), (5, 257)])
@pytest.mark.parametrize("form,offset", [("copy", 0), ("both", 0), ("both", 1), ("rows", 0), ("rows", 1), ("rows", 2)])
def test_field_shift(W, X, form, offset):
    vb, xi, mf = _inputs(W, X)
    want, sums = _expected(vb, xi, mf)
    xs, planes, cmf, cfb = _shift(vb, xi, mf, form, offset)
    if xs is not None:
        assert float((xs.T - want).abs().max()) < 1e-14
    if planes is not None:
        hi, lo = planes
        got = (hi.double() + lo.double())[:, :, :X] / 64.0
        assert float((torch.complex(got[:, 0], got[:, 1]) - want).abs().max()) < 2.0 ** -21 * 8
        assert bool((hi[:, :, X:] == -7).all()) and bool((lo[:, :, X:] == -7).all())  # the padding is not written
    for got, ref in ((cmf, sums[0]), (cfb, sums[1])):
        assert float(((got - ref.sum(1)).abs() / ref.abs().sum(1)).max()) < 1e-12


@pytest.mark.parametrize("form", ["copy", "both", "rows"])
def test_nan_stays_in_its_walker(form):
    vb, xi, mf = _inputs(9, 65)
    vb[4, 64] = float("nan")  # NaN + 0i: the imaginary part of xbar, no other
    want, sums = _expected(vb, xi, mf)
    xs, planes, cmf, cfb = _shift(vb, xi, mf, form)
    if xs is not None:
        d = (xs.T - want).abs()
        assert bool(torch.isnan(d[4, 64])) and int(torch.isnan(d).sum()) == 1
    if planes is not None:
        assert torch.isnan(planes[0]).nonzero().tolist() == [[4, 1, 64]]
    for got, ref in ((cmf, sums[0]), (cfb, sums[1])):
        assert torch.isnan(got).nonzero().flatten().tolist() == [4]
        ok = torch.arange(9, device="cuda") != 4
        assert float(((got - ref.sum(1)).abs() / ref.abs().sum(1))[ok].max()) < 1e-12
