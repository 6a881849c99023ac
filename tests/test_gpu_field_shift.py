"""The field shift (with its transposed copy, and as binary16 rows) at the edges of its walker groups, field
steps and X splits, on a force bias that meets the bound, against torch in FP64 (cmf and cfb: sums of X
terms, 1e-12 of their absolute sums; the binary16 head and remainder: 2^-21 of the largest field)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,X", [(1, 1), (8, 64), (9, 65), (64, 120), (640, 600), (33, 129), (3, 2000)])
@pytest.mark.parametrize("mixed", [False, True])
def test_field_shift(W, X, mixed):
    from ipie_b200._lib import call, ptr, stream

    rng = np.random.default_rng(W + X)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    vb, xi, mf = torch.complex(real(W, X), real(W, X)) * 12, real(W, X), torch.complex(real(X), real(X))
    vb[0, 0] = float("nan")  # stays where it is
    sdt, c128 = 0.005 ** 0.5, dict(dtype=torch.complex128, device="cuda")
    cmf, cfb, xs = torch.zeros(W, **c128), torch.zeros(W, **c128), torch.zeros(X, W, **c128)
    xbar = -sdt * (1j * vb - mf)
    a = xbar.abs()
    xbar = torch.where(a > 1.0, xbar / a, xbar)
    want = xi - xbar
    if mixed:
        ldx = (X + 7) // 8 * 8
        hi, lo = (torch.zeros(W, 2, ldx, dtype=torch.float16, device="cuda") for _ in range(2))
        call("ipie_b200_field_shift_mixed", ptr(vb), ptr(xi), ptr(mf), W, X, sdt, 1.0, ptr(xs) if X % 2 else None,
             ptr(hi), ptr(lo), ptr(cmf), ptr(cfb), stream())
        got = (hi.double() + lo.double())[:, :, :X] / 64.0
        got = torch.complex(got[:, 0], got[:, 1])
        assert float((got - want).abs()[1:].max() if W > 1 else 0.0) < 2.0 ** -21 * 8
    if not mixed or X % 2:
        if not mixed:
            call("ipie_b200_field_shift", ptr(vb), ptr(xi), ptr(mf), W, X, sdt, 1.0, ptr(xs), ptr(cmf), ptr(cfb),
                 stream())
        d = (xs.T - want).abs()
        assert bool(torch.isnan(d[0, 0])) and int(torch.isnan(d).sum()) == 1
        assert float(torch.nan_to_num(d).max()) < 1e-14
    assert bool(torch.isnan(cmf[0])) and bool(torch.isnan(cfb[0]))
    for got, ref in ((cmf, -sdt * (want * mf)), (cfb, xi * xbar - 0.5 * xbar * xbar)):
        err = (got - ref.sum(1)).abs() / ref.abs().sum(1)
        assert W == 1 or float(err[1:].max()) < 1e-12
