"""The FP64 exchange at both of its tile shapes and the edges of their whole-vector, whole-walker tiles,
against torch in complex128 (sums of products in FP64: relative error below (M + N^2 X) eps, 1e-12)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,X,M,N", [(1, 1, 1, 1), (7, 40, 9, 1), (9, 30, 33, 5), (65, 26, 26, 8), (5, 27, 31, 11),
                                     (11, 25, 40, 12), (4, 17, 52, 15), (3, 18, 37, 17), (5, 9, 64, 24),
                                     (3, 9, 65, 25), (2, 5, 70, 32)])
def test_exchange(W, X, M, N):
    from ipie_b200._lib import call, lib, ptr, stream

    rng = np.random.default_rng(N)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    r, g = real(X, N * M), torch.complex(real(W, N, M), real(W, N, M))
    rows = lib().ipie_b200_exchange_rows(W, X, M, N)
    old = 8 if N <= 8 else 16 if N <= 16 else 32
    assert 1 <= rows <= (X + 128 // old - 1) // (128 // old)  # no more than N padded to 8, 16 or 32 takes
    part = torch.full((rows, W), float("nan"), dtype=torch.complex128, device="cuda")
    call("ipie_b200_exchange", ptr(r), ptr(g), W, X, M, N, ptr(part), stream())
    t = torch.einsum("xim,wjm->wxij", r.reshape(X, N, M).to(g.dtype), g)
    want = torch.einsum("wxij,wxji->w", t, t)
    scale = (t.abs() ** 2).sum(dim=(1, 2, 3))
    assert float(((part.sum(0) - want).abs() / scale).max()) < 1e-12
