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


@pytest.mark.parametrize("W,X,M", [(31, 150, 20), (64, 120, 26), (256, 60, 20)])
def test_few_electrons_cost_no_more_than_eight(W, X, M):
    """One to five electrons are 1/64 to 1/3 of the work of eight on the same walkers and vectors, however the
    packed tiles divide it.  A factor of two is left for launch overhead and for fewer, fuller tiles."""
    from ipie_b200._lib import call, lib, ptr, stream

    def us(N):
        r, g = (torch.rand(n, dtype=torch.float64, device="cuda") for n in (X * N * M, 2 * W * N * M))
        part = torch.empty(lib().ipie_b200_exchange_rows(W, X, M, N) * W * 2, dtype=torch.float64, device="cuda")
        best = float("inf")
        for _ in range(8):
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            ev[0].record()
            for _ in range(20):
                call("ipie_b200_exchange", ptr(r), ptr(g), W, X, M, N, ptr(part), stream())
            ev[1].record()
            torch.cuda.synchronize()
            best = min(best, ev[0].elapsed_time(ev[1]) * 50.0)
        return best

    eight = us(8)
    for N in (1, 2, 3, 5):
        assert us(N) < 2.0 * eight, N
