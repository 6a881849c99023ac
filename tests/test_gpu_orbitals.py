"""The fused FP64 orbital update (one-body, exp(VHS), one-body) in both kernels (operands resident up to
M = 80, streamed above) at the edges of their tiles, ring depths and register classes, against torch in
complex128 (seven chained products of M terms: 1e-12 relative)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,W,pre,post,nmax", [(1, 1, 3, 1, 1, 6), (26, 5, 64, 1, 1, 6), (7, 3, 2, 0, 1, 1),
                                                 (64, 17, 3, 0, 0, 6), (80, 32, 2, 1, 0, 3), (81, 8, 3, 1, 1, 6),
                                                 (108, 15, 5, 1, 1, 6), (128, 32, 2, 0, 0, 2), (129, 24, 2, 1, 1, 6),
                                                 (160, 26, 3, 1, 1, 6), (161, 9, 2, 0, 1, 6), (200, 32, 2, 1, 1, 6),
                                                 (209, 1, 2, 1, 1, 6), (255, 32, 2, 1, 1, 2), (256, 32, 1, 1, 0, 6)])
def test_propagate_orbitals(M, N, W, pre, post, nmax):
    from ipie_b200._lib import call, ptr, stream

    rng = np.random.default_rng(M + N)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    v = torch.complex(real(W, M, M), real(W, M, M)) / M ** 0.5
    lda = M + (M & 1)
    e = torch.full((M, lda), float("nan"), dtype=torch.float64, device="cuda")  # the row padding is not read
    e[:, :M] = torch.eye(M, device="cuda") + 0.1 * real(M, M) / M ** 0.5
    phi = torch.complex(real(W, M, N), real(W, M, N))
    out = torch.full_like(phi, float("nan"))
    call("ipie_b200_propagate_orbitals", ptr(v), ptr(e), lda, ptr(phi), ptr(out), W, M, N, nmax, pre, post, stream())
    one = e[:, :M].to(phi.dtype)
    want = one @ phi if pre else phi
    t = want
    for n in range(1, nmax + 1):
        t = v @ t / n
        want = want + t
    if post:
        want = one @ want
    assert float((out - want).norm() / want.norm()) < 1e-12
