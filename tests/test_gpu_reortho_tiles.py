"""Cholesky-QR reorthogonalisation at the edges of the tensor-core kernel's tiles (N = 8, 16, 24, 32) and
chunks of M, both spins of unequal size, against torch's QR with the sign of diag(R) fixed.  Blocks of cond below
10: factors and log-determinants to cond^2 eps times the block's sums, 1e-11."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _qr(phi):
    q, r = torch.linalg.qr(phi)
    d = torch.diagonal(r, dim1=1, dim2=2)
    return q * (d / d.abs())[:, None, :], d.abs().log().sum(1)


@pytest.mark.parametrize("M,na,nb,W", [(1, 1, 0, 2), (9, 3, 1, 5), (26, 8, 7, 65), (33, 9, 16, 3), (149, 23, 17, 5),
                                       (48, 24, 25, 3), (200, 32, 31, 3), (64, 32, 32, 7), (31, 17, 0, 4)])
def test_reortho(M, na, nb, W):
    from ipie_b200._lib import call, ptr, stream

    rng = np.random.default_rng(M + na)

    def block(n):
        a = rng.normal(size=(W, M, n)) + 1j * rng.normal(size=(W, M, n))
        q = np.linalg.qr(a)[0] if n else a
        mix = np.eye(n) + 0.3 * (rng.normal(size=(W, n, n)) + 1j * rng.normal(size=(W, n, n))) / max(n, 1) ** 0.5
        return torch.from_numpy(np.ascontiguousarray(q @ mix)).cuda()

    pa, pb = block(na), block(nb)
    wa, la = _qr(pa)
    wb, lb = _qr(pb) if nb else (pb.clone(), 0.0)
    real = lambda v: torch.from_numpy(v).cuda()
    shift, ldet = real(rng.normal(size=W)), real(rng.normal(size=W))
    det, ov = torch.zeros_like(shift), real(rng.normal(size=W) + 1j * rng.normal(size=W))
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    l0, o0 = ldet.clone(), ov.clone()
    call("ipie_b200_reortho", ptr(pa), ptr(pb), W, M, na, nb, ptr(shift), ptr(det), ptr(ldet), ptr(ov), ptr(status),
         stream())
    assert float((pa - wa).abs().max()) < 1e-11
    if nb:
        assert float((pb - wb).abs().max()) < 1e-11
    logd = la + lb - shift
    assert float((det.log() - logd).abs().max()) < 1e-10
    assert float((ldet - l0 - logd).abs().max()) < 1e-10
    assert float(((ov - o0 * torch.exp(-logd)) / o0).abs().max() / float(torch.exp(-logd).max())) < 1e-10
    assert int(status.item()) == 0
