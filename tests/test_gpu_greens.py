"""Green's functions and overlaps at the edges of the tensor-core kernel's tiles (N = 8, 16, 24, 32), of its
chunks of M and of its pivoting (overlap blocks whose leading entries vanish), against torch in complex128.

The inverse's error grows with the condition number of O: random overlap blocks reach 1e3 to 1e4 here, so
1e-10 leaves a factor of ten over N cond eps."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


def _reference(phi, psi_conj):
    o = phi.transpose(1, 2) @ psi_conj
    return torch.linalg.solve(o, phi.transpose(1, 2)), torch.linalg.det(o)


@pytest.mark.parametrize("M,na,nb,W", [(1, 1, 0, 2), (5, 3, 1, 9), (26, 5, 5, 64), (16, 8, 7, 5), (33, 9, 8, 3),
                                       (76, 16, 10, 7), (40, 17, 15, 3), (149, 23, 17, 5), (48, 24, 24, 3),
                                       (50, 25, 2, 4), (200, 32, 32, 3), (32, 32, 31, 2)])
@pytest.mark.parametrize("zero_lead", [False, True])
def test_greens_function(M, na, nb, W, zero_lead):
    from ipie_b200._lib import call, ptr, stream

    rng = np.random.default_rng(M + na)
    cplx = lambda *s: torch.from_numpy(rng.normal(size=s) + 1j * rng.normal(size=s)).cuda()
    pa, pb, qa, qb = cplx(W, M, na), cplx(W, M, nb), cplx(M, na), cplx(M, nb)
    if zero_lead and na > 1:
        # O[i, j] = 0 for i < na // 2, j < na // 2: the first pivots come from the lower rows
        h = na // 2
        pa[:, : M // 2, :h] = 0
        qa[M // 2:, :h] = 0
    ls = torch.from_numpy(rng.normal(size=W)).cuda()
    ga, gb = torch.full((W, na, M), float("nan"), dtype=pa.dtype, device="cuda"), cplx(W, nb, M)
    ov, ld = torch.zeros(W, dtype=pa.dtype, device="cuda"), torch.zeros(W, 2, dtype=pa.dtype, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("ipie_b200_greens_function_single_det_batch", ptr(pa), ptr(pb), W, M, na, nb, ptr(qa), ptr(qb), ptr(ls),
         ptr(ga), ptr(gb), ptr(ov), ptr(ld), ptr(status), stream())
    wa, da = _reference(pa, qa)
    assert float((ga - wa).norm() / wa.norm()) < 1e-10
    det = da
    if nb:
        wb, db = _reference(pb, qb)
        assert float((gb - wb).norm() / wb.norm()) < 1e-10
        det = da * db
    want = det * torch.exp(-ls)
    assert float(((ov - want).abs() / want.abs()).max()) < 1e-10
    assert float((torch.exp(ld[:, 0].real) - da.abs()).abs().max() / da.abs().max()) < 1e-10
    ov2 = torch.zeros_like(ov)
    call("ipie_b200_calc_overlap_single_det_uhf", ptr(pa), ptr(pb), W, M, na, nb, ptr(qa), ptr(qb), ptr(ls), ptr(ov2),
         ptr(status), stream())
    assert torch.equal(ov2, ov)
    assert int(status.item()) == 0


def test_singular_overlap_is_flagged():
    from ipie_b200._lib import call, ptr, stream

    M, N, W = 20, 10, 3
    rng = np.random.default_rng(0)
    pa = torch.from_numpy(rng.normal(size=(W, M, N)) + 0j).cuda()
    pa[1, :, 4] = 0  # a zero row of O: every candidate of one pivot is exactly zero
    q, ls = torch.from_numpy(rng.normal(size=(M, N)) + 0j).cuda(), torch.zeros(W, dtype=torch.float64, device="cuda")
    g, ov = torch.zeros(W, N, M, dtype=pa.dtype, device="cuda"), torch.zeros(W, dtype=pa.dtype, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("ipie_b200_greens_function_single_det_batch", ptr(pa), ptr(pa), W, M, N, 0, ptr(q), ptr(q), ptr(ls), ptr(g),
         ptr(g), ptr(ov), None, ptr(status), stream())
    assert int(status.item()) & 2
    want, det = _reference(pa[::2], q)
    assert float((g[::2] - want).norm() / want.norm()) < 1e-10  # the other walkers are unharmed


@pytest.mark.parametrize("N", [5, 10, 19, 32])
@pytest.mark.parametrize("scale", [1e-25, 1e-100, 1e60])
def test_pivot_of_a_scaled_column(N, scale):
    """A column of O far from 1 whose first entry is zero: the pivot is still the column's largest entry."""
    from ipie_b200._lib import call, ptr, stream

    M, W = 40, 3
    rng = np.random.default_rng(N)
    cplx = lambda *s: torch.from_numpy(rng.normal(size=s) + 1j * rng.normal(size=s)).cuda()
    pa, q = cplx(W, M, N), cplx(M, N)
    pa[:, : M // 2, 0] = 0  # O[0, 0] = 0
    q[M // 2:, 0] = 0
    q[:, 0] *= scale
    ls = torch.zeros(W, dtype=torch.float64, device="cuda")
    g, ov = torch.empty(W, N, M, dtype=pa.dtype, device="cuda"), torch.empty(W, dtype=pa.dtype, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("ipie_b200_greens_function_single_det_batch", ptr(pa), ptr(pa), W, M, N, 0, ptr(q), ptr(q), ptr(ls), ptr(g),
         ptr(g), ptr(ov), None, ptr(status), stream())
    assert int(status.item()) == 0
    want, det = _reference(pa, q)
    err = (g - want).abs().amax(dim=(0, 2)) / want.abs().amax(dim=(0, 2))  # row by row: row 0 carries 1 / scale
    assert float(err.max()) < 1e-10
    assert float(((ov - det).abs() / det.abs()).max()) < 1e-10


def _extended(phi, psi_conj):
    """Ghalf (W, N, M) and det O in extended precision: elimination, and an FP64 inverse refined."""
    p = phi.astype(np.clongdouble)
    o = np.einsum("wmi,mj->wij", p, psi_conj.astype(np.clongdouble))
    a, det, w = o.copy(), np.ones(len(o), dtype=np.clongdouble), np.arange(len(o))
    for k in range(o.shape[1]):
        r = k + np.argmax(np.abs(a[:, k:, k]), axis=1)
        t = a[w, r].copy()
        a[w, r] = a[:, k]
        a[:, k] = t
        det *= np.where(r != k, -1, 1) * a[:, k, k]
        a[:, k + 1:, k:] -= (a[:, k + 1:, k] / a[:, k, k][:, None])[:, :, None] * a[:, None, k, k:]
    x, one = np.linalg.inv(o.astype(complex)).astype(np.clongdouble), np.eye(o.shape[1])
    for _ in range(3):
        x = x + np.einsum("wij,wjk->wik", x, one - np.einsum("wij,wjk->wik", o, x))
    return np.einsum("wij,wmj->wim", x, p), det


@pytest.mark.parametrize("M,N,W,most_g,most_o", [(200, 32, 48, 5.4e-16, 2.5e-15), (76, 10, 96, 3.4e-16, 8.5e-16)])
def test_greens_rounding(M, N, W, most_g, most_o):
    """Rounding for a complex trial and walkers near it, rms over the batch.  The bounds are about 1.2 times what
    O's sums of M terms and one rounding of an entry per panel show; both halves of a complex product in
    one chain, of 2 M terms and on the entries themselves, show 1.3 to 2 times."""
    from ipie_b200._lib import call, ptr, stream

    rng = np.random.default_rng(1)
    psi = np.linalg.qr(rng.normal(size=(M, N)) + 1j * rng.normal(size=(M, N)))[0]
    phi = psi + 0.3 / M ** 0.5 * (rng.normal(size=(W, M, N)) + 1j * rng.normal(size=(W, M, N)))
    psi_conj = np.ascontiguousarray(psi.conj())
    want, det = _extended(phi, psi_conj)
    p, q = torch.from_numpy(phi).cuda(), torch.from_numpy(psi_conj).cuda()
    g, ov = torch.empty(W, N, M, dtype=p.dtype, device="cuda"), torch.empty(W, dtype=p.dtype, device="cuda")
    ls, status = torch.zeros(W, dtype=torch.float64, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    call("ipie_b200_greens_function_single_det_batch", ptr(p), ptr(p), W, M, N, 0, ptr(q), ptr(q), ptr(ls), ptr(g),
         ptr(g), ptr(ov), None, ptr(status), stream())
    assert int(status.item()) == 0
    assert float(np.linalg.norm((g.cpu().numpy() - want).ravel()) / np.linalg.norm(want.ravel())) < most_g
    assert float(np.sqrt(np.mean(np.abs(ov.cpu().numpy() / det - 1) ** 2))) < most_o
