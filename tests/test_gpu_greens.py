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
