"""One batch of walkers against the same walkers in two halves.  The K splits of the FP64 products, the X split of the
field shift and the runs of the mixed exchange follow from the batch size, so a walker's sums are added in
another order (bitwise reproducible for a fixed batch, not across batches): the difference is bounded by the
rounding of two sums of n terms, 2 n 2^-53 of the absolute sum, and has to be within that."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def _data(seed):
    rng = np.random.default_rng(seed)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    return real, lambda *s: torch.complex(real(*s), real(*s))


def _halves(f, W):
    """f(lo, hi) over the whole batch and over its two (unequal) halves, concatenated."""
    h = W // 2 - 1
    return f(0, W), tuple(torch.cat(p) for p in zip(f(0, h), f(h, W)))


@pytest.mark.parametrize("W,X,M,na,nb", [(640, 600, 108, 15, 15), (66, 120, 26, 5, 5), (1030, 200, 45, 3, 2), (2400, 520, 9, 2, 1)])
def test_force_bias_and_field_shift(W, X, M, na, nb):
    from ipie_b200._lib import call, ptr, stream

    real, cplx = _data(W)
    ra, rb, ga, gb, xi, mf = real(X, na * M), real(X, nb * M), cplx(W, na * M), cplx(W, nb * M), real(W, X), cplx(X)

    def run(lo, hi):
        n = hi - lo
        v, cmf, cfb = cplx(n, X), cplx(n), cplx(n)
        xs = cplx(X, n)
        call("ipie_b200_construct_force_bias_batch_single_det", ptr(ra), ptr(rb), ptr(ga[lo:hi]), ptr(gb[lo:hi]), n, X,
             M, na, nb, ptr(v), stream())
        call("ipie_b200_field_shift", ptr(v), ptr(xi[lo:hi]), ptr(mf), n, X, 0.07, 1e300, ptr(xs), ptr(cmf), ptr(cfb),
             stream())
        return v, xs.T.contiguous(), cmf, cfb

    (v, xs, cmf, cfb), (v2, xs2, cmf2, cfb2) = _halves(run, W)
    size = ga.abs() @ ra.T.abs() + gb.abs() @ rb.T.abs()
    dv = 2 * (na + nb) * M * U * size  # of the force bias
    assert bool(((v - v2).abs() <= dv).all())
    xb = (xi - xs).abs()
    dx = 0.07 * dv + 4 * U * (xs.abs() + xb)  # of a shifted field (and xbar)
    assert bool(((xs - xs2).abs() <= dx).all())
    assert bool(((cmf - cmf2).abs() <= 0.07 * (dx * mf.abs() + 2 * X * U * xs.abs() * mf.abs()).sum(1)).all())
    assert bool(((cfb - cfb2).abs() <= ((xi.abs() + xb) * dx + 2 * X * U * (xi.abs() + xb) * xb).sum(1)).all())


@pytest.mark.parametrize("W,X,M,N", [(300, 64, 40, 7), (150, 90, 76, 10), (40, 50, 64, 20)])
def test_energies(W, X, M, N):
    from ipie_b200._lib import call, lib, ptr, stream

    real, cplx = _data(W)
    r, g = real(X, N * M), cplx(W, N, M)
    np_ = 8 if N <= 8 else 16 if N <= 16 else 32
    mp = (M + 7) // 8 * 8
    pair = torch.zeros((2, X * np_, mp), dtype=torch.float16, device="cuda")
    call("ipie_b200_rchol_pad_split", ptr(r), X, N, M, 256.0, ptr(pair[0]), ptr(pair[1]), stream())
    status = torch.zeros(1, dtype=torch.int32, device="cuda")

    def run(lo, hi):
        n = hi - lo
        part = cplx(lib().ipie_b200_exchange_rows(n, X, M, N), n)
        call("ipie_b200_exchange", ptr(r), ptr(g[lo:hi]), n, X, M, N, ptr(part), stream())
        gwork = torch.empty(4 * n * 32 * M, dtype=torch.float32, device="cuda")
        mpart, out = cplx((X * np_ + 127) // 128 + 1, n), cplx(n)
        call("ipie_b200_exchange_mixed", ptr(pair[0]), ptr(pair[1]), 256.0, ptr(g[lo:hi]), None, None, None, n, X, M, N,
             ptr(gwork), ptr(mpart), ptr(out), ptr(status), stream())
        return part.sum(0), out

    (e, mixed), (e2, mixed2) = _halves(run, W)
    assert int(status) == 0
    t = torch.einsum("xim,wjm->wxij", r.reshape(X, N, M).abs(), g.abs())
    size = torch.einsum("wxij,wxji->w", t, t)
    assert bool(((e - e2).abs() <= 2 * (2 * M + N * N * X) * U * size).all())
    # the FP32 sums inside a tile of 32 products do not move; those over tiles are FP64
    assert bool(((mixed - mixed2).abs() <= 2 * N * N * X * U * size).all())
