"""The mixed exchange with the Green's function in tensor memory (M <= 256) and streamed (M > 256, and longer rows on
one or two tiles per SM): runs that split a walker tile, several walker tiles per run, K steps that end inside a chunk, every row padding;
against torch in complex128.  Each product carries ~3 x 2^-22 from the split operands and ~2^-17 x K / 2048
at most from FP32 accumulation over chunks of 128 K; relative to sum |T_ij|^2 that stays below 3e-6."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,X,M,N", [(1, 1, 4, 1), (3, 5, 26, 5), (17, 333, 65, 8), (9, 41, 64, 9), (300, 23, 133, 15),
                                     (5, 700, 128, 16), (1, 601, 129, 17), (301, 7, 200, 23), (33, 150, 256, 32),
                                     (7, 30, 257, 12), (4, 9, 264, 32),
                                     # streamed for few tiles, for runs across walker tiles; neither; short rows
                                     (4, 100, 224, 12), (12, 600, 200, 12), (8, 600, 200, 12), (12, 600, 120, 12)])
def test_exchange_mixed(W, X, M, N):
    from ipie_b200._lib import call, ptr, stream

    rng = np.random.default_rng(M)
    real = lambda *s: torch.from_numpy(rng.normal(size=s)).cuda()
    r, g = real(X, N * M), torch.complex(real(W, N, M), real(W, N, M))
    np_ = 8 if N <= 8 else 16 if N <= 16 else 32
    mp = (M + 7) // 8 * 8
    pair = torch.zeros((2, X * np_, mp), dtype=torch.float16, device="cuda")
    scale = 256.0
    call("ipie_b200_rchol_pad_split", ptr(r), X, N, M, scale, ptr(pair[0]), ptr(pair[1]), stream())
    gwork = torch.empty(4 * W * 32 * max(M, 8), dtype=torch.float32, device="cuda")
    part = torch.full(((X * np_ + 127) // 128 + 1, W), float("nan"), dtype=torch.complex128, device="cuda")
    out = torch.empty(W, dtype=torch.complex128, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    call("ipie_b200_exchange_mixed", ptr(pair[0]), ptr(pair[1]), scale, ptr(g), None, None, None, W, X, M, N,
         ptr(gwork), ptr(part), ptr(out), ptr(status), stream())
    t = torch.einsum("xim,wjm->wxij", r.reshape(X, N, M).to(g.dtype), g)
    want = torch.einsum("wxij,wxji->w", t, t)
    size = (t.abs() ** 2).sum(dim=(1, 2, 3))
    assert int(status) == 0
    assert float(((out - want).abs() / size).max()) < 3e-6
