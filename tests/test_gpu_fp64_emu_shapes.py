"""FP64 products on the int8 tensor cores at the shapes where a tile, a slab or a part can go wrong: every
tile width of the SM-pair kernel, ragged rows and columns, slabs of the exponent passes, and complex
products (stacked parts) with every op, odd rows, beta and parts of very different size.

The reference is torch's FP64 product of the same operands; each side is within a few ulp of the
sums of magnitudes, so 1e-13 |A||B| holds for K up to 10^4 (the bar the solver's shapes are held to)."""
import numpy as np
import pytest

import ommgpu as G

pytestmark = pytest.mark.gpu


def _mat(t):
    buf = t.t().contiguous()
    return G.Matrix.register_gden(buf.data_ptr(), t.shape[0], t.shape[1], t.is_complex(), keep=buf), buf


def _op(t, o):
    return t if o == "n" else t.t() if o == "t" else t.mH


def _check(M, N, K, opA, opB, cplx, alpha=1.0, beta=0.0, scale_im=1.0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)

    def rnd(*shape):
        x = torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64)
        if cplx:
            x = torch.complex(x, scale_im * torch.randn(*shape, generator=g, device="cuda", dtype=torch.float64))
        return x

    A = rnd(*((M, K) if opA == "n" else (K, M)))
    B = rnd(*((K, N) if opB == "n" else (N, K)))
    C0 = rnd(M, N)
    (a, ka), (b, kb), (c, kc) = _mat(A), _mat(B), _mat(C0)
    torch.cuda.synchronize()
    G.mm_multiply(a, opA, b, opB, c, alpha, beta)
    x, y = _op(A, opA), _op(B, opB)
    ref = alpha * (x @ y) + beta * C0
    err = (kc.t() - ref)
    if cplx:  # each part against its own sums of magnitudes
        mre = x.real.abs() @ y.real.abs() + x.imag.abs() @ y.imag.abs() + C0.real.abs()
        mim = x.real.abs() @ y.imag.abs() + x.imag.abs() @ y.real.abs() + C0.imag.abs()
        assert float((err.real.abs() / mre).max()) <= 1e-13
        assert float((err.imag.abs() / mim).max()) <= 1e-13
    else:
        assert float((err.abs() / (x.abs() @ y.abs() + C0.abs())).max()) <= 1e-13


@pytest.mark.parametrize("N", [128, 130, 161, 193, 225, 257, 300, 385, 515, 777])
@pytest.mark.parametrize("M,K,opA", [(255, 8192, "n"), (1001, 2003, "t"), (129, 9001, "n")])
def test_real_tile_widths(M, N, K, opA):
    _check(M, N, K, opA, "n" if N % 2 else "t", False)


@pytest.mark.parametrize("opA", ["n", "t", "c"])
@pytest.mark.parametrize("opB", ["n", "t", "c"])
@pytest.mark.parametrize("M,N,K", [(257, 131, 4099), (1030, 601, 258)])
def test_complex_ops(M, N, K, opA, opB):
    _check(M, N, K, opA, opB, True, 0.75, -1.25)


@pytest.mark.parametrize("scale_im", [1e-12, 1e9])
def test_complex_parts_keep_their_own_precision(scale_im):
    _check(259, 300, 2001, "n", "c", True, scale_im=scale_im)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [(1100, 261), (1031, 384)])
def test_hermitian_blocks_start_inside_tiles(m, n, cplx):
    """omm's W matrices and density with n and m off the tile sizes: the density of the converged
    coefficients is (2 - S_W) contracted with them, and idempotent."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    dt = torch.complex128 if cplx else torch.float64
    Q, _ = torch.linalg.qr(torch.randn(m, m, generator=g, device="cuda", dtype=dt))
    lam = torch.linspace(-2.0, -1.0, m, device="cuda", dtype=torch.float64)
    lam[n:] += 2.5
    H = (Q * lam) @ Q.mH
    (h, kh), (c, kc), (d, kd) = _mat(0.5 * (H + H.mH)), _mat(H[:n] * 0), _mat(H * 0)
    torch.cuda.synchronize()
    G.set_log(None)
    e, rc = G.omm(m, n, h, None, True, d, False, 0.0, c, False, cg_tol=1e-12, dealloc=True)
    assert rc == 0 and abs(e - float(lam[:n].sum())) <= 1e-9 * abs(e)
    D, C = kd.t(), kc.t()
    ref = C.mH @ (2.0 * C - (C @ C.mH) @ C)
    assert float((D - ref).abs().max()) <= 1e-12
    assert float((D - D.mH).abs().max()) == 0.0
    P = Q[:, :n] @ Q[:, :n].mH
    assert float((D - P).abs().max()) <= 1e-4


@pytest.mark.parametrize("cplx,N", [(True, 140001), (False, 530003)])
def test_more_columns_than_one_reconstruction_grid(cplx, N):
    """Emulated products of so many columns that one launch of the reconstruction could not number its blocks:
    the columns before, at and behind the panels' ends."""
    import torch

    M, K = 256, 1000 if cplx else 512
    g = torch.Generator(device="cuda").manual_seed(N)
    dt = torch.complex128 if cplx else torch.float64
    A = torch.randn(M, K, generator=g, device="cuda", dtype=dt)
    B = torch.randn(N, K, generator=g, device="cuda", dtype=dt)  # column-major K x N
    C = torch.zeros(N, M, device="cuda", dtype=dt)
    a, ka = _mat(A)
    b = G.Matrix.register_gden(B.data_ptr(), K, N, cplx, keep=B)
    c = G.Matrix.register_gden(C.data_ptr(), M, N, cplx, keep=C)
    torch.cuda.synchronize()
    G.mm_multiply(a, "n", b, "n", c)
    at = 130816 if cplx else 524032
    for lo, hi in ((0, 300), (at - 300, at + 300), (N - 300, N)):
        x = B[lo:hi].t()
        assert float(((C[lo:hi].t() - A @ x).abs() / (A.abs() @ x.abs())).max()) <= 1e-13
