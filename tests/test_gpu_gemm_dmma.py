"""FP64 products on the FP64 tensor cores at the edges of their tiles, chunks and K splits (mm_multiply picks
them for products too small for the int8 emulation), against torch's FP64 products of the same operands:
both sides are within a few ulp of the sums of magnitudes, so 1e-13 |A||B| holds at K up to 10^4."""
import numpy as np
import pytest

import ommgpu as G

pytestmark = pytest.mark.gpu


def _mat(t):
    buf = t.t().contiguous()
    return G.Matrix.register_gden(buf.data_ptr(), t.shape[0], t.shape[1], t.is_complex(), keep=buf), buf


def _op(t, o):
    return t if o == "n" else t.t() if o == "t" else t.mH


def _check(M, N, K, opA, opB, cplx, alpha=1.0, beta=0.0):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + 7 * K)
    dt = torch.complex128 if cplx else torch.float64
    A = torch.randn(*((M, K) if opA == "n" else (K, M)), generator=g, device="cuda", dtype=dt)
    B = torch.randn(*((K, N) if opB == "n" else (N, K)), generator=g, device="cuda", dtype=dt)
    C0 = torch.randn(M, N, generator=g, device="cuda", dtype=dt)
    (a, ka), (b, kb), (c, kc) = _mat(A), _mat(B), _mat(C0)
    torch.cuda.synchronize()
    G.mm_multiply(a, opA, b, opB, c, alpha, beta)
    x, y = _op(A, opA), _op(B, opB)
    ref = alpha * (x @ y) + beta * C0
    mag = abs(alpha) * (x.abs() @ y.abs()) + abs(beta) * C0.abs()
    assert float(((kc.t() - ref).abs() / mag.clamp_min(1e-300)).max()) <= 1e-13


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("opA", ["n", "t", "c"])
@pytest.mark.parametrize("opB", ["n", "t", "c"])
@pytest.mark.parametrize("M,N,K", [(33, 31, 17), (64, 96, 100), (37, 53, 61), (130, 257, 70)])
def test_ops(M, N, K, opA, opB, cplx):
    _check(M, N, K, opA, opB, cplx, (0.75 - 0.5j) if cplx else 0.75, (-1.25 + 0.25j) if cplx else -1.25)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("K", [1, 3, 4, 15, 16, 17, 95, 96, 97, 200, 385, 4099])
@pytest.mark.parametrize("M,N", [(1, 1), (32, 32), (35, 66)])
def test_chunks_and_splits(M, N, K, cplx):
    _check(M, N, K, "n", "t" if K % 2 else "n", cplx)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("m,n", [(60, 30), (101, 33), (200, 65)])
def test_small_solve(m, n, cplx):
    """The pair launches of a small CG step (D [H, S], both Gram products) and the Hermitian products:
    energy against the constructed spectrum, density Hermitian and a projector."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(m)
    dt = torch.complex128 if cplx else torch.float64
    Q, _ = torch.linalg.qr(torch.randn(m, m, generator=g, device="cuda", dtype=dt))
    L = torch.eye(m, device="cuda", dtype=dt) + 0.1 / m ** 0.5 * torch.randn(m, m, generator=g, device="cuda", dtype=dt)
    lam = torch.linspace(-2.0, -1.0, m, device="cuda", dtype=torch.float64)
    lam[n:] += 2.5
    W = L @ Q
    H, S = (W * lam) @ W.mH, L @ L.mH
    (h, kh), (s, ks) = _mat(0.5 * (H + H.mH)), _mat(0.5 * (S + S.mH))
    (c, kc), (d, kd) = _mat(H[:n] * 0), _mat(H * 0)
    torch.cuda.synchronize()
    G.set_log(None)
    e, rc = G.omm(m, n, h, s, True, d, False, 0.0, c, False, cg_tol=1e-12, dealloc=True)
    assert rc == 0 and abs(e - float(lam[:n].sum())) <= 1e-9 * abs(e)
    D = kd.t()
    assert float((D - D.mH).abs().max()) == 0.0
    U = torch.linalg.solve(L.mH, Q[:, :n])
    assert float((D - U @ U.mH).abs().max()) <= 1e-4


def test_solves_in_turn():
    """Solves of different shapes and types one after another (the CG loop's graph is made anew or takes the
    next call's parameters): each gives the same bits as it did alone."""
    import torch

    G.set_log(None)
    cases = []
    for m, n, dt in ((60, 30, torch.float64), (101, 33, torch.float64), (60, 30, torch.complex128),
                     (200, 65, torch.float64)):
        g = torch.Generator(device="cuda").manual_seed(m + n)
        Q, _ = torch.linalg.qr(torch.randn(m, m, generator=g, device="cuda", dtype=dt))
        lam = torch.linspace(-2.0, -1.0, m, device="cuda", dtype=torch.float64)
        lam[n:] += 2.5
        H = (Q * lam) @ Q.mH
        cases.append((m, n, _mat(0.5 * (H + H.mH)), _mat(H[:n] * 0), _mat(H * 0)))
    torch.cuda.synchronize()

    def solve(m, n, h, c, d):
        e, rc = G.omm(m, n, h[0], None, True, d[0], False, 0.0, c[0], False, dealloc=True)
        assert rc == 0
        return e, d[1].clone(), G.stats()["icg"]

    first = [solve(*c) for c in cases]
    for order in ((0, 0, 1, 2, 3), (3, 1, 3, 2, 0, 2)):
        for k in order:
            e, d, steps = solve(*cases[k])
            assert e == first[k][0] and steps == first[k][2] and torch.equal(d, first[k][1])


def test_solve_with_emulated_operator_products():
    """m = 2,000, n = 400: the Gram products and calc_G stay on the FP64 tensor cores, so the steps run ahead
    in a graph, while D H and D S are large enough for the int8 emulation: it is part of the graph."""
    test_small_solve(2000, 400, False)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("M,N,K", [(515, 301, 16), (1025, 417, 33), (64, 1500, 2501), (40, 40, 1501), (301, 261, 401)])
def test_short_and_long_k(M, N, K, cplx):
    """Unsplit tiles written from the accumulators (short K, odd edges), and both sides of the rule that leaves
    products with a long K to cuBLAS."""
    _check(M, N, K, "t", "n", cplx, 0.75, -1.25)
    _check(M, N, min(K, 1499), "n", "t", cplx)


def test_kept_graph_follows_the_kernels_of_its_steps():
    """The m = 2,000, n = 400 solve, whose steps hold emulated products, with those products on SM pairs (clusters
    of two CTAs), on single SMs and on pairs again: a kept graph of the one form does not serve the other, and
    all forms give the same bits."""
    import torch

    m, n = 2000, 400
    g = torch.Generator(device="cuda").manual_seed(m)
    Q, _ = torch.linalg.qr(torch.randn(m, m, generator=g, device="cuda", dtype=torch.float64))
    lam = torch.linspace(-2.0, -1.0, m, device="cuda", dtype=torch.float64)
    lam[n:] += 2.5
    H = (Q * lam) @ Q.mH
    (h, kh), (c, kc), (d, kd) = _mat(0.5 * (H + H.mH)), _mat(H[:n] * 0), _mat(H * 0)
    torch.cuda.synchronize()
    G.set_log(None)
    got = []
    try:
        for pairs in (1, 1, 0, 0, 1):
            assert G.lib().omm_gpu_tc_set_pairs(pairs) == 0
            e, rc = G.omm(m, n, h, None, True, d, False, 0.0, c, False, dealloc=True)
            assert rc == 0 and G.tc_errors() == 0
            got.append((e, G.stats()["icg"], kd.clone()))
    finally:
        assert G.lib().omm_gpu_tc_set_pairs(1) == 0
    for e, steps, dens in got[1:]:
        assert e == got[0][0] and steps == got[0][1] and torch.equal(dens, got[0][2])


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("beta", [0.0, 1.0, -0.5])
@pytest.mark.parametrize("M,N,K", [(33, 31, 17), (700, 300, 90), (1100, 1000, 1200)])
def test_zero_alpha_reads_no_operand(M, N, K, beta, cplx):
    """alpha = 0 scales C alone: an Inf or NaN in A or B does not reach it, and beta = 0 clears what C held."""
    import torch

    dt = torch.complex128 if cplx else torch.float64
    A = torch.full((M, K), float("nan"), device="cuda", dtype=dt)
    B = torch.full((K, N), float("inf"), device="cuda", dtype=dt)
    C0 = torch.randn(M, N, device="cuda", dtype=dt, generator=torch.Generator(device="cuda").manual_seed(M))
    if beta == 0.0:
        C0[0, 0] = float("nan")
    (a, ka), (b, kb), (c, kc) = _mat(A), _mat(B), _mat(C0)
    torch.cuda.synchronize()
    G.mm_multiply(a, "n", b, "n", c, 0.0, beta)
    assert torch.equal(kc.t(), torch.zeros_like(C0) if beta == 0.0 else beta * C0)


@pytest.mark.parametrize("cplx,M,N,K", [(False, 512, 512, 4096), (False, 130, 1611, 3000), (False, 500, 500, 500),
                                        (False, 45, 37, 260), (False, 256, 128, 832), (True, 500, 500, 500),
                                        (True, 256, 128, 832), (True, 45, 37, 260), (True, 300, 150, 3000),
                                        (True, 37, 53, 61), (False, 897, 865, 700)])
@pytest.mark.parametrize("opA,opB", [("n", "n"), ("t", "c")])
def test_errors_do_not_grow_with_k(M, N, K, opA, opB, cplx):
    """K is added up in runs of 32 products, eights of runs and those: the rms error over sqrt(sum |a|^2 |b|^2).
    A chain of L additions of terms of one variance rounds partial sums of variance j = 1 .. L; each rounding is
    at most a half unit in the last place of its sum, of rms 2u / sqrt(12) of it, so the chain's relative variance
    is at most (u^2 / 3) L / 2.  The levels' add: L = 32, 8 and K / 256 (complex: twice the products; and at most
    eight parts of a split K).  One chain of K = 4,096 would be at 26 u.  A margin of 15 % for the sample.  Small
    products, in runs of 64, are held to the same: of sums spread evenly over an octave's logarithm the half units
    have 0.54 of that variance."""
    rng = np.random.default_rng(M + N + K)

    def rnd(r, c):
        a = rng.standard_normal((r, c))
        return np.asfortranarray(a + 1j * rng.standard_normal((r, c)) if cplx else a)

    A = rnd(*((M, K) if opA == "n" else (K, M)))
    B = rnd(*((K, N) if opB == "n" else (N, K)))
    C = G.Matrix.allocate(M, N, "gzden" if cplx else "gdden")
    G.mm_multiply(G.Matrix.from_numpy(A), opA, G.Matrix.from_numpy(B), opB, C)
    a = (A if opA == "n" else A.T)[:40]
    b = (B if opB == "n" else B.conj().T)[:, :30]
    long = np.clongdouble if cplx else np.longdouble
    err = np.abs(C.numpy()[:40, :30] - a.astype(long) @ b.astype(long)).astype(float)
    size = np.sqrt(np.abs(a) ** 2 @ np.abs(b) ** 2)
    bar = 2.0 ** -53 * np.sqrt((32 + 8 + (2 if cplx else 1) * K / 256 + 8) / 6)
    assert np.sqrt(np.mean((err / size) ** 2)) <= 1.15 * bar
