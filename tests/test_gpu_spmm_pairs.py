"""The second matrix of a pattern seen in a fused product: its plan has to serve products of its own."""
import numpy as np
import pytest

import ommgpu as G
from ommgpu import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("norb", [13, 24])
def test_second_matrix_of_a_fused_product_alone(norb, cplx):
    """functional_grad multiplies H and S (one pattern) as a pair; S alone afterwards in psp_gemspm, psp_gespmm
    and energy_adjoint gives the products of a matrix that was never part of one.  The gradient itself against
    numpy (complex pairs are two products that share the column groups)."""
    p = synth.lattice((5, 5, 5), seed=7, norb=norb, nocc=2, compute_mu=False)
    assert np.array_equal(p.H.colptr, p.S.colptr) and np.array_equal(p.H.rowind, p.S.rowind)
    rng = np.random.default_rng(norb)
    m, n = p.m, 70

    def mat(M):
        z = np.exp(1j * rng.uniform(0, 6, M.nnz)) if cplx else 1.0
        return synth.CSCMatrix(M.dim1, M.dim2, M.colptr, M.rowind, M.val * z)

    hh, ss = mat(p.H), mat(p.S)
    Cn = rng.standard_normal((n, m)) + (1j * rng.standard_normal((n, m)) if cplx else 0)
    Cn = np.asfortranarray(Cn / np.sqrt(m))
    C = G.Matrix.from_numpy(Cn)
    Gm, out, ref = (G.Matrix.allocate(n, m, "gzden" if cplx else "gdden") for _ in range(3))
    H, S, alone = G.Matrix.from_csc(hh), G.Matrix.from_csc(ss), G.Matrix.from_csc(ss)
    omega = G.functional_grad(m, n, H, S, C, Gm)
    for M, R in ((S, out), (alone, ref)):
        G.psp_gemspm(n, m, m, C, "n", M, "n", R)
    assert np.array_equal(out.numpy(), ref.numpy())
    Hd, Sd = hh.to_dense(), ss.to_dense()
    HC, SC = Cn @ Hd, Cn @ Sd
    HW, SW = HC @ Cn.conj().T, SC @ Cn.conj().T
    # every product is within its inner length times eps of the sum of magnitudes (at most 33 norb, m and 2 n
    # terms here); a margin of 4 covers complex terms and the sums of products
    eps, aC = np.finfo(float).eps, np.abs(Cn)
    aH, aS = aC @ np.abs(Hd), aC @ np.abs(Sd)
    aHW, aSW = aH @ aC.T, aS @ aC.T
    assert np.all(np.abs(out.numpy() - SC) <= 4 * 33 * norb * eps * aS)
    bar = 4 * (33 * norb + m + 2 * n) * eps * (4 * aH + 2 * aSW @ aH + 2 * aHW @ aS)
    assert np.all(np.abs(Gm.numpy() - (4 * HC - 2 * SW @ HC - 2 * HW @ SC)) <= bar)
    want = (2 * np.trace(HW) - np.sum(HW.conj() * SW)).real
    assert abs(omega - want) <= 4 * (33 * norb + m + n * n) * eps * (2 * np.trace(aHW) + np.sum(aHW * aSW))
    Ct, tall = G.Matrix.from_numpy(np.asfortranarray(Cn.T)), G.Matrix.allocate(m, n, "gzden" if cplx else "gdden")
    G.psp_gespmm(m, n, m, S, "t", Ct, "n", tall)
    assert np.all(np.abs(tall.numpy() - Sd.T @ Cn.T) <= 4 * 33 * norb * eps * aS.T)
    got = [G.energy_adjoint(m, n, M, C, [H]) for M in (S, alone)]
    assert np.array_equal(got[0], got[1])
