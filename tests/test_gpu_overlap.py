"""Products whose result shares memory with an operand: the operand is read in full before the result is
written, so they equal the products into a matrix of their own."""
import numpy as np
import pytest

import ommgpu as G
from ommgpu import synth

pytestmark = pytest.mark.gpu


def _rnd(g, *shape, cplx=False):
    import torch

    return torch.randn(*shape, generator=g, device="cuda", dtype=torch.complex128 if cplx else torch.float64)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("opA,opB", [("n", "t"), ("t", "t"), ("n", "n"), ("t", "c"), ("c", "c")])
@pytest.mark.parametrize("norb", [13, 24])
def test_csc_times_dense_in_place(norb, opA, opB, cplx):
    """C = alpha op(A) op(C) + beta C of a square atom-block A (24: no zero cell in its column groups)."""
    import torch

    H = synth.lattice((5, 5, 5), seed=norb, norb=norb, nocc=1, compute_mu=False).H
    if cplx:
        rng = np.random.default_rng(norb)
        H = synth.CSCMatrix(H.dim1, H.dim2, H.colptr, H.rowind, H.val * np.exp(1j * rng.uniform(0, 6, H.nnz)))
    A, m = G.Matrix.from_csc(H), H.dim1
    X = _rnd(torch.Generator(device="cuda").manual_seed(norb), m, m, cplx=cplx)
    for _ in range(4):
        own, both = X.clone(), X.clone()  # column-major: the handles see X^T
        src = X.clone()
        hs, ho, hb = (G.Matrix.register_gden(t.data_ptr(), m, m, cplx, keep=t) for t in (src, own, both))
        torch.cuda.synchronize()
        G.psp_gespmm(m, m, m, A, opA, hs, opB, ho, 0.7, 0.3)
        G.psp_gespmm(m, m, m, A, opA, hb, opB, hb, 0.7, 0.3)
        # both routes form the same Z; alpha Z + beta C is rounded at most four times per part, each within
        # eps of |alpha Z| + |beta C| <= |result| + 2 |beta C|
        bar = 4 * np.finfo(float).eps * (float(own.abs().max()) + 2 * float(X.abs().max()))
        assert float((both - own).abs().max()) <= bar


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("shift", [0, 1, 300 * 600, 600 * 600 - 1])
@pytest.mark.parametrize("which", ["A", "B"])
def test_dense_result_inside_an_operand(which, shift, cplx):
    """C = A B with C registered `shift` elements into the memory of A or B, at a size where the int8 emulation
    (which reads its operands first) is not the faster engine."""
    import torch

    m = 600
    g = torch.Generator(device="cuda").manual_seed(shift)
    A, B = _rnd(g, m, m, cplx=cplx), _rnd(g, m, m, cplx=cplx)
    ref, mag = A.t() @ B.t(), A.abs().t() @ B.abs().t()  # the handles see the transposes
    for _ in range(4):
        store = torch.zeros(2 * m * m, dtype=A.dtype, device="cuda")
        other = (B if which == "A" else A).clone()
        store[:m * m] = (A if which == "A" else B).reshape(-1)
        C = store[shift:shift + m * m]
        hs, ho, hc = (G.Matrix.register_gden(t.data_ptr(), m, m, cplx, keep=t) for t in (store, other, C))
        torch.cuda.synchronize()
        G.mm_multiply(*((hs, "n", ho, "n") if which == "A" else (ho, "n", hs, "n")), hc)
        # both products are within m eps |A||B| (complex: four real ones), the kept 53 bits included
        assert float(((C.view(m, m).t() - ref).abs() / mag).max()) <= 8 * m * np.finfo(float).eps
