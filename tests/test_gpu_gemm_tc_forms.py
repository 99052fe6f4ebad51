"""Every tile form of the bf16 GEMM (256 x 256 on SM pairs, 128 x 256, 128 x 128 and 128 x 64 on single SMs)
at shapes whose estimated times pick it, with ragged rows, columns and K: plain products within 2e-6 of
sum_k |a_ik b_jk| and split ones within 1e-5 (the bars of the GEMM's own tests); and the columns of a wide
product agree bit for bit with the same columns formed in a narrow one (all forms add up K in the same
order)."""
import ctypes as ct

import pytest

import ommgpu as G

pytestmark = pytest.mark.gpu


def _gemm(M, N, K, A, B, lda, nseg=1, Al=None, Bl=None):
    import torch

    f = G.lib().omm_gpu_gemm_bf16
    f.argtypes = [ct.c_int, ct.c_int, ct.c_int, ct.c_void_p, ct.c_void_p, ct.c_int, ct.c_void_p, ct.c_void_p, ct.c_int,
                  ct.c_int, ct.c_double, ct.c_double, ct.c_void_p, ct.c_int]
    out = torch.zeros(N, M, device="cuda", dtype=torch.float64)
    torch.cuda.synchronize()
    rc = f(M, N, K, A.data_ptr(), Al.data_ptr() if Al is not None else None, lda, B.data_ptr(),
           Bl.data_ptr() if Bl is not None else None, lda, nseg, 1.0, 0.0, out.data_ptr(), M)
    assert rc == 0
    return out.t()


@pytest.mark.parametrize("nseg", [1, 3])
@pytest.mark.parametrize("M,N,K", [(1, 1, 8), (129, 65, 70), (250, 125, 1000), (750, 375, 3000), (375, 3000, 750),
                                   (648, 5184, 1296), (1029, 4100, 514), (2058, 1029, 4104)])
def test_forms(M, N, K, nseg):
    import torch

    g = torch.Generator(device="cuda").manual_seed(M + N)
    lda = (K + 7) // 8 * 8
    mk = lambda r, s: (s * torch.randn(r, lda, generator=g, device="cuda")).bfloat16()  # noqa: E731
    Ah, Al, Bh, Bl = mk(M, 1.0), mk(M, 1e-3), mk(N, 1.0), mk(N, 1e-3)
    got = _gemm(M, N, K, Ah, Bh, lda, nseg, Al, Bl)
    a, al, b, bl = (t[:, :K].double() for t in (Ah, Al, Bh, Bl))
    ref, mag = a @ b.t(), a.abs() @ b.abs().t()
    if nseg == 3:
        ref = ref + a @ bl.t() + al @ b.t()
        mag = mag + a.abs() @ bl.abs().t() + al.abs() @ b.abs().t()
    assert float(((got - ref).abs() / mag).max()) <= (2e-6 if nseg == 1 else 1e-5)
    part = min(N, 40)
    narrow = _gemm(M, part, K, Ah, Bh[:part].contiguous(), lda, nseg, Al, Bl[:part].contiguous())
    assert torch.equal(got[:, :part], narrow)
