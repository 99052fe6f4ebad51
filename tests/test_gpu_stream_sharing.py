"""The library on a stream that its caller uses from another thread at the same time."""
import threading

import pytest

import ommgpu as G

pytestmark = pytest.mark.gpu


def test_work_of_another_thread_on_the_stream_runs_once():
    """Small solves (whose steps run as graphs) on the caller's stream while another thread counts up on it:
    every addition is carried out exactly once, and the solves are those of an undisturbed stream."""
    import torch

    m, n = 120, 40
    g = torch.Generator(device="cuda").manual_seed(3)
    Q, _ = torch.linalg.qr(torch.randn(m, m, generator=g, device="cuda", dtype=torch.float64))
    lam = torch.linspace(-2.0, -1.0, m, device="cuda", dtype=torch.float64)
    lam[n:] += 2.5
    H = (Q * lam) @ Q.t()
    H = 0.5 * (H + H.t())
    C, D = torch.zeros(m, n, device="cuda", dtype=torch.float64), torch.zeros_like(H)
    h, c, d = (G.Matrix.register_gden(t.data_ptr(), r, m, False, keep=t) for t, r in ((H, m), (C, n), (D, m)))
    G.set_log(None)
    torch.cuda.synchronize()

    def solve():
        e, rc = G.omm(m, n, h, None, True, d, False, 0.0, c, False, dealloc=True)
        assert rc == 0
        return e, G.stats()["icg"], D.clone()

    ref = solve()
    stream = torch.cuda.Stream()
    count, queued, stop = torch.zeros(1, device="cuda", dtype=torch.float64), [0], threading.Event()
    torch.cuda.synchronize()

    def busy():
        with torch.cuda.stream(stream):
            while not stop.is_set():
                count.add_(1.0)
                queued[0] += 1

    t = threading.Thread(target=busy)
    G.set_stream(stream.cuda_stream)
    try:
        t.start()
        got = []
        for _ in range(20):
            got.append(solve())
    finally:
        stop.set()
        t.join()
        stream.synchronize()
        G.set_stream(0)
    torch.cuda.synchronize()
    assert queued[0] > 0 and float(count) == queued[0]
    for e, steps, dens in got:
        assert e == ref[0] and steps == ref[1] and torch.equal(dens, ref[2])
