"""Plans of different sizes in several threads at once: a kernel's limit of
dynamic shared memory belongs to the process, and a launch that needs more than
another thread has just allowed is refused."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _together(jobs, rounds):
    """Every job (set-up -> one call) in a thread of its own, on its own stream."""
    errors, start = [], threading.Barrier(len(jobs))

    def work(make):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                with make() as call:
                    start.wait()
                    for _ in range(rounds):
                        call()
                    torch.cuda.current_stream().synchronize()
        except Exception as e:  # noqa: BLE001 -- reported below
            errors.append(e)
            start.abort()

    threads = [threading.Thread(target=work, args=(j,)) for j in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


class _Solver:
    def __init__(self, N, K=6):
        from miscellaneous_gb300.nfft import Plan
        self.p = Plan(N, N, K=K, stream=torch.cuda.current_stream())
        self.p.set_points(*[torch.rand(500, device="cuda") - 0.5 for _ in range(2)])
        self.F = torch.randn(N, N, device="cuda", dtype=torch.complex64)
        self.f = torch.randn(500, device="cuda", dtype=torch.complex64)
        self.out, self.Out = torch.empty_like(self.f), torch.empty_like(self.F)

    def __enter__(self):
        return lambda: (self.p.forward(self.F, out=self.out), self.p.adjoint(self.f, out=self.Out))

    def __exit__(self, *exc):
        self.p.close()


class _Type3:
    def __init__(self, eps):
        from miscellaneous_gb300.nufft3 import NUFFT_2D
        d = [torch.rand(200, device="cuda", dtype=torch.float64) for _ in range(4)]
        f = torch.randn(200, device="cuda", dtype=torch.complex64)
        self.call = lambda: NUFFT_2D(*d, f, eps)

    def __enter__(self):
        return self.call

    def __exit__(self, *exc):
        pass


def test_mixed_radix_passes():
    # 54, 68 and 94 KB of shared memory a column CTA
    _together([lambda N=N: _Solver(N) for N in (400, 500, 700, 420)], 3000)


def test_type3():
    _together([lambda e=e: _Type3(e) for e in (1e-4, 1e-6, 1e-9, 1e-13)], 150)
