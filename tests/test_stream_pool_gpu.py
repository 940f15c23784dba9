"""The pool of side streams: work of one caller's stream does not queue up behind
another's, concurrent threads get bundles of their own, and a capture takes none
of the pool's."""
import threading

import pytest

from mnpbem_b200 import _native as nat

pytestmark = pytest.mark.gpu


class _LU:
    """A factorisation with the look-ahead schedule (two leases) on its own buffers."""

    def __init__(self, n, seed):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed)
        self.n = n
        self.A = torch.randn((n, n), dtype=torch.complex128, device="cuda", generator=g) / n ** 0.5
        self.A += 4 * torch.eye(n, dtype=self.A.dtype, device="cuda")
        self.F = torch.empty_like(self.A)
        self.rowmap, self.ipiv = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
        self.info = torch.zeros(1, dtype=torch.int32, device="cuda")
        self.wsb = int(nat.lib().bem200_getrf_workspace_size(nat.C128, 0, n))
        self.ws = torch.empty(self.wsb, dtype=torch.uint8, device="cuda")

    def run(self):
        self.F.copy_(self.A)
        nat.call("bem200_getrf_ex", nat.C128, 0, self.n, nat.ptr(self.F), self.n, nat.ptr(self.rowmap), nat.ptr(self.ipiv),
                 nat.ptr(self.info), nat.ptr(self.ws), self.wsb, 0, 0, nat.stream_ptr())


def test_streams_do_not_wait_for_each_other(cuda):
    """Long factorisations on one stream, a short one on another: the short one is
    done first, also when its stream had no side streams before."""
    import torch
    big, small = _LU(4000, 1), _LU(600, 2)
    s1 = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s1):
        big.run()
    torch.cuda.synchronize()
    for _ in range(4):
        done = torch.cuda.Event()
        with torch.cuda.stream(s1):
            for _ in range(6):
                big.run()
            done.record()
        s2 = torch.cuda.Stream()
        with torch.cuda.stream(s2):
            small.run()
        s2.synchronize()
        assert not done.query()
        torch.cuda.synchronize()


def test_threads_share_the_pool(cuda):
    import torch
    lus = [_LU(600 + 64 * i, i) for i in range(6)]
    refs = []
    for lu in lus:
        lu.run()
        torch.cuda.synchronize()
        refs.append(lu.F.clone())
        lu.F.zero_()
    torch.cuda.synchronize()
    errors = []

    def work(lu, ref):
        try:
            for _ in range(10):
                s = torch.cuda.Stream()
                with torch.cuda.stream(s):
                    lu.run()
                s.synchronize()
                assert torch.equal(lu.F, ref)
                lu.F.zero_()
                torch.cuda.synchronize()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)
    threads = [threading.Thread(target=work, args=a) for a in zip(lus, refs)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, errors


def test_capture_between_pooled_calls(cuda):
    import torch
    lu = _LU(700, 3)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        lu.run()
        s.synchronize()
        ref = lu.F.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s, capture_error_mode="thread_local"):
            lu.run()
        lu.F.zero_()
        g.replay()
        s.synchronize()
        assert torch.equal(lu.F, ref)
        lu.F.zero_()
        lu.run()
        s.synchronize()
        assert torch.equal(lu.F, ref)
