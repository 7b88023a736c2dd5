"""MMA steps of one kernel and two sizes at once, from two threads on their own streams.

Numbers of constraints that share the assemble and advance kernels need different amounts of
shared memory, and the kernels are launched at every Newton step.  Each thread's results equal, bit
for bit, those of the same call made alone (the passes' sums have a fixed order).
"""

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(6, 8), (21, 24), (33, 47)])
def test_two_threads_with_two_sizes_of_one_kernel(pkg, sizes):
    from sttopt_b200 import mma

    n, calls = 3000, 20

    def args(m):
        g = torch.Generator(device="cuda")
        g.manual_seed(m)
        r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)
        x = 0.05 + 0.9 * torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
        h = mma.History((x + 0.02 * r(n)).clamp(0, 1), (x + 0.03 * r(n)).clamp(0, 1), x - 0.2, x + 0.2)
        return h, 2, x, torch.full_like(x, 0.05), 0.0, r(n) * (4.0 / n), r(m) * 0.1, r(m, n) * (4.0 / n)

    def step(a):
        x, lam, _ = mma.unit_box_step(*a, a0=1.0, c=1000.0, raa0=1e-5 / n)
        return x, lam

    inputs = {m: args(m) for m in sizes}
    alone = {m: step(inputs[m]) for m in sizes}
    torch.cuda.synchronize()
    got, errors = {m: [] for m in sizes}, []

    def work(m):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(calls):
                    got[m].append(step(inputs[m]))
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    threads = [threading.Thread(target=work, args=(m,)) for m in sizes]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for m in sizes:
        assert len(got[m]) == calls
        for x, lam in got[m]:
            assert torch.equal(x, alone[m][0]) and torch.equal(lam, alone[m][1])
