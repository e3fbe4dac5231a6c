"""Choosing the launch shape costs a call no more for a long thin volume than for a small one."""
import time

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _prepare_us(ws, pairs, p):
    """A call of no iterations: it lays the batch out, chooses the shapes and uploads the tables."""
    times = []
    for _ in range(20):
        torch.cuda.synchronize()
        t = time.perf_counter()
        ws.evolve_batched(pairs, p, 0)
        times.append(time.perf_counter() - t)
    return 1e6 * min(times)


def test_long_thin_volumes_without_a_valid_region(cuda, rsflib):
    from rsf_gb300 import Params, Workspace

    p = Params(sigma=3.0)

    def pairs(*shapes):
        return [(torch.zeros(s, dtype=torch.uint8, device="cuda"), torch.zeros(s, device="cuda")) for s in shapes]

    n = 1 << 20
    with Workspace(3 * 4 * n, 3) as ws:
        base = _prepare_us(ws, pairs((24, 24, 24)), p)
        for shapes in (((n, 2, 2),), ((2, n, 2),), ((24, 24, 24), (n, 2, 2), (2, n, 2))):
            assert _prepare_us(ws, pairs(*shapes), p) <= base + 200.0, shapes
