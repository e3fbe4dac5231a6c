"""Batched evolutions long enough to run as a captured graph (pairs of iterations replayed, and a single
one where the count is odd): the box window, the Gaussian data term, the TMA z-pass, every launch shape
and per-kernel timing, whose kernels mix programmatic and ordinary launches and event records, bit for
bit against the oracle; and the direct launches of fewer iterations beside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(40, 44, 48), (9, 9, 9), (26, 60, 31)]


def _inputs(seed, dtype=np.uint8):
    rng = np.random.default_rng(seed)
    out = []
    for s in SHAPES:
        phi = np.clip(4.0 * rng.standard_normal(s), -3.0, 3.0).astype(np.float32)
        out.append((rng.integers(0, 256, s).astype(dtype), phi))
    return out


def _batch(ws, inputs, p, iters):
    pairs = [(torch.from_numpy(i).cuda(), torch.from_numpy(q.copy()).cuda()) for i, q in inputs]
    ws.evolve_batched(pairs, p, iters)
    ws.check()
    return [q.cpu().numpy() for _, q in pairs]


def _want(orc, inputs, p, iters):
    prm = orc.params(sigma=p.sigma, dt=p.dt, mu=p.mu, lambda1=p.lambda1, lambda2=p.lambda2, nu=p.nu, eps=p.eps,
                     sigma2=p.sigma2, data_term=1 if p.data_term == "gaussian" else 0)
    return [orc.evolve(q, i.astype(np.float32), prm, iters) for i, q in inputs]


def _same(got, want):
    for g, w in zip(got, want):
        assert np.array_equal(g.view(np.uint32), w.view(np.uint32)), g.shape


PRM = dict(sigma=3.0, dt=0.1, mu=1.0, lambda1=1.0, lambda2=0.5, nu=65.025, eps=1.0)
OPTIONS = {"plain": {}, "box": dict(sigma2=1.0), "gaussian": dict(data_term="gaussian"), "k17": dict(sigma=2.5)}


@pytest.mark.parametrize("iters", [3, 4, 5])
@pytest.mark.parametrize("option", OPTIONS)
def test_graph_and_direct_launches(option, iters, orc, ws_big):
    from rsf_gb300 import Params

    p = Params(**{**PRM, **OPTIONS[option]})
    inputs = _inputs(iters)
    _same(_batch(ws_big, inputs, p, iters), _want(orc, inputs, p, iters))


@pytest.mark.parametrize("sigma", [3.0, 5.0])
def test_tma_z_pass_in_a_graph(sigma, orc, ws_big, monkeypatch):
    from rsf_gb300 import Params

    p = Params(**{**PRM, "sigma": sigma})
    inputs = _inputs(11, np.float32)
    monkeypatch.setenv("RSF_ZPASS", "tma")
    got = _batch(ws_big, inputs, p, 5)
    monkeypatch.delenv("RSF_ZPASS")
    _same(got, _want(orc, inputs, p, 5))


def test_launch_shapes_in_a_graph(orc, ws_big):
    from rsf_gb300 import Params, autotune

    p = Params(**PRM)
    inputs = _inputs(12)
    want = _want(orc, inputs, p, 5)
    try:
        for shape in autotune.LAUNCH_CANDIDATES + ((5, 32, 0), (0, 32, -1)):
            ws_big.set_launch_shape(*shape)
            _same(_batch(ws_big, inputs, p, 5), want)
    finally:
        ws_big.set_launch_shape(0, 0, -1)


@pytest.mark.parametrize("iters", [2, 5])
@pytest.mark.parametrize("option", OPTIONS)
def test_kernel_timing_changes_nothing(option, iters, orc, cuda, rsflib):
    """Event records between the kernels, direct and captured."""
    from rsf_gb300 import Params, Workspace

    p = Params(**{**PRM, **OPTIONS[option]})
    inputs = _inputs(13)
    with Workspace(sum(q.size for _, q in inputs), len(inputs)) as ws:
        ws.set_kernel_timing(True)
        got = _batch(ws, inputs, p, iters)
        times = ws.kernel_times()
        ws.set_kernel_timing(False)
    _same(got, _want(orc, inputs, p, iters))
    assert all(n == iters and ms > 0.0 for ms, n in times.values()), times
