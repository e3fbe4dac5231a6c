"""Columns cut along y, with a shorter last piece, for each compiled tap count (a volume this small leaves
the SMs short of blocks), and tap counts at the ends of the run-time range: bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run(orc, shape, sigma, dtype, boundary="reference"):
    from rsf_gb300 import Params, Workspace

    rng = np.random.default_rng(sum(shape))
    phi = np.clip(4.0 * rng.standard_normal(shape), -3.0, 3.0).astype(np.float32)
    img = rng.integers(0, 256, shape).astype(dtype)
    p = Params(sigma=sigma, dt=0.1, mu=1.0, lambda1=1.0, lambda2=0.5, nu=65.025, eps=0.2, boundary=boundary)
    want = orc.evolve(phi, img.astype(np.float32),
                      orc.params(sigma=sigma, dt=0.1, mu=1.0, lambda1=1.0, lambda2=0.5, nu=65.025, eps=0.2,
                                 boundary=0 if boundary == "reference" else 1), 2)
    with Workspace(phi.size) as ws:
        t = torch.from_numpy(phi.copy()).cuda()
        ws.evolve(torch.from_numpy(img).cuda(), t, p, 2)
        got = t.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("sigma,k", [(1.5, 11), (2.0, 15), (3.0, 21), (4.0, 29), (5.0, 35)])
@pytest.mark.parametrize("more", [(0, 0), (1, 2), (3, 29)])  # beyond 3 k valid rows, and along z
def test_columns_cut_along_y(sigma, k, more, orc, cuda, rsflib):
    assert len(orc.taps(sigma)) == k
    _run(orc, (k + more[1], 4 * k - 1 + more[0], k + 2), sigma, np.uint8 if more[0] else np.float32)


@pytest.mark.parametrize("sigma", [1.2, 2.2, 18.0])
@pytest.mark.parametrize("extra", [(0, 0, 0), (1, 17, 10)])
def test_run_time_tap_counts_between_and_beyond(sigma, extra, orc, cuda, rsflib):
    k = len(orc.taps(sigma))
    _run(orc, tuple(k + e for e in extra), sigma, np.uint8, "clamp" if extra[0] else "reference")
