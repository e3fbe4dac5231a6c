"""delta far out, where eps^2 + phi^2 leaves the packed quotient's range or overflows: bit for bit against
the oracle, with weights that make what is left of delta visible in phi."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("eps", [1.0, 2.0 ** 20])
@pytest.mark.parametrize("phi", [2.0 ** 58, 2.0 ** 60, 2.0 ** 62, 2.0 ** 63.5, 2.0 ** 64, 1e20, 1e30])
def test_delta_of_a_large_level_set(phi, eps, orc, cuda, rsflib):
    from rsf_gb300 import Params, Workspace

    shape = (5, 9, 11)  # no valid blur region: the data factor is lambda1 (I - 1)^2
    p0 = np.full(shape, phi, np.float32)
    img = (1e15 * (1.0 + np.random.default_rng(1).random(shape))).astype(np.float32)
    p = Params(sigma=3.0, dt=1e16, mu=1.0, lambda1=1.0, lambda2=0.0, nu=1.0, eps=eps)
    want = orc.evolve(p0, img, orc.params(sigma=3.0, dt=p.dt, mu=p.mu, lambda1=1.0, lambda2=0.0, nu=p.nu, eps=eps), 1)
    with Workspace(p0.size) as ws:
        t = torch.from_numpy(p0.copy()).cuda()
        ws.evolve(torch.from_numpy(img).cuda(), t, p, 1)
        got = t.cpu().numpy()
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), (got.flat[0], want.flat[0])
