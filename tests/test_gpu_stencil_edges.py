"""The stencil / update kernel at the edges of its tiles (30 columns x 14 rows
of row pairs, planes streamed in groups of three through a ring of six) and at
the ends of its packed arithmetic's ranges, bit for bit against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (L, H, W): one voxel below, at and above a tile's extents, and the smallest volumes
SHAPES = [(2, 2, 2), (3, 13, 29), (4, 14, 30), (5, 15, 31), (6, 16, 32), (7, 17, 33), (8, 28, 60), (9, 29, 61),
          (13, 30, 62), (27, 31, 35), (140, 9, 12)]


def _run(orc, ws, shape, p, phi, img, iters=3):
    want = orc.evolve(phi, img.astype(np.float32),
                      orc.params(sigma=p.sigma, dt=p.dt, mu=p.mu, lambda1=p.lambda1, lambda2=p.lambda2, nu=p.nu,
                                 eps=p.eps, boundary=0 if p.boundary == "reference" else 1), iters)
    t = torch.from_numpy(phi.copy()).cuda()
    ws.evolve(torch.from_numpy(img).cuda(), t, p, iters)
    got = t.cpu().numpy()
    # a NaN's payload is the platform's own: the oracle's and the GPU's count as equal
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), f"{int((~same).sum())} voxels differ"


@pytest.mark.parametrize("boundary", ["reference", "clamp"])
@pytest.mark.parametrize("shape", SHAPES)
def test_tile_edges(shape, boundary, orc, ws_big):
    from rsf_gb300 import Params

    rng = np.random.default_rng(sum(shape))
    phi = np.clip(4.0 * rng.standard_normal(shape), -3.0, 3.0).astype(np.float32)
    img = rng.integers(0, 256, shape).astype(np.uint8 if shape[0] % 2 else np.float32)
    _run(orc, ws_big, shape, Params(sigma=1.0, dt=0.1, mu=1.0, lambda1=1.0, lambda2=1.0, nu=65.025, eps=1.0,
                                    boundary=boundary), phi, img)


# scale of phi: gradients whose squares are 0, denormal, below and above 2^-100, and delta's far tail
@pytest.mark.parametrize("scale", [0.0, 1e-30, 1e-21, 1e-16, 3e-15, 1e-6, 1e12, 1e18])
@pytest.mark.parametrize("eps", [1.0, 0.2, 1e-8])
def test_value_ranges(scale, eps, orc, cuda, rsflib):
    from rsf_gb300 import Params, Workspace

    shape = (11, 18, 34)
    rng = np.random.default_rng(3)
    phi = (scale * rng.standard_normal(shape)).astype(np.float32)
    phi[:, 6:9, 10:20] = 0.0  # flat
    img = rng.integers(0, 256, shape).astype(np.uint8)
    with Workspace(phi.size) as ws:  # its own: some of these leave the non-finite flag set
        _run(orc, ws, shape, Params(sigma=1.0, dt=0.1, mu=0.1, lambda1=1e-3, lambda2=2e-3, nu=0.1, eps=eps), phi, img, 2)
