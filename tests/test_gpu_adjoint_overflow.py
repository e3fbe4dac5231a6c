"""Where dL/dphi' overflows FP32 in one voxel: only the voxels whose derivative reads it may become
non-finite, and the workspace reports it.  The reach is the chain's own: out(i) gathers w at the axis
neighbours of i (and at i itself on a face), w(i) gathers kappa_bar and Lap_bar, u dt (nu delta - mu)
and u dt mu, at the axis neighbours of i (and at i itself on a face)."""
import numpy as np
import pytest

from test_gpu_adjoint import _params

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPE = (9, 8, 10)  # 11 taps: no valid blur region, so the blurs carry nothing further


def _readers(voxels, shape, boundary):
    """Voxels whose transposed difference along some axis reads one of `voxels`."""
    L, H, W = shape
    n = L * H * W
    out = set()
    for z, y, x in voxels:
        i = (z * H + y) * W + x
        # D_x f(i) = (f(r) - f(l)) / 2 writes its adjoint to r and l
        r = i + 1 if x + 1 < W else i
        l = i - 1 if x > 0 else (max(i - 1, 0) if boundary == "reference" else i)
        out |= {r, l}
        out |= {i + H * W * min(1, L - 1 - z), i - H * W * min(1, z), i + W * min(1, H - 1 - y), i - W * min(1, y)}
    assert all(0 <= i < n for i in out)
    return {(i // (H * W), i // W % H, i % W) for i in out}


@pytest.mark.parametrize("boundary", ["reference", "clamp"])
@pytest.mark.parametrize("at", [(4, 4, 5), (0, 0, 0), (8, 7, 9), (4, 0, 5), (3, 4, 9), (5, 3, 0)])
def test_overflow_stays_where_the_chain_carries_it(at, boundary, ws_big):
    from rsf_gb300 import RsfError

    rng = np.random.default_rng(3)
    phi = rng.standard_normal(SHAPE).astype(np.float32)
    img = rng.random(SHAPE).astype(np.float32)
    u = np.zeros(SHAPE, np.float32)
    u[at] = 3e38
    p = _params(sigma=1.5, boundary=boundary, dt=10.0, mu=1.0)  # u dt overflows
    got = ws_big.step_adjoint(torch.from_numpy(img).cuda(), torch.from_numpy(phi).cuda(), torch.from_numpy(u).cuda(),
                              p).cpu().numpy()
    with pytest.raises(RsfError, match="overflow"):
        ws_big.check()
    w = _readers({at}, SHAPE, boundary)
    may = _readers(w, SHAPE, boundary) | {at}
    bad = {tuple(int(v) for v in i) for i in np.argwhere(~np.isfinite(got))}
    assert bad and bad <= may, sorted(bad - may)
