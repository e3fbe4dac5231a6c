"""The tiled signed distance where most voxels are far from the other class (surfaces along and across
the axes, slanted ones, single features, features at the distance where the search by rows ends), bit
for bit against SciPy's exact transform, on shapes whose columns, groups of four rows and rows of x do
not divide evenly; and the time such seeds take beside seeds whose every voxel is near."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SHAPES = [(97, 101, 40), (66, 130, 3), (3, 559, 7), (200, 2, 33), (5, 1407, 2), (561, 6, 5), (64, 63, 31), (1, 1408, 1)]
KINDS = ["z", "y", "x", "zy", "zyx", "steep", "one", "corner", "pairs", "stripes", "sparse", "ball"]


def _inside(kind, shape):
    z, y, x = np.meshgrid(*[np.arange(n) for n in shape], indexing="ij")
    n = sum(shape)
    if kind in ("z", "y", "x"):
        return {"z": z, "y": y, "x": x}[kind] < 1
    if kind == "zy":
        return z + y < (shape[0] + shape[1]) // 3
    if kind == "zyx":
        return z + y + x < n // 2
    if kind == "steep":
        return 10 * z + 3 * y + x < 2 * n
    if kind == "corner":
        return z + y + x < 1
    if kind == "ball":
        return ((z - shape[0] / 2) / shape[0]) ** 2 + ((y - shape[1] / 2) / shape[1]) ** 2 + ((x - shape[2] / 2) / shape[2]) ** 2 < 0.1
    if kind == "stripes":  # gaps of 7 .. 12 rows of either class around the end of the search by rows
        edges = np.cumsum([7, 8, 9, 10, 11, 12, 17, 18, 19, 20, 40] * 60)
        return np.searchsorted(edges, z + y, side="right") % 2 == 0
    m = np.zeros(shape, bool)
    if kind == "one":
        m[tuple(int(v * 0.7) for v in shape)] = True
    elif kind == "pairs":  # single voxels 17 .. 21 rows apart along y and z
        for i, d in enumerate(np.cumsum([3, 17, 18, 19, 20, 21, 33, 34, 35] * 12)):
            m[min(d, shape[0] - 1) if shape[0] > shape[1] else i % shape[0], d % shape[1], i % shape[2]] = True
    else:
        m = np.random.default_rng(n).random(shape) < 3.0 / m.size
        m.flat[m.size // 3] = True
    return m


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("shape", SHAPES)
def test_far_from_the_other_class(shape, kind, ws_big):
    from scipy import ndimage

    inside = _inside(kind, shape)
    for m in (inside, ~inside):
        if m.all() or not m.any():
            want = np.full(shape, sum(shape) if m.all() else -sum(shape))
        else:
            want = np.where(m, ndimage.distance_transform_edt(m), -ndimage.distance_transform_edt(~m))
        got = ws_big.signed_distance(torch.from_numpy(np.where(m, 200, 13).astype(np.uint8)).cuda()).cpu().numpy()
        assert np.array_equal(got, want.astype(np.float32))


def _time(ws, seed, reps=7):
    out = torch.empty(seed.shape, device="cuda")
    times = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        ws.signed_distance(seed, out=out)
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


@pytest.mark.parametrize("axes", ["zy", "zyx"])
def test_time_does_not_follow_the_distance(axes, cuda, rsflib):
    """A volume cut in two by a slanted plane against noise, whose every voxel is near: 3 times its time; 5 (zy) and
    7 times (zyx) where the search went on row by row."""
    from rsf_gb300 import Workspace

    n = 500
    at = torch.arange(n, device="cuda", dtype=torch.int16)
    far = at[:, None, None] + at[None, :, None] + (at[None, None, :] if axes == "zyx" else at[None, None, :] * 0)
    far = (far < n * len(axes) // 2).to(torch.uint8).mul_(200)
    near = (torch.rand((n, n, n), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1)) < 0.5)
    with Workspace(n ** 3) as ws:
        t = [_time(ws, m) for m in (near.to(torch.uint8).mul_(200), far)]
    assert t[1] <= 4.5 * t[0], t
