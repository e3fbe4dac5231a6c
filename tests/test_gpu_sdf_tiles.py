"""The tiled signed distance at the edges of its tiles (32 columns, groups of
four rows, 24 rows searched one by one, blocks of 16 skipped beyond, 256 or 512
threads) against SciPy's exact transform, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# shape (L, H, W), share of inside voxels (0: a single one)
CASES = [((1, 1, 70), 0.3), ((3, 1, 33), 0.2), ((5, 7, 31), 0.5), ((4, 33, 65), 0.05), ((130, 3, 32), 0.0),
         ((2, 561, 34), 0.001), ((559, 2, 5), 0.0), ((40, 90, 64), 0.0), ((60, 61, 62), 0.0005), ((9, 1408, 3), 0.002),
         ((3, 2, 1409), 0.01), ((37, 53, 41), 0.9995)]


@pytest.mark.parametrize("dtype", ["u8", "f32"])
@pytest.mark.parametrize("shape,share", CASES)
def test_tiled_signed_distance_matches_scipy(shape, share, dtype, ws_big):
    from scipy import ndimage

    rng = np.random.default_rng(sum(shape))
    inside = rng.random(shape) < share
    if share == 0.0:
        inside[tuple(int(n * 0.3) for n in shape)] = True
    if not inside.any():
        inside.flat[0] = True
    want = np.where(inside, ndimage.distance_transform_edt(inside), -ndimage.distance_transform_edt(~inside))
    seed = np.where(inside, 200, 13).astype(np.uint8 if dtype == "u8" else np.float32)
    got = ws_big.signed_distance(torch.from_numpy(seed).cuda()).cpu().numpy()
    assert np.array_equal(got, want.astype(np.float32))
