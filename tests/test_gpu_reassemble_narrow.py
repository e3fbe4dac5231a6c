"""Stitching volumes of few columns, where a block takes several rows side by side: widths around the
row lengths that the launch chooses, against the CPU restatement (as test_gpu_reassemble.py), and the
time per voxel beside a wide volume's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("width", [1, 2, 3, 5, 9, 15, 17, 31, 33, 47, 63, 65, 70, 97, 129])
def test_narrow_volumes(width, ws_big):
    from oracle import reassembly
    from rsf_gb300 import tiling

    shape = (11, 23, width)
    tiles = tiling.plan(shape, (5, 9, max(width // 2, 1)), 2)
    rng = np.random.default_rng(width)
    parts = [rng.standard_normal(t.shape).astype(np.float32) * 5 for t in tiles]
    dparts = [torch.from_numpy(p).cuda() for p in parts]
    got = tiling.reassemble_device(ws_big, tiles, dparts, shape, "core").cpu().numpy()
    assert np.array_equal(got, reassembly.reassemble_cores(shape, tiles, parts))
    got = tiling.reassemble_device(ws_big, tiles, dparts, shape, "blend").cpu().numpy()
    want = reassembly.blend_grid(shape, tiles, parts)
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("mode", ["core", "blend"])
@pytest.mark.parametrize("width", [3, 17])
def test_narrow_volumes_keep_the_time_per_voxel(mode, width, cuda, rsflib):
    """With a block of one row of 64 threads a width of 3 took 25 times the wide volume's time per voxel."""
    from rsf_gb300 import Workspace, tiling

    per_voxel = []
    for shape in ((2000, 2000, width), (300, 300, 320)):
        tiles = tiling.plan(shape, 500, 8)
        parts = [torch.zeros(t.shape, device="cuda") for t in tiles]
        out = torch.empty(shape, device="cuda")
        with Workspace(8, len(tiles)) as ws:
            times = []
            for _ in range(7):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record()
                tiling.reassemble_device(ws, tiles, parts, shape, mode, out=out)
                b.record()
                b.synchronize()
                times.append(a.elapsed_time(b))
        per_voxel.append(min(times) / out.numel())
    assert per_voxel[0] <= 6.0 * per_voxel[1], per_voxel
