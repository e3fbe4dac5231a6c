"""RSF_ARITH_REFERENCE on the GPU against the stored outputs of the reference's own kernels
(tests/golden/reference_kernels_*.npz): whole iterations, bit for bit, where test_reference_kernels.py
needs the reference's sources."""
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
GOLDEN = sorted((Path(__file__).resolve().parent / "golden").glob("reference_kernels_*.npz"))


@pytest.mark.parametrize("path", GOLDEN, ids=lambda p: p.stem)
@pytest.mark.parametrize("iters", [1, 3])
def test_whole_iterations(path, iters, ws_big):
    from rsf_gb300 import Params

    g = np.load(path)
    p = Params(sigma=float(g["sigma"]), dt=0.1, mu=1.0, lambda1=1.0, lambda2=1.0, nu=65.025, eps=0.2, arith="reference")
    t = torch.from_numpy(g["phi0"].astype(np.float32)).cuda()
    ws_big.evolve(torch.from_numpy(np.ascontiguousarray(g["image"])).cuda(), t, p, iters)
    ws_big.check()
    got, want = t.cpu().numpy(), g[f"phi{iters}"]
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)), float(np.abs(got - want).max())
