"""The blurred fields and local fits of the specialised tap counts (21, 29, 35)
at the edges of their tiles: valid regions of one voxel and of ragged rows,
columns cut along z, and images at the ends of the packed quotient's range.
Bit for bit against the oracle (a NaN's payload is the platform's own)."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _run(orc, shape, p, phi, img, iters):
    from rsf_gb300 import Workspace

    want = orc.evolve(phi, img.astype(np.float32),
                      orc.params(sigma=p.sigma, dt=p.dt, mu=p.mu, lambda1=p.lambda1, lambda2=p.lambda2, nu=p.nu,
                                 eps=p.eps), iters)
    with Workspace(phi.size) as ws:
        t = torch.from_numpy(phi.copy()).cuda()
        ws.evolve(torch.from_numpy(img).cuda(), t, p, iters)
        got = t.cpu().numpy()
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), f"{int((~same).sum())} voxels differ"


@pytest.mark.parametrize("sigma,k", [(3.0, 21), (4.0, 29), (5.0, 35)])
@pytest.mark.parametrize("extra", [(0, 0, 0), (1, 2, 3), (2, 0, 40), (75, 3, 9), (130, 1, 1)])
def test_valid_region_edges(sigma, k, extra, orc, cuda, rsflib):
    from rsf_gb300 import Params

    shape = tuple(k + e for e in extra)
    rng = np.random.default_rng(sum(shape))
    phi = np.clip(4.0 * rng.standard_normal(shape), -3.0, 3.0).astype(np.float32)
    img = rng.integers(0, 256, shape).astype(np.uint8 if extra[0] % 2 else np.float32)
    img[:, : k // 2] = 0  # a black background: blurs of exactly 0
    _run(orc, shape, Params(sigma=sigma, dt=0.1, mu=1.0, lambda1=1.0, lambda2=1.0, nu=65.025, eps=1.0), phi, img, 2)


@pytest.mark.parametrize("scale", [0.0, 1e-42, 1e-33, 1e-25, -1.0, 1e18, 3e38])
@pytest.mark.parametrize("eps,spread", [(1.0, 3.0), (0.2, 1e9), (1e-7, 3.0), (3e6, 1e20)])
def test_value_ranges(scale, eps, spread, orc, cuda, rsflib):
    from rsf_gb300 import Params

    shape = (23, 24, 25)
    rng = np.random.default_rng(5)
    phi = (spread * rng.standard_normal(shape)).astype(np.float32)
    with np.errstate(over="ignore"):
        img = (scale * rng.random(shape)).astype(np.float32)
    _run(orc, shape, Params(sigma=3.0, dt=0.1, mu=0.1, lambda1=1e-3, lambda2=2e-3, nu=0.1, eps=eps), phi, img, 1)


@pytest.mark.parametrize("sigma", [0.75, 1.0, 1.5, 2.0, 2.5, 6.0, 10.0])
@pytest.mark.parametrize("extra", [(0, 0, 0), (1, 2, 3), (8, 16, 5), (9, 33, 41)])
def test_run_time_tap_counts(sigma, extra, orc, cuda, rsflib):
    """Tap counts without kernels of their own: chunks of 5 or 9 (x), 16 (y) and 8 (z) taps and outputs."""
    from rsf_gb300 import Params

    k = len(orc.taps(sigma))
    shape = tuple(k + e for e in extra)
    rng = np.random.default_rng(k)
    phi = np.clip(4.0 * rng.standard_normal(shape), -3.0, 3.0).astype(np.float32)
    img = rng.integers(0, 256, shape).astype(np.uint8 if extra[0] % 2 else np.float32)
    _run(orc, shape, Params(sigma=sigma, dt=0.1, mu=1.0, lambda1=1.0, lambda2=0.5, nu=65.025, eps=0.2), phi, img, 2)


@pytest.mark.parametrize("sigma2", [1.0, 2.0, 3.0])
@pytest.mark.parametrize("kind", ["u8", "black", "f32", "tiny", "huge", "mixed"])
def test_box_term_in_float_pairs(sigma2, kind, orc, cuda, rsflib):
    """The box sum's float pairs against the double sequence: integers, zeros (fits of exactly 0), fractions,
    and values that leave the pairs' range."""
    from rsf_gb300 import Params, Workspace

    shape = (19, 23, 31)
    rng = np.random.default_rng(7)
    phi = np.clip(4.0 * rng.standard_normal(shape), -3.0, 3.0).astype(np.float32)
    img = {"u8": rng.integers(0, 256, shape).astype(np.uint8), "black": np.zeros(shape, np.uint8),
           "f32": (200.0 * rng.random(shape)).astype(np.float32), "tiny": (1e-25 * rng.random(shape)).astype(np.float32),
           "huge": (1e15 * rng.random(shape)).astype(np.float32),
           "mixed": (10.0 ** rng.uniform(-12, 4, shape)).astype(np.float32)}[kind]
    p = Params(sigma=1.0, dt=0.1, mu=0.5, lambda1=1e-3, lambda2=2e-3, nu=1.0, eps=1.0, sigma2=sigma2)
    want = orc.evolve(phi, img.astype(np.float32),
                      orc.params(sigma=1.0, dt=p.dt, mu=p.mu, lambda1=p.lambda1, lambda2=p.lambda2, nu=p.nu, eps=p.eps,
                                 sigma2=sigma2), 2)
    with Workspace(phi.size) as ws:
        t = torch.from_numpy(phi.copy()).cuda()
        ws.evolve(torch.from_numpy(img).cuda(), t, p, 2)
        got = t.cpu().numpy()
    same = (got.view(np.uint32) == want.view(np.uint32)) | (np.isnan(got) & np.isnan(want))
    assert same.all(), f"{int((~same).sum())} voxels differ"


@pytest.mark.parametrize("iters", [2, 5])
def test_batched_is_refused_on_a_capturing_stream(iters, cuda, rsflib):
    """With and without a graph of its own (a refused capture spoils the process's next call: a child process)."""
    code = f"""
import os, torch
from rsf_gb300 import Params, RsfError, Workspace
img, phi = torch.zeros((24, 24, 24), dtype=torch.uint8, device="cuda"), torch.randn((24, 24, 24), device="cuda")
ws = Workspace(phi.numel())
ws.evolve_batched([(img, phi)], Params(sigma=1.0), {iters})
torch.cuda.synchronize()
answer = "accepted"
try:
    with torch.cuda.graph(torch.cuda.CUDAGraph()):
        try:
            ws.evolve_batched([(img, phi)], Params(sigma=1.0), {iters})
        except RsfError:
            answer = "refused"
except RuntimeError:
    pass
print(answer, flush=True)
os._exit(0)
"""
    pkg = Path(__file__).resolve().parent.parent / "paper-rsf-vesselseg_gb300"
    r = subprocess.run([sys.executable, "-c", code], cwd=str(pkg), capture_output=True, text=True, timeout=300)
    assert r.stdout.split() == ["refused"], r.stdout + r.stderr


@pytest.mark.parametrize("sigma,k", [(1.5, 11), (2.0, 15)])
@pytest.mark.parametrize("extra", [(0, 0, 0), (1, 2, 3), (2, 0, 40), (75, 3, 9), (130, 1, 1), (14, 15, 150)])
def test_valid_region_edges_of_short_taps(sigma, k, extra, orc, cuda, rsflib):
    """The compiled tap counts below 21, as test_valid_region_edges."""
    assert len(orc.taps(sigma)) == k
    test_valid_region_edges(sigma, k, extra, orc, cuda, rsflib)


@pytest.mark.parametrize("shape", [(15, 15, 15), (16, 18, 20), (34, 31, 45)])
def test_step_adjoint_of_15_taps(shape, orc, cuda, rsflib):
    """Against float64 autograd, at the tolerance of the other tap counts (test_gpu_adjoint.py)."""
    from test_adjoint_ref_cpu import smooth_case
    from test_gpu_adjoint import _params, _rel, _vjp_fp64
    from rsf_gb300 import Workspace

    img, phi, _ = smooth_case(shape)
    p = _params(sigma=2.0, lambda2=0.7)
    u = np.random.default_rng(sum(shape)).standard_normal(shape).astype(np.float32)
    g = torch.zeros(4, dtype=torch.float64, device="cuda")
    with Workspace(phi.size) as ws:
        got = ws.step_adjoint(torch.from_numpy(img).cuda(), torch.from_numpy(phi).cuda(), torch.from_numpy(u).cuda(), p,
                              param_grads=g).cpu().numpy()
    want, want_p = _vjp_fp64(orc, phi, img, u, p, "reference")
    assert _rel(got, want) <= 1e-4
    gp = g.cpu().numpy()
    for k in range(4):
        assert abs(gp[k] - want_p[k]) <= 1e-4 * max(abs(want_p[k]), 1e-3 * np.abs(want_p).max()), k
