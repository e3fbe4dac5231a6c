"""One volume's evolution, adjoint step and signed distance captured into a caller's graph, whose programmatic
edges and launch parameters then stand in it: replays equal direct calls, also after the workspace has
served another volume in between."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("sigma", [1.0, 3.0])
def test_replays_equal_direct_calls(sigma, cuda, rsflib):
    from rsf_gb300 import Params, Workspace

    shape, other = (30, 41, 52), (50, 33, 37)
    gen = torch.Generator(device="cuda").manual_seed(3)
    img = torch.randint(0, 256, shape, dtype=torch.uint8, device="cuda", generator=gen)
    phi0 = torch.randn(shape, device="cuda", generator=gen).mul_(3.0)
    u = torch.randn(shape, device="cuda", generator=gen)
    img2 = torch.randint(0, 256, other, dtype=torch.uint8, device="cuda", generator=gen)
    phi2 = torch.randn(other, device="cuda", generator=gen)
    p = Params(sigma=sigma, dt=0.1, mu=0.2, lambda1=1e-4, lambda2=2e-4, nu=0.1, eps=1.0)
    with Workspace(80_000) as ws, Workspace(80_000) as direct:
        phi, bar, dist = phi0.clone(), torch.empty_like(phi0), torch.empty_like(phi0)
        grads = torch.zeros(4, dtype=torch.float64, device="cuda")

        def calls(w, phi, bar, dist, grads):
            w.evolve(img, phi, p, 3)
            w.step_adjoint(img, phi, u, p, out=bar, param_grads=grads)
            w.signed_distance(img, threshold=128.0, out=dist)

        stream = torch.cuda.Stream()
        stream.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(stream):
            calls(ws, phi, bar, dist, grads)  # warm-up
        torch.cuda.current_stream().wait_stream(stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            calls(ws, phi, bar, dist, grads)
        want_phi, want = phi0.clone(), [torch.empty_like(phi0), torch.empty_like(phi0),
                                        torch.zeros(4, dtype=torch.float64, device="cuda")]
        phi.copy_(phi0)
        grads.zero_()
        for _ in range(3):
            graph.replay()
            ws.evolve(img2, phi2, p, 2)  # its tables are the workspace's now
            calls(direct, want_phi, *want)
            torch.cuda.synchronize()
            assert torch.equal(phi, want_phi) and torch.equal(bar, want[0]) and torch.equal(dist, want[1])
            assert np.allclose(grads.cpu().numpy(), want[2].cpu().numpy(), rtol=1e-12, atol=0.0)
        ws.check()
