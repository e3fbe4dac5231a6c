"""The launch-shape tuner can keep the workspace's own stencil depth, and times the captured loop."""


class _Workspace:
    def __init__(self):
        self.shape = None

    def set_launch_shape(self, *shape):
        self.shape = shape


def test_the_automatic_depth_is_a_candidate_and_wins_where_it_is_fastest():
    from rsf_gb300 import Params, autotune

    assert {xb for xb, zc, _ in autotune.LAUNCH_CANDIDATES if zc == 0} == {5, 9}
    assert {zt for _, zc, zt in autotune.LAUNCH_CANDIDATES if zc == 0} == {0, 1}
    ws = _Workspace()
    # a small batch: the automatic choice takes shallower blocks than any fixed candidate
    best = autotune.tune_launch_shape(ws, [], Params(sigma=3.0), timer=lambda s: 2.0 + (s[1] or 16) / 64 + s[2])
    assert best.stencil_planes == 0 and ws.shape == (5, 0, 0)


def test_timed_runs_are_long_enough_for_the_graph():
    import re
    from pathlib import Path

    from rsf_gb300 import autotune

    capi = Path(autotune.__file__).resolve().parents[1] / "csrc" / "rsf_capi.cu"
    assert autotune.GRAPH_FROM == int(re.search(r"kGraphFrom = (\d+);", capi.read_text()).group(1))
