"""Step timing observes: with it on, the same kernels run and give the same
bits as without (a FAST batch gradient sums its images in another order when it
streams), and a sweep in one launch counts the work of its steps.  The launch
shape tuner, which goes by that timing, sees the sweeps that its result will
run.  Beside them the streaming kernels' timing inside captured loops."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model
from tests.gpu_helpers import t

pytestmark = pytest.mark.gpu


def case(torch, ns=3, nt=240, tuning=None, **kw):
    import swfwi_b200 as S
    s = Survey(nz=80, nx=200, dx=25.0, dt=0.002, nt=nt, fm=10.0, nb=20, ns=ns, sxbeg=10, jsx=60, ng=200)
    m = S.Damp4t10d.from_survey(s, arith=S.ARITH_FAST)
    if tuning:
        m.set_tuning(*tuning)
    vel = t(torch, m.expandDomain(layered_model(s.nx, s.nz, seed=3)))
    m.bindVelocity(vel)
    return s, m, vel, t(torch, S.ricker_wavelet(s.nt, s.fm, s.dt))


def gradient(torch, s, m, vel, wlt):
    d = torch.randn((s.ns, s.nt, s.ng), generator=torch.Generator().manual_seed(1)).cuda()
    grad = torch.zeros_like(vel)
    obj = m.gradient_batch(wlt, d, np.arange(s.ns, dtype=np.int32), grad)
    return grad.cpu(), obj


@pytest.mark.parametrize("period", [1, 7, 1 << 30])
def test_timing_changes_neither_kernels_nor_bits(cuda, period):
    import swfwi_b200 as S
    torch = cuda
    s, m, vel, wlt = case(torch)
    gradient(torch, s, m, vel, wlt)              # the first call also forms 1/vt
    S.stats_reset()
    want = gradient(torch, s, m, vel, wlt)
    launches = S.stats_read()["kernel_launches"]
    assert launches < s.nt                       # sweeps in one launch each
    S.stats_enable_step_timing(period)
    try:
        S.stats_reset()
        got = gradient(torch, s, m, vel, wlt)
        st = S.stats_read()
    finally:
        S.stats_enable_step_timing(False)
    assert torch.equal(got[0], want[0])
    np.testing.assert_array_equal(got[1], want[1])
    assert st["kernel_launches"] == launches
    # forward steps, and two propagations a step back while t > 0.3
    steps = s.nt + 2 * sum(1 for it in range(s.nt) if float(np.float32(s.dt) * np.float32(it)) > 0.3)
    points = (s.nxpad - 12) * (s.nzpad - 12) * s.ns
    assert st["step_launches"] == steps
    assert st["step_point_updates"] == float(points) * steps
    assert st["step_bytes"] == float(points) * 12 * steps + points / s.ns * 4.0 * steps
    assert st["step_timed_launches"] == -(-steps // period)
    assert st["step_ms"] > 0


def test_tuner_sees_the_sweeps_it_chooses(cuda):
    import swfwi_b200 as S
    from swfwi_b200 import autotune
    torch = cuda
    s, m, vel, wlt = case(torch, ns=1)
    cfg, table = autotune.tune(s, vel.cpu().numpy(), S.ARITH_FAST)
    assert cfg["kernel"] == 6 and cfg["rows_per_cta"] == 0, table[:3]
    autotune.apply(m, cfg)
    d = torch.zeros((1, s.nt, s.ng), device="cuda")
    S.stats_reset()
    m.forward_batch(wlt, d, np.zeros(1, np.int32))
    assert S.stats_read()["kernel_launches"] < s.nt


def test_timing_inside_captured_streaming_loops(cuda):
    """The loops that stream (an explicit task length keeps them): replayed
    graphs count and time what direct launches do, with the same bits."""
    import swfwi_b200 as S
    torch = cuda
    stats, outs = {}, {}
    for graphs in (0, 2):
        s, m, vel, wlt = case(torch, tuning=(6, 120, 40, 3))
        m.set_graphs(graphs)
        S.stats_enable_step_timing(4)
        try:
            for _ in range(2):
                gradient(torch, s, m, vel, wlt)
            S.stats_reset()
            for _ in range(3):
                outs[graphs] = gradient(torch, s, m, vel, wlt)
            stats[graphs] = S.stats_read()
        finally:
            S.stats_enable_step_timing(False)
    assert torch.equal(outs[0][0], outs[2][0])
    a, b = stats[0], stats[2]
    assert a["kernel_launches"] == b["kernel_launches"] > 3 * s.nt
    assert a["step_launches"] == b["step_launches"] and a["step_point_updates"] == b["step_point_updates"]
    assert abs(a["step_timed_launches"] - b["step_timed_launches"]) <= 6      # each loop counts from its start
    assert a["step_ms"] > 0 and b["step_ms"] > 0
