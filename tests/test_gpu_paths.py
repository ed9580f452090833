"""Which form a sweep takes.  The shapes that other tests use for the on-chip
sweeps do run on chip (a launch a sweep, not a launch a step), and the
streaming kernels' captured loops, which small surveys take only with an
explicit task length, replay with the bits of direct launches and read current
data."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model
from tests.gpu_helpers import t

pytestmark = pytest.mark.gpu

STREAM = (6, 120, 40, 3)      # an explicit task length


def method(torch, s, arith, streaming=False):
    import swfwi_b200 as S
    m = S.Damp4t10d.from_survey(s, arith=arith)
    if streaming:
        m.set_tuning(*STREAM)
    vel = t(torch, m.expandDomain(layered_model(s.nx, s.nz, seed=3)))
    m.bindVelocity(vel)
    return m, vel, t(torch, S.ricker_wavelet(s.nt, s.fm, s.dt))


@pytest.mark.parametrize("streaming", [False, True])
@pytest.mark.parametrize("arith,nx,nz,ns", [
    (0, 31, 20, 2), (1, 31, 20, 2), (0, 64, 41, 3), (1, 64, 41, 3), (0, 50, 42, 5), (1, 50, 42, 5), (0, 97, 55, 26),
    (1, 97, 55, 26), (0, 400, 60, 1), (1, 400, 60, 1), (0, 130, 301, 17), (1, 130, 301, 17), (0, 14, 20, 1),
    (1, 160, 33, 1), (1, 700, 64, 1), (0, 860, 30, 1), (0, 461, 101, 1), (1, 480, 560, 1), (0, 300, 170, 30),
    (1, 300, 170, 30),
])
def test_form_of_the_sweeps(cuda, arith, nx, nz, ns, streaming):
    import swfwi_b200 as S
    torch = cuda
    s = Survey(nz=nz, nx=nx, dx=25.0, dt=0.002, nt=181, fm=10.0, nb=10, ns=ns, sxbeg=1, jsx=max(1, (nx - 2) // ns),
               ng=nx, szbeg=2, gzbeg=3)
    m, vel, wlt = method(torch, s, arith, streaming)
    m.set_graphs(False)
    ids = np.arange(ns, dtype=np.int32)
    d = torch.zeros((ns, s.nt, s.ng), device="cuda")
    enc = wlt[:, None].repeat(1, ns).contiguous()
    grad = torch.zeros_like(vel)
    for call in (lambda: m.forward_batch(wlt, d, ids), lambda: m.calgradient_ess(enc, d[0], grad),
                 lambda: m.gradient_batch(wlt, d, ids, grad)):
        torch.cuda.synchronize()
        S.stats_reset()
        call()
        launches = S.stats_read()["kernel_launches"]
        assert launches >= s.nt if streaming else launches <= 12, launches


def test_streaming_loops_replay_current_data(cuda):
    """Repeated calls of the streaming loops are graphs from the second on:
    the bits of direct launches, other buffers, new contents."""
    import swfwi_b200 as S
    torch = cuda
    s = Survey(nz=100, nx=200, dx=25.0, dt=0.002, nt=200, fm=10.0, nb=20, ns=3, sxbeg=10, jsx=60, ng=200)
    m, vel, wlt = method(torch, s, S.ARITH_FAST, streaming=True)
    ids = np.arange(s.ns, dtype=np.int32)
    obs = torch.randn((s.ns, s.nt, s.ng), generator=torch.Generator().manual_seed(1)).cuda()
    want, grad = torch.zeros((s.ns, s.nt, s.ng), device="cuda"), torch.zeros_like(vel)
    m.set_graphs(False)
    m.forward_batch(wlt, want, ids)
    m.gradient_batch(wlt, obs, ids, grad)
    m.set_graphs(True)
    got = [torch.zeros_like(want) for _ in range(2)]
    again = torch.zeros_like(grad)
    for _ in range(3):
        for d in got:
            d.zero_()
            m.forward_batch(wlt, d, ids)
            assert torch.equal(d, want)
        m.gradient_batch(wlt, obs, ids, again)
        assert torch.equal(again, grad)
    wlt.mul_(2.0)
    m.forward_batch(wlt, got[0], ids)
    # doubling is exact for normal floats; subnormals round on a fixed grid
    assert float((got[0] - want * 2).norm() / (want * 2).norm()) < 1e-6
