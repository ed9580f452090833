"""Calls whose sweeps run on chip inside a caller's CUDA graph: the LSRTM
operator from its first call on (it allocates nothing in a call), modelling
once its buffers are there; replays read current data."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model
from tests.gpu_helpers import t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact", [False, True])
def test_lsrtm_calls_captured_from_the_first(cuda, exact):
    import swfwi_b200 as S
    torch = cuda
    nx, nz, nt, ng, ns = 120, 80, 150, 100, 3
    rng = np.random.default_rng(5)
    vel = t(torch, rng.uniform(1500, 2500, (nx, nz)).astype(np.float32))
    mod = t(torch, rng.standard_normal((nx, nz)).astype(np.float32))
    out = []
    for captured in (False, True):
        op = S.Prtm2d(vel, dz=10.0, dx=10.0, dt=0.001, amp=1.0, fm=25.0, nb=15, nt=nt, ns=ns, ng=ng, sxbeg=5, szbeg=2,
                      jsx=50, jsz=0, gxbeg=0, gzbeg=2, jgx=1, jgz=0, arith=S.ARITH_FAST)
        op.set_adjoint(S.PRTM_ADJ_EXACT if exact else S.PRTM_ADJ_REFERENCE)
        x, d, m = mod.clone(), torch.zeros((ns, ng, nt), device="cuda"), torch.zeros((nx, nz), device="cuda")

        def calls():
            op.lop(False, False, x, d)
            op.lop(True, False, m, d)

        if captured:
            g = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(g):
                calls()
        for scale in (1.0, 2.0):
            x.copy_(mod * scale)
            g.replay() if captured else calls()
            torch.cuda.synchronize()
            out += [d.cpu(), m.cpu()]
        op.check()
        op.close()
    for a, b in zip(out[:4], out[4:]):
        assert float(a.abs().max()) > 0 and torch.equal(a, b)


def test_modelling_captured(cuda):
    import swfwi_b200 as S
    torch = cuda
    s = Survey(nz=90, nx=200, dx=25.0, dt=0.002, nt=200, fm=10.0, nb=20, ns=2, sxbeg=10, jsx=90, ng=200)
    m = S.Damp4t10d.from_survey(s, arith=S.ARITH_FAST)
    vel = t(torch, m.expandDomain(layered_model(s.nx, s.nz, seed=3)))
    m.bindVelocity(vel)
    wlt = t(torch, S.ricker_wavelet(s.nt, s.fm, s.dt))
    want, got = torch.zeros((2, s.nt, s.ng), device="cuda")
    m.FwiForwardModeling(wlt, want, 1)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        m.set_stream()
        m.FwiForwardModeling(wlt, got, 1)
    got.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
