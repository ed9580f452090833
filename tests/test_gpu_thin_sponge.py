"""Surveys whose sponge is thinner than the stencil's reach: the boundary
strips then cover rows and depths outside the computing zone.  Every cell of a
strip has to be saved, also those, or the backward sweep restores what the
buffer held before: here the strips of a larger model."""
import pytest

from swfwi_b200.survey import Survey, layered_model

pytestmark = pytest.mark.gpu


def gradients(torch, s, arith, streaming):
    import swfwi_b200 as S
    m = S.Damp4t10d.from_survey(s.scaled(nx=s.nx + 20, nz=s.nz + 12), arith=arith)
    if streaming:   # an explicit task length keeps the streaming kernels
        m.set_tuning(6, 120, 40, 3)
    wlt = torch.from_numpy(S.ricker_wavelet(s.nt, s.fm, s.dt)).cuda()
    res = torch.randn((s.nt, s.ng), generator=torch.Generator().manual_seed(1)).cuda()
    out = []
    for nx, nz in ((s.nx + 20, s.nz + 12), (s.nx, s.nz)):
        m.setModelSize(nx, nz)
        vel = torch.from_numpy(m.expandDomain(layered_model(nx, nz, seed=3))).cuda()
        m.bindVelocity(vel)
        for shot in range(s.ns):
            grad = torch.full_like(vel, 0.5)
            m.calgradient_fwi(wlt, res, grad, shot)
            out.append(grad.cpu())
    return out


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("nb", [0, 1, 3, 5, 6])
def test_thin_sponges_match_the_streaming_kernels(cuda, arith, nb):
    s = Survey(nz=40, nx=70, dx=25.0, dt=0.002, nt=601, fm=10.0, nb=nb, ns=2, sxbeg=3, jsx=41, ng=70, szbeg=2, gzbeg=3)
    for a, b in zip(gradients(cuda, s, arith, False), gradients(cuda, s, arith, True)):
        assert cuda.equal(a, b)
