"""Sources in the six rows or depths around the model that the boundary strips
save: the backward sweep takes the source out of the field, images it, and then
restores the strip over it, in this order.

A FAST batch gradient of the streaming kernels, which restores the strips in
the launch that subtracts the sources where the two are disjoint, against the
reference arithmetic, which has a launch for each."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model
from tests.conftest import rel_l2
from tests.test_gpu_resident import sweep

pytestmark = pytest.mark.gpu

PLACES = ["left", "right", "below", "corner", "down the edge"]


def survey(where, nb=10):
    at = {"left": dict(sxbeg=-3, jsx=1, szbeg=5), "right": dict(sxbeg=70, jsx=2, szbeg=5),
          "below": dict(sxbeg=10, jsx=17, szbeg=42), "corner": dict(sxbeg=-6, jsx=5, szbeg=39),
          "down the edge": dict(sxbeg=-1, jsx=0, szbeg=30, jsz=7)}[where]
    return Survey(nz=40, nx=70, dx=25.0, dt=0.002, nt=201, fm=10.0, nb=nb, ns=3, ng=70, gzbeg=3, **at)


@pytest.mark.parametrize("shots", [1, 3])
@pytest.mark.parametrize("where", PLACES)
def test_streamed_batch_gradient(cuda, where, shots):
    import swfwi_b200 as S
    torch = cuda
    s = survey(where)
    wlt = torch.from_numpy(S.ricker_wavelet(s.nt, s.fm, s.dt)).cuda()
    ids = np.arange(shots, dtype=np.int32)
    dobs = torch.randn((shots, s.nt, s.ng), generator=torch.Generator().manual_seed(2)).cuda()
    out = []
    for arith in (S.ARITH_FAST, S.ARITH_REF):
        m = S.Damp4t10d.from_survey(s, arith=arith)
        m.set_tuning(6, 120, 40, 3)   # an explicit task length keeps the streaming kernels
        vel = torch.from_numpy(m.expandDomain(layered_model(s.nx, s.nz, seed=3))).cuda()
        m.bindVelocity(vel)
        grad = torch.zeros_like(vel)
        m.gradient_batch(wlt, dobs, ids, grad)
        out.append(grad.cpu().numpy())
    # the FAST arithmetic's bound on gradients
    assert rel_l2(out[0], out[1]) < 1e-4


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("where", PLACES)
@pytest.mark.parametrize("nb", [8, 10])
def test_resident_sweeps(cuda, arith, where, nb):
    """The resident sweep, which does both in one phase of a step, against
    the streaming kernels: the same bits."""
    s = survey(where, nb)
    for a, b in zip(sweep(cuda, s, arith, False), sweep(cuda, s, arith, True)):
        assert cuda.equal(a, b)
