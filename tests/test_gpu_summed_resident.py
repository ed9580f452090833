"""A FAST batch gradient whose sweeps are resident (an image per shot) against
the streamed one (one image, summed step by step)."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,ns", [(60, 40, 2), (150, 61, 7), (200, 90, 20)])
def test_summed_gradient_resident_and_streamed(cuda, nx, nz, ns):
    import swfwi_b200 as S
    torch = cuda
    s = Survey(nz=nz, nx=nx, dx=25.0, dt=0.002, nt=260, fm=10.0, nb=10, ns=ns, sxbeg=1, jsx=max(1, (nx - 2) // ns),
               ng=nx, szbeg=2, gzbeg=3)
    wlt = torch.from_numpy(S.ricker_wavelet(s.nt, s.fm, s.dt)).cuda()
    ids = np.arange(ns, dtype=np.int32)
    out = []
    for streamed in (False, True):
        m = S.Damp4t10d.from_survey(s, arith=S.ARITH_FAST)
        if streamed:
            m.set_tuning(6, 120, 40, 3)
        vel = torch.from_numpy(m.expandDomain(layered_model(nx, nz, seed=5))).cuda()
        m.bindVelocity(vel)
        dobs = torch.randn((ns, s.nt, m.getng()), generator=torch.Generator("cuda").manual_seed(2), device="cuda")
        grad = torch.zeros_like(vel)
        obj = m.gradient_batch(wlt, dobs, ids, grad)
        out.append((grad.double(), obj))
    (a, oa), (b, ob) = out
    np.testing.assert_array_equal(oa, ob)              # the forward sweeps agree bit for bit
    # the same products, at most 260 * 20 of them in another order: FP32
    # roundings add up as a random walk, sqrt(5200) * 2^-24 = 4.3e-6 of their
    # root sum square, which the gradient's own norm bounds within a factor of a few
    assert float((a - b).norm() / b.norm()) < 2e-5
