"""A FAST batch gradient on chip in two rounds of slots, at the plain survey's
size: its images are those of the shots alone (each of which has the streaming
kernels' bits), summed in FP32."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model
from tests.gpu_helpers import t

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,ns", [(461, 151, 20), (200, 100, 33)])
def test_two_rounds_sum_the_shots_images(cuda, nx, nz, ns):
    import swfwi_b200 as S
    torch = cuda
    s = Survey(nz=nz, nx=nx, dx=25.0, dt=0.002, nt=260, fm=10.0, nb=30, ns=ns, sxbeg=1, jsx=(nx - 2) // ns, ng=nx)
    wlt = t(torch, S.ricker_wavelet(s.nt, s.fm, s.dt))
    dobs = torch.randn((ns, s.nt, nx), generator=torch.Generator("cuda").manual_seed(2), device="cuda")

    def method(streaming):
        m = S.Damp4t10d.from_survey(s, arith=S.ARITH_FAST)
        if streaming:   # an explicit task length keeps the streaming kernels
            m.set_tuning(6, 120, 40, 3)
        vel = t(torch, m.expandDomain(layered_model(nx, nz, seed=3)))
        m.bindVelocity(vel)
        return m, vel

    m, vel = method(False)
    m.gradient_batch(wlt, dobs, np.array([0], np.int32), torch.zeros_like(vel))      # forms 1/vt
    every = torch.zeros_like(vel)
    S.stats_reset()
    obj = m.gradient_batch(wlt, dobs, np.arange(ns, dtype=np.int32), every)
    assert 4 < S.stats_read()["kernel_launches"] <= 14          # two launches a sweep
    total, size = torch.zeros_like(vel, dtype=torch.float64), torch.zeros_like(vel, dtype=torch.float64)
    streamed, _ = method(True)
    for k in range(ns):
        one, other = torch.zeros_like(vel), torch.zeros_like(vel)
        assert m.gradient_batch(wlt, dobs, np.array([k], np.int32), one)[0] == obj[k]
        if k % 8 == 0:
            streamed.gradient_batch(wlt, dobs, np.array([k], np.int32), other)
            assert torch.equal(one, other)
        total += one.double()
        size += one.double().abs()
    # ns - 1 additions and the scaling of each gradient, FP32
    assert bool(((every.double() - total).abs() <= (ns + 4) * 2.0 ** -24 * size).all())
