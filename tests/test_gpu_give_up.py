"""A sweep whose bounded wait on its neighbours runs out (a wait limit of one
unsuccessful poll): the call's results are NaN where the sweep did not get,
the failure is reported once, and the next sweep of the same object is whole."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model
from tests.gpu_helpers import t

pytestmark = pytest.mark.gpu

TIMEOUT = 3        # SWFWI_ERR_TIMEOUT
LIMIT = 1 << 31    # the default


def raises_timeout(call):
    import swfwi_b200 as S
    with pytest.raises(S.SwfwiError) as e:
        call()
    assert e.value.status == TIMEOUT


def propagator(torch, arith, ns=3):
    import swfwi_b200 as S
    s = Survey(nz=90, nx=300, dx=25.0, dt=0.002, nt=300, fm=10.0, nb=20, ns=ns, sxbeg=10, jsx=90, ng=300)
    m = S.Damp4t10d.from_survey(s, arith=arith)
    vel = t(torch, m.expandDomain(layered_model(s.nx, s.nz, seed=3)))
    m.bindVelocity(vel)
    return s, m, vel, t(torch, S.ricker_wavelet(s.nt, s.fm, s.dt))


@pytest.mark.parametrize("arith", [0, 1])
def test_modelling(cuda, arith):
    torch = cuda
    s, m, _, wlt = propagator(torch, arith)
    want, got = torch.zeros((2, s.nt, s.ng), device="cuda")
    m.FwiForwardModeling(wlt, want, 1)
    m.check()
    m.set_wait_limit(0)
    m.FwiForwardModeling(wlt, got, 1)
    raises_timeout(m.check)
    m.check()                                   # once
    assert bool(got[-1].isnan().any()) and not bool(got[0].isnan().any())
    m.set_wait_limit(LIMIT)
    m.FwiForwardModeling(wlt, got, 1)
    m.check()
    assert torch.equal(got, want)


@pytest.mark.parametrize("arith", [0, 1])
def test_gradients(cuda, arith):
    torch = cuda
    s, m, vel, wlt = propagator(torch, arith)
    res = torch.randn((s.nt, s.ng), generator=torch.Generator().manual_seed(1)).cuda()
    enc = (wlt[:, None] * torch.tensor([1.0, -1.0, 1.0], device="cuda")).contiguous()
    want, got = torch.zeros((2, *vel.shape), device="cuda")
    m.calgradient_ess(enc, res, want)
    m.set_wait_limit(0)
    m.calgradient_ess(enc, res, got)
    raises_timeout(m.check)
    assert bool(got.isnan().any())
    # a flag still up poisons no later sweep
    m.calgradient_ess(enc, res, got)
    m.set_wait_limit(LIMIT)
    got.zero_()
    m.calgradient_ess(enc, res, got)
    assert torch.equal(got, want)
    raises_timeout(m.check)
    # calls that return to the host report it themselves
    m.set_wait_limit(0)
    dobs = torch.zeros((3, s.nt, s.ng), device="cuda")
    raises_timeout(lambda: m.gradient_batch(wlt, dobs, np.arange(3, dtype=np.int32), got))


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("adj", [False, True])
@pytest.mark.parametrize("exact", [False, True])
def test_lsrtm(cuda, arith, adj, exact):
    import swfwi_b200 as S
    torch = cuda
    nx, nz, nt, ng = 200, 90, 260, 150
    rng = np.random.default_rng(3)
    vel = t(torch, rng.uniform(1500, 2500, (nx, nz)).astype(np.float32))
    mod = t(torch, rng.standard_normal((nx, nz)).astype(np.float32))
    dat = t(torch, rng.standard_normal((1, ng, nt)).astype(np.float32))
    a = dict(dz=10.0, dx=10.0, dt=0.001, amp=1.0, fm=25.0, nb=20, nt=nt, ns=1, ng=ng, sxbeg=50, szbeg=2, jsx=0, jsz=0,
             gxbeg=0, gzbeg=2, jgx=1, jgz=0, arith=arith)

    def run(op):
        out = (mod if adj else dat).clone()
        op.lop(adj, False, out if adj else mod, dat if adj else out)
        return out

    op = S.Prtm2d(vel, **a)
    op.set_adjoint(S.PRTM_ADJ_EXACT if exact else S.PRTM_ADJ_REFERENCE)
    want = run(op)
    op.check()
    op.close()
    op = S.Prtm2d(vel, **a)
    op.set_adjoint(S.PRTM_ADJ_EXACT if exact else S.PRTM_ADJ_REFERENCE)
    op.set_wait_limit(0)
    got = run(op)
    assert bool(got.isnan().any())
    raises_timeout(op.check)                    # by the call that asks
    op.check()
    run(op)
    torch.cuda.synchronize()
    raises_timeout(lambda: run(op))             # or by the next one
    op.set_wait_limit(LIMIT)
    assert torch.equal(run(op), want)
    op.check()
    op.close()


def test_operators_report_for_themselves(cuda):
    """Several operators alive, made and closed in turn: one that gave up is
    the only one to say so, and a new one starts clean."""
    import swfwi_b200 as S
    torch = cuda
    nx, nz, nt, ng = 200, 60, 100, 100
    vel = torch.full((nx, nz), 2000.0, device="cuda")
    mod = torch.ones((nx, nz), device="cuda")
    dat = torch.zeros((1, ng, nt), device="cuda")

    def make():
        return S.Prtm2d(vel, dz=10.0, dx=10.0, dt=0.001, amp=1.0, fm=25.0, nb=20, nt=nt, ns=1, ng=ng, sxbeg=50, szbeg=2,
                        jsx=0, jsz=0, gxbeg=0, gzbeg=2, jgx=1, jgz=0, arith=S.ARITH_FAST)

    ops = [make() for _ in range(5)]
    ops[2].set_wait_limit(0)
    for op in ops:
        op.lop(False, False, mod, dat)
    torch.cuda.synchronize()
    for k in (0, 1, 3, 4):
        ops[k].check()
    ops[2].close()                              # unasked
    fresh = make()                              # may take over its word
    fresh.lop(False, False, mod, dat)
    fresh.check()
    for op in (*ops[:2], *ops[3:], fresh):
        op.check()
        op.close()


def test_host_gradient_without_objectives_reports(cuda):
    import ctypes as C
    import swfwi_b200 as S
    torch = cuda
    s, m, vel, wlt = propagator(torch, S.ARITH_FAST)
    v, w = vel.cpu().numpy(), wlt.cpu().numpy()
    d, g, ids = np.zeros((3, s.nt, s.ng), np.float32), np.zeros_like(v), np.arange(3, dtype=np.int32)

    def call():
        f, i = C.POINTER(C.c_float), C.POINTER(C.c_int)
        S._check(S.lib().swfwi_gradient_host(m.h, v.ctypes.data_as(f), w.ctypes.data_as(f), d.ctypes.data_as(f),
                                             ids.ctypes.data_as(i), 3, g.ctypes.data_as(f), None))

    call()
    m.set_wait_limit(0)
    raises_timeout(call)
    m.set_wait_limit(LIMIT)
    call()
    m.check()


@pytest.mark.parametrize("regularised", [False, True])
def test_encoded_epoch_reports_and_keeps_its_model(cuda, regularised):
    import swfwi_b200 as S
    torch = cuda
    s, m, vel, wlt = propagator(torch, S.ARITH_FAST)
    dobs = np.random.default_rng(1).standard_normal((3, s.nt, s.ng)).astype(np.float32)
    fw = S.EssFwiFramework(m, vel.cpu().numpy(), s.vmin, s.vmax, s.nita, s.maxdv, wlt.cpu().numpy(), dobs)
    if regularised:
        fw.setRegularization(1.0, 1.0)
    fw.epoch(0)
    before = fw.velocity()
    m.set_wait_limit(0)
    raises_timeout(lambda: fw.epoch(1))
    np.testing.assert_array_equal(fw.velocity(), before)
    m.set_wait_limit(LIMIT)
    fw.epoch(1)
    assert np.isfinite(fw.velocity()).all() and not np.array_equal(fw.velocity(), before)
