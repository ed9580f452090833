"""The resident time loop (fields held on chip for a whole sweep) against the
streaming kernels: the same bits in both arithmetics, at depths that are and
are not multiples of the 4-depth groups, slabs down to 6 rows, several
launches a sweep, uneven spreads and vertical receiver lines."""
import numpy as np
import pytest

from swfwi_b200.survey import Survey, layered_model

pytestmark = pytest.mark.gpu


def sweep(torch, s, arith, streaming, spreads=None):
    import swfwi_b200 as S
    s = s.scaled(spreads=spreads)
    m = S.Damp4t10d.from_survey(s, arith=arith)
    if streaming:   # an explicit task length keeps the streaming kernels
        m.set_tuning(6, 120, 40, 3)
    vel = torch.from_numpy(m.expandDomain(layered_model(s.nx, s.nz, seed=3))).cuda()
    m.bindVelocity(vel)
    wlt = torch.from_numpy(S.ricker_wavelet(s.nt, s.fm, s.dt)).cuda()
    ids = np.arange(s.ns, dtype=np.int32)
    dcal = torch.full((s.ns, s.nt, m.getng()), 7.0, device="cuda")
    m.forward_batch(wlt, dcal, ids)
    out = [dcal]
    g = torch.Generator().manual_seed(1)
    codes = torch.from_numpy(S.random_codes(1, s.ns).astype(np.float32)).cuda()
    enc = (wlt[:, None] * codes[None, :]).contiguous()
    res = torch.randn((s.nt, s.ng), generator=g).cuda()
    seis = torch.zeros((s.nt, s.ng), device="cuda")
    m.EssForwardModeling(enc, seis)
    grad = torch.full_like(vel, 0.5)
    m.calgradient_ess(enc, res, grad)
    m.calgradient_fwi(wlt, res, grad, s.ns - 1)
    one = torch.zeros_like(vel)
    obj = m.gradient_batch(wlt, dcal[:1].flip(1).contiguous(), ids[:1], one)
    out += [seis, grad, one, torch.from_numpy(obj)]
    if arith == S.ARITH_REF:   # per-shot images, summed in shot order
        every = torch.zeros_like(vel)
        m.gradient_batch(wlt, dcal.flip(1).contiguous(), ids, every)
        out.append(every)
    torch.cuda.synchronize()
    return [t.cpu() for t in out]


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("nx,nz,ns,uneven", [(31, 20, 2, False), (64, 41, 3, True), (50, 42, 5, False),
                                             (97, 55, 26, True), (400, 60, 1, False), (130, 301, 17, False)])
def test_resident_sweeps_match_the_streaming_kernels(cuda, arith, nx, nz, ns, uneven):
    torch = cuda
    s = Survey(nz=nz, nx=nx, dx=25.0, dt=0.002, nt=201, fm=10.0, nb=10, ns=ns, sxbeg=1, jsx=max(1, (nx - 2) // ns),
               ng=nx, szbeg=2, gzbeg=3)
    spreads = None
    if uneven:
        off = np.cumsum([0] + [3 + (7 * i) % (nx - 3) for i in range(ns)]).astype(np.int32)
        gx = np.concatenate([np.arange(b - a) for a, b in zip(off[:-1], off[1:])]).astype(np.int32)
        spreads = (off, gx, np.full(gx.size, 3, np.int32))
    for a, b in zip(sweep(torch, s, arith, False, spreads), sweep(torch, s, arith, True, spreads)):
        assert torch.equal(a, b)


def test_resident_vertical_lines(cuda):
    """Sources and receivers down one column: every point on one row."""
    s = Survey(nz=60, nx=40, dx=25.0, dt=0.002, nt=190, fm=10.0, nb=10, ns=3, sxbeg=20, jsx=0, jsz=7, szbeg=5, ng=50,
               gxbeg=9, jgx=0, gzbeg=4, jgz=1)
    for a, b in zip(sweep(cuda, s, 1, False), sweep(cuda, s, 1, True)):
        assert cuda.equal(a, b)


def test_resident_members_match_single_sweeps(cuda):
    """One velocity per slot, in several rounds of slots."""
    import swfwi_b200 as S
    torch = cuda
    s = Survey(nz=70, nx=110, dx=25.0, dt=0.002, nt=60, fm=10.0, nb=10, ns=4, sxbeg=11, jsx=27, ng=110)
    m = S.Damp4t10d.from_survey(s, arith=S.ARITH_FAST)
    vels = torch.stack([torch.from_numpy(m.expandDomain(layered_model(s.nx, s.nz, seed=i))) for i in range(64)]).cuda()
    wlt = torch.from_numpy(S.ricker_wavelet(s.nt, s.fm, s.dt)).cuda()
    enc = (wlt[:, None] * torch.tensor([1.0, -1.0, -1.0, 1.0], device="cuda")).contiguous()
    hona = torch.empty((64, s.ng * s.nt), device="cuda")
    m.ess_forward_members(enc, vels, hona)
    one = torch.zeros((s.nt, s.ng), device="cuda")
    m.set_tuning(6, 120, 40, 3)
    for i in (0, 31, 63):
        m.bindVelocity(vels[i])
        m.EssForwardModeling(enc, one)
        assert torch.equal(hona[i], one.t().contiguous().reshape(-1))
