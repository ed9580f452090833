"""The LSRTM operator's two forms, on-chip sweeps and launched time loops: the
form that set_resident asks for is the one that runs, the launched loops replay
as graphs with the same bits and counts, and the forms agree: bit for bit in
the reference arithmetic, also where calls alternate between them (the Born
branch continues from the fields of the call before)."""
import ctypes

import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.gpu_helpers import t
from tests.test_gpu_lsrtm import _op

pytestmark = pytest.mark.gpu


def calls(torch, op, g, modes, launched=None):
    """Two rounds of modelling and migration; launched(i): whether call i
    takes the launched loops."""
    mod, dat = t(torch, g["line_mod"]), t(torch, g["line_dat"])
    b, m = torch.zeros_like(dat), torch.zeros_like(mod)
    out = []
    for mode in modes:
        op.set_adjoint(mode)
        for _ in range(3):
            for adj in (False, True):
                if launched is not None:
                    op.set_resident(not launched(len(out)))
                op.lop(adj, False, m if adj else mod, dat if adj else b)
                out.append((m if adj else b).cpu().numpy().copy())
    return out


@pytest.mark.parametrize("arith", [0, 1])
def test_launched_loops_replay_bit_identical(cuda, arith):
    import swfwi_b200 as S
    outs, counts = [], []
    for graphs in (True, False):
        op, g = _op(cuda, "line", arith)
        op.set_resident(False)
        op.set_graphs(graphs)
        cuda.cuda.synchronize()
        S.stats_reset()
        outs.append(calls(cuda, op, g, (S.PRTM_ADJ_REFERENCE, S.PRTM_ADJ_EXACT)))
        counts.append(S.stats_read()["kernel_launches"])
        op.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)
    assert counts[0] == counts[1]
    assert counts[0] > 12 * 2 * g["line_dat"].shape[-1]     # launches every step


@pytest.mark.parametrize("arith", [0, 1])
def test_on_chip_sweeps_are_few_launches(cuda, arith):
    import swfwi_b200 as S
    op, g = _op(cuda, "line", arith)
    cuda.cuda.synchronize()
    S.stats_reset()
    calls(cuda, op, g, (S.PRTM_ADJ_REFERENCE, S.PRTM_ADJ_EXACT))
    shots = g["line_dat"].shape[0] if arith == S.ARITH_REF else 1
    assert S.stats_read()["kernel_launches"] <= 12 * 3 * shots
    op.close()


@pytest.mark.parametrize("pattern", ["never", "always", "every other", "first half"])
def test_forms_agree_bit_for_bit_in_reference_arithmetic(cuda, pattern):
    import swfwi_b200 as S
    pick = {"never": lambda i: False, "always": lambda i: True, "every other": lambda i: i % 2 == 0,
            "first half": lambda i: i < 6}[pattern]
    outs = []
    for launched in (lambda i: True, pick):
        op, g = _op(cuda, "line", S.ARITH_REF)
        outs.append(calls(cuda, op, g, (S.PRTM_ADJ_REFERENCE, S.PRTM_ADJ_EXACT), launched))
        op.close()
    for a, b in zip(*outs):
        np.testing.assert_array_equal(a, b)


def test_forms_agree_in_fast_arithmetic(cuda):
    import swfwi_b200 as S
    outs = []
    for on in (True, False):
        op, g = _op(cuda, "line", S.ARITH_FAST)
        op.set_resident(on)
        outs.append(calls(cuda, op, g, (S.PRTM_ADJ_REFERENCE, S.PRTM_ADJ_EXACT)))
        op.close()
    for a, b in zip(*outs):     # each within the FAST bound of 64 bits
        assert rel_l2(a, b) < 2e-4


def stale_blocks(torch, size, n=64):
    """Frees every other of n device blocks of `size` bytes filled with 12.08f,
    so that allocations of that size find them; returns the others, to be
    freed by the caller (the driver clears memory that it maps anew)."""
    rt = ctypes.CDLL("libcudart.so.12")
    blocks = []
    for _ in range(n):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0
        assert rt.cudaMemset(p, 0x41, ctypes.c_size_t(size)) == 0
        blocks.append(p)
    torch.cuda.synchronize()
    for p in blocks[::2]:
        assert rt.cudaFree(p) == 0
    return rt, blocks[1::2]


@pytest.mark.parametrize("arith", [0, 1])
@pytest.mark.parametrize("nb", [2, 3, 4])
def test_thin_sponge_ring_is_saved_whole(cuda, arith, nb):
    """With a sponge of 2 or 3 cells the saved ring has cells in the grid's
    outer rows: they have to be written too, or the migration restores what
    the memory held before."""
    import swfwi_b200 as S
    nx, nz, nt, ng = 24, 16, 200, 12
    rng = np.random.default_rng(nb)
    vel = t(cuda, rng.uniform(1500, 2500, (nx, nz)).astype(np.float32))
    dat = t(cuda, rng.standard_normal((1, ng, nt)).astype(np.float32))
    out = []
    for resident in (False, True):
        rt, kept = stale_blocks(cuda, nt * 4 * (nx + nz) * 4)
        op = S.Prtm2d(vel, dz=10.0, dx=10.0, dt=0.001, amp=1.0, fm=25.0, nb=nb, nt=nt, ns=1, ng=ng, sxbeg=12, szbeg=8,
                      jsx=0, jsz=0, gxbeg=0, gzbeg=2, jgx=2, jgz=0, arith=arith)
        op.set_resident(resident)
        m = cuda.zeros((nx, nz), device="cuda")
        op.lop(True, False, m, dat)
        out.append(m.cpu().numpy())
        op.close()
        for p in kept:
            rt.cudaFree(p)
    if arith == S.ARITH_REF:
        np.testing.assert_array_equal(out[1], out[0])
    else:
        assert rel_l2(out[1], out[0]) < 2e-4


@pytest.mark.parametrize("arith,nx,nz,ns,nb,on_chip", [
    (1, 120, 90, 3, 20, True), (0, 120, 90, 2, 20, True), (1, 300, 400, 6, 20, True), (0, 400, 300, 2, 20, True),
    (1, 46, 1250, 1, 20, False), (0, 36, 1521, 2, 10, False), (1, 70, 1329, 11, 10, False),
])
def test_the_faster_form_is_chosen(cuda, arith, nx, nz, ns, nb, on_chip):
    """Deep grids, which on-chip sweeps cut into slabs of two or three rows,
    take the launched loops, with their bits; others the sweeps."""
    import swfwi_b200 as S
    nt = 60
    rng = np.random.default_rng(nx)
    vel = t(cuda, rng.uniform(1500, 2500, (nx, nz)).astype(np.float32))
    mod = t(cuda, rng.standard_normal((nx, nz)).astype(np.float32))
    dat = t(cuda, rng.standard_normal((ns, nx, nt)).astype(np.float32))
    out = []
    for resident in (True, False):
        op = S.Prtm2d(vel, dz=10.0, dx=10.0, dt=0.001, amp=1.0, fm=25.0, nb=nb, nt=nt, ns=ns, ng=nx, sxbeg=0, szbeg=1,
                      jsx=(nx - 1) // ns, jsz=0, gxbeg=0, gzbeg=2, jgx=1, jgz=0, arith=arith)
        op.set_resident(resident)
        for exact in (False, True):
            op.set_adjoint(S.PRTM_ADJ_EXACT if exact else S.PRTM_ADJ_REFERENCE)
            for adj in (False, True):
                o = cuda.zeros_like(mod if adj else dat)
                cuda.cuda.synchronize()
                S.stats_reset()
                op.lop(adj, False, o if adj else mod, dat if adj else o)
                launches = S.stats_read()["kernel_launches"]
                assert (launches < nt) == (resident and on_chip), (exact, adj, launches)
                out.append(o.cpu().numpy())
        op.close()
    for a, b in zip(out[:4], out[4:]):
        if on_chip and arith == S.ARITH_FAST:
            assert rel_l2(a, b) < 2e-4
        else:
            np.testing.assert_array_equal(a, b)
