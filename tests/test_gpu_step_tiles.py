"""The tiled stencil step at the edges of its two tile shapes (16 rows for
small grids, 32 for large) and in a row of dependent launches: the damped
step of one grid equals the FP64 step to FP32 rounding, and the reference
arithmetic of a batch equals that of its fields alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz", [(13, 13), (28, 44), (29, 45), (44, 76), (45, 77), (1201, 525)])
def test_batch_equals_single_and_fp64(cuda, nx, nz):
    # 1201 x 525: 608 tiles of 32 rows for one field, above the line at 592;
    # (13, 13) x 600 fields crosses it by the batch
    import swfwi_b200 as S
    torch = cuda
    nb = min(8, nx - 12, nz - 12)
    n = 600 if nx == 13 else 3
    g = torch.Generator(device="cuda").manual_seed(nx)
    p0 = torch.randn((n, nx, nz), generator=g, device="cuda")
    p1 = torch.randn((n, nx, nz), generator=g, device="cuda")
    vt = torch.rand((nx, nz), generator=g, device="cuda") * 70 + 5
    a, b = p0.clone(), p1.clone()
    for _ in range(4):
        S.fd4t10s_step_batch(a, b, vt, nb, True, S.ARITH_REF)
        a, b = b, a
    for k in (0, n - 1):
        c, d = p0[k].clone(), p1[k].clone()
        e, f = p0[k].double(), p1[k].double()
        for _ in range(4):
            S.fd4t10s_damp_zjh_2d_vtrans(c, d, vt, nb)
            S.fd4t10s_step_f64(e, f, vt.double(), nb)
            c, d = d, c
            e, f = f, e
        np.testing.assert_array_equal(b[k].cpu().numpy(), d.cpu().numpy())
        # four steps of some ten FP32 roundings of values up to the field's
        # largest, each step at most doubling what came before
        err = (d.double() - f).abs().max() / f.abs().max()
        assert float(err) < 4 * 10 * 2.0 ** -24 * 2 ** 4, float(err)
