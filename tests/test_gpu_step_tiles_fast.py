"""The tiled stencil step in FAST arithmetic around the line between its two
tile shapes: the fields of a batch equal those fields alone, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,nz,n", [(814, 72, 12), (85, 1850, 5), (85, 1850, 6), (44, 44, 889)])
def test_fast_batch_equals_single(cuda, nx, nz, n):
    # FAST changes tiles at 888 tiles of 32 rows: batches of 624, 870, 1044
    # and 889 of them, each field alone far below
    import swfwi_b200 as S
    torch = cuda
    g = torch.Generator(device="cuda").manual_seed(nx)
    p0 = torch.randn((n, nx, nz), generator=g, device="cuda")
    p1 = torch.randn((n, nx, nz), generator=g, device="cuda")
    vt = torch.rand((nx, nz), generator=g, device="cuda") * 70 + 5
    a, b = p0.clone(), p1.clone()
    for _ in range(4):
        S.fd4t10s_step_batch(a, b, vt, 8, True, S.ARITH_FAST)
        a, b = b, a
    for k in (0, n - 1):
        c, d = p0[k:k + 1].clone(), p1[k:k + 1].clone()
        for _ in range(4):
            S.fd4t10s_step_batch(c, d, vt, 8, True, S.ARITH_FAST)
            c, d = d, c
        np.testing.assert_array_equal(b[k].cpu().numpy(), d[0].cpu().numpy())
