"""The resident time loop's forms and exchange layouts against the streaming
kernels, bit for bit: slabs of one to five rows (rows exchanged with slabs
further away), the two-pass form at one round of items, a remainder and its
limit, and the march where the two-pass form does not fit or is slower."""
import pytest

from swfwi_b200.survey import Survey
from tests.test_gpu_resident import sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arith,nx,nz,ns", [
    (0, 14, 20, 1),      # 22 slabs of a row, every exchange across several slabs
    (1, 160, 33, 1),     # slabs of 1 and 2 rows
    (1, 700, 64, 1),     # slabs of 4 and 5 rows
    (0, 860, 30, 1),     # of 5 and 6
    (0, 461, 101, 1),    # thin, REF, two-pass
    (1, 480, 560, 1),    # FAST beyond the two-pass limit: the march, slabs of 6 rows or more
    (0, 300, 170, 30),   # REF where u2 does not fit beside the fields: the march
    (1, 300, 170, 30),
])
def test_forms_match_the_streaming_kernels(cuda, arith, nx, nz, ns):
    s = Survey(nz=nz, nx=nx, dx=25.0, dt=0.002, nt=181, fm=10.0, nb=10, ns=ns, sxbeg=1, jsx=max(1, (nx - 2) // ns),
               ng=nx, szbeg=2, gzbeg=3)
    for a, b in zip(sweep(cuda, s, arith, False), sweep(cuda, s, arith, True)):
        assert cuda.equal(a, b)
