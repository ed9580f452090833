"""The EnKF analysis at the edges of its tiles: member counts around a tensor
tile and the eigen solver's tournament (odd, two, full), rows around a chunk,
model points around a tile; and concurrent calls, which share the kept
scratch."""
import threading

import numpy as np
import pytest

from oracle import enkf_oracle as E
from tests.gpu_helpers import t

pytestmark = pytest.mark.gpu


def _data(n, rows, seed):
    rng = np.random.default_rng(seed)
    base = rng.standard_normal(rows).astype(np.float32)
    hona = (base[None, :] + 0.3 * rng.standard_normal((n, rows))).astype(np.float32)
    dobs = (base + 0.1 * rng.standard_normal(rows)).astype(np.float32)
    return hona, dobs, rng.standard_normal((n, rows))


@pytest.mark.parametrize("n,rows,model", [(2, 31, 1), (3, 33, 127), (4, 32, 128), (7, 65, 129), (8, 4736, 500),
                                          (9, 4737, 1000), (33, 5000, 257), (63, 9001, 385), (64, 4769, 3)])
def test_analysis_edges_match_oracle(cuda, n, rows, model):
    import swfwi_b200 as S
    hona, dobs, z = _data(n, rows, seed=100 + n)
    dx, dt = 20.0, 0.002
    rng = np.random.default_rng(n)
    vels = E.vel_trans((2500 + 200 * rng.standard_normal((n, model))).astype(np.float32), dx, dt)
    want, sigma, clip = E.gain_matrix(hona, dobs, z, 0.05)
    v = t(cuda, vels)
    got, gs, gclip = S.enkf_analyze(t(cuda, hona), t(cuda, dobs), v, dx, dt, z=t(cuda, z), sigfac=0.05)
    assert gs == sigma and gclip == clip
    # FP64 sums of well-conditioned data (spreads within a factor of ten, so
    # s^-4 within 1e4): 1e4 * 1e-13 at most
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err < 1e-9, err
    # one FP32 rounding of the velocity, squared: 2 * 6e-8, and its inverse
    rel = np.abs(v.cpu().numpy() - E.analyze_update(vels, want, dx, dt)) / np.abs(vels)
    assert rel.max() < 1e-6, rel.max()


def test_concurrent_gains_match_serial(cuda):
    import swfwi_b200 as S
    torch = cuda
    cases = [(16, 3000, 1), (64, 9000, 2), (33, 7000, 3)]
    data = [tuple(t(torch, x) for x in _data(*c)) for c in cases]
    want = [S.enkf_gain_matrix(h, d, z, sigfac=0.05)[0] for h, d, z in data]
    torch.cuda.synchronize()
    got = [[] for _ in cases]

    def work(k):
        st = torch.cuda.Stream()
        h, d, z = data[k]
        for _ in range(5):
            got[k].append(S.enkf_gain_matrix(h, d, z, sigfac=0.05, stream=st)[0])

    th = [threading.Thread(target=work, args=(k,)) for k in range(len(cases))]
    for x in th:
        x.start()
    for x in th:
        x.join()
    for k in range(len(cases)):
        assert len(got[k]) == 5
        for g in got[k]:
            np.testing.assert_array_equal(g, want[k])
