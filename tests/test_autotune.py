"""The launch-shape tuner never ends on a launch slower than the one that leaves the shape open."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seconds(S, prob, ks, ti):
    t = []
    for _ in range(3):
        t0 = time.perf_counter()
        _, st, _ = S.solvept(prob, ks, ti, output="delta_m")
        t.append(time.perf_counter() - t0)
        assert np.all(st == 0)
    return min(t)


# above 2,048 modes (few and many rounds of the longest modes) and below
@pytest.mark.parametrize("n,kmax", [(2400, 0.2), (9000, 0.05), (300, 0.2)])
def test_tuned_is_not_slower_than_open(n, kmax):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import symboltz as S
    M = S.ΛCDM(lmax_gamma=30, lmax_nu=10, lmax_h=10, nx=5)
    ks = S.k_from_hMpc(np.geomspace(1e-4, kmax, n))
    ti = lambda k: np.minimum(1e-2 / k, 1e-4)  # noqa: E731
    prob = S.CosmologyProblem(M, S.parameters_Planck18(M))
    open_s = _seconds(S, prob, ks, ti)
    tune = S.autotune(prob, ks, ti, output="delta_m")
    assert len(tune["candidates_ms"]) == 9 and all(v > 0 for v in tune["candidates_ms"].values())
    best = (tune["warps_per_mode"], tune["blocks_per_sm"])
    assert tune["candidates_ms"][best] <= tune["candidates_ms"][0, 0]
    # another shape was at least 2 % faster where it was timed; 5 % for what a timing varies
    assert _seconds(S, prob, ks, ti) <= 1.05 * open_s, tune
