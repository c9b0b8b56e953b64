"""Which kernel a perturbation launch takes (host logic, no device)."""
import ctypes as C
import os

import numpy as np
import pytest


@pytest.fixture(scope="module")
def S():
    import symboltz
    if not os.path.exists(symboltz._lib.LIB_PATH):
        pytest.skip("library not built")
    return symboltz


def shape(S, model, nk, sms=152, ks=None, ntau=0, **kw):
    from symboltz import _lib as L
    M = S.ΛCDM(**model)
    p = S.CosmologyProblem(M, S.parameters_Planck18(M), **kw)
    out = L.i32(np.zeros(4))
    ks = None if ks is None else L.f64(ks)
    L.check(L.lib().sbz_pt_launch_shape(p._h, nk, None if ks is None else L.dptr(ks), ntau, sms, L.iptr(out)))
    return tuple(int(v) for v in out)


GENERIC, LATENCY, THROUGHPUT = 0, 1, 2
N133 = dict(lmax_gamma=30, lmax_nu=10, lmax_h=10, nx=5)
N181 = dict(lmax_gamma=30, lmax_nu=17, lmax_h=11, nx=8)


def test_few_modes_have_an_sm_each(S):
    assert shape(S, dict(lmax=5), 4) == (LATENCY, 4, 1, 4)
    assert shape(S, N133, 152, ks=np.geomspace(1, 600, 152)) == (LATENCY, 4, 1, 4)
    assert shape(S, N181, 4)[0] == GENERIC  # eight momentum bins
    assert shape(S, dict(lmax=5), 4, warps_per_mode=4, blocks_per_sm=2)[:2] == (GENERIC, 4)
    assert shape(S, dict(lmax=5), 4, warps_per_mode=4, blocks_per_sm=1) == (LATENCY, 4, 1, 4)
    assert shape(S, N181, 5000, warps_per_mode=2)[0] == GENERIC
    assert shape(S, N133, 5000, warps_per_mode=1)[0] == GENERIC


# equal modes, many to an SM: eight of two warps where shared memory holds two blocks of four of them; where it holds
# one (all-FP64 133 equations take 34 KB per mode, mixed 181 take 31), the rule counts four, which two warps each run
# as fast as four in all-FP64 and slower in mixed precision
@pytest.mark.parametrize("model,precision,modes,warps", [
    (dict(lmax=5), "mixed", 8, 2), (dict(lmax=5), "fp64", 8, 2), (N133, "mixed", 8, 2), (N133, "fp64", 4, 2), (N181, "mixed", 4, 4),
    (N181, "fp64", 4, 2)])
@pytest.mark.parametrize("per_sm", [12, 31])
def test_no_more_modes_per_sm_than_fit(S, model, precision, modes, warps, per_sm):
    assert shape(S, model, per_sm * 152, ks=np.full(per_sm * 152, 10.0), precision=precision) == (THROUGHPUT, 4, modes, warps)
    s = shape(S, model, 40 * 152, ks=np.full(40 * 152, 10.0), precision=precision)
    assert s == (THROUGHPUT, 1, modes, warps)


def test_sharing_grows_with_the_work(S):
    """r longest modes' worth of work per SM: alone, then two, three, four, eight to an SM."""
    got = [shape(S, dict(lmax=10), int(r * 152), ks=np.full(int(r * 152), 10.0))[2] for r in (1, 2, 3, 4, 8)]
    assert got == [1, 2, 3, 4, 8]
