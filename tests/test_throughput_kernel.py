"""The throughput kernel (several modes per SM) against the generic kernel at the launch shape whose results
it reproduces: every sum keeps its order, so mixed-precision results are equal bit for bit.  All-FP64
solves differ by the rounding of the pivots' reciprocals (1e-16, times the condition of the
tight-coupling head, about 1e5, over some thousand solves): 1e-9 of the result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODELS = {
    "n18": dict(lmax_gamma=3, lmax_nu=3, massive_nu=False),
    "n47": dict(lmax=5),
    "n128 full slots": dict(lmax_gamma=30, lmax_nu=10, lmax_h=9, nx=5),
    "n129": dict(lmax_gamma=30, lmax_nu=11, lmax_h=9, nx=5),
    "n181 eight momentum bins": dict(lmax_gamma=30, lmax_nu=17, lmax_h=11, nx=8),
}


@pytest.fixture(scope="module")
def S():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import symboltz
    return symboltz


def _sms():
    import torch
    return torch.cuda.get_device_properties(0).multi_processor_count


def _solve(S, model, per_sm, output="delta_m", taus=None, kmax=15.0, **kw):
    """per_sm modes per SM (one more than a multiple) of three cosmologies, 40 of them distinct in k."""
    M = S.ΛCDM(**model)
    base = S.parameters_Planck18(M)
    p = S.CosmologyProblem(M, [dict(base, h=0.66 + 0.01 * i) for i in range(3)], **kw)
    n = per_sm * _sms() - 3
    ks = np.geomspace(0.3, kmax, 40)[np.arange(n) % 40]
    cos = np.arange(n) % 3
    if taus is not None:
        bg = p.solvebg()
        taus = np.stack([np.concatenate([[1e-6], np.linspace(0.05, bg.tau0[c], taus - 1)]) for c in range(3)])
    ti = (lambda k: np.minimum(1e-2 / k, 1e-4)) if taus is None else 1e-6
    return S.solvept(p, ks, ti, saveat=taus, output=output, cosmo=cos)


def _check(a, b, exact=True):
    assert np.all(a[1] == 0)
    np.testing.assert_array_equal(a[1], b[1])
    if exact:
        np.testing.assert_array_equal(a[0], b[0])
        np.testing.assert_array_equal(a[2], b[2])
    else:
        np.testing.assert_allclose(a[0], b[0], rtol=1e-9)


# modes per SM at both ends of each sharing level, and the generic shape with the same sums
@pytest.mark.parametrize("per_sm,generic", [(8, dict(warps_per_mode=4, blocks_per_sm=2)), (10, dict(warps_per_mode=4, blocks_per_sm=2)),
                                            (16, dict(warps_per_mode=4, blocks_per_sm=2)), (29, dict(warps_per_mode=4, blocks_per_sm=2)),
                                            (33, dict(warps_per_mode=1))])
@pytest.mark.parametrize("model", ["n47", "n129"])
def test_same_bits_as_the_generic_kernel(S, model, per_sm, generic):
    _check(_solve(S, MODELS[model], per_sm), _solve(S, MODELS[model], per_sm, **generic))


# modes of far different lengths: fewer share an SM (one to four at these counts)
@pytest.mark.parametrize("per_sm", [4, 7, 10, 17])
@pytest.mark.parametrize("model", ["n47", "n129"])
def test_far_apart_lengths(S, model, per_sm):
    _check(_solve(S, MODELS[model], per_sm, kmax=300.0), _solve(S, MODELS[model], per_sm, kmax=300.0, warps_per_mode=4, blocks_per_sm=2))


@pytest.mark.parametrize("per_sm", [9, 33])
@pytest.mark.parametrize("model", list(MODELS))
def test_state_sizes_two_warp_order(S, model, per_sm):
    _check(_solve(S, MODELS[model], per_sm, warps_per_mode=2), _solve(S, MODELS[model], per_sm, warps_per_mode=2, blocks_per_sm=2))


@pytest.mark.parametrize("per_sm", [12, 33])
@pytest.mark.parametrize("output", ["sources", "sources4", "factors", "state"])
def test_saved_times(S, output, per_sm):
    g = dict(warps_per_mode=4, blocks_per_sm=2) if per_sm <= 32 else dict(warps_per_mode=1)
    _check(_solve(S, MODELS["n47"], per_sm, output, 9), _solve(S, MODELS["n47"], per_sm, output, 9, **g))


def test_all_fp64(S):
    _check(_solve(S, MODELS["n129"], 12, precision="fp64"), _solve(S, MODELS["n129"], 12, precision="fp64", warps_per_mode=4, blocks_per_sm=2),
           exact=False)


def test_failed_modes(S):
    """The iteration limit reached by every mode, and modes that start at τ0."""
    M = S.ΛCDM(lmax=5)
    n = 12 * _sms()
    ti = np.where(np.arange(n) % 5 == 0, 100.0, 1e-5)
    r = []
    for kw in ({}, dict(warps_per_mode=4, blocks_per_sm=2)):
        p = S.CosmologyProblem(M, S.parameters_Planck18(M), maxiters=40, **kw)
        r.append(S.solvept(p, np.linspace(1.0, 50.0, n), ti, output="delta_m"))
    assert np.all(r[0][1] == np.where(np.arange(n) % 5 == 0, 0, 1))
    for x, y in zip(*r):
        np.testing.assert_array_equal(x, y)
