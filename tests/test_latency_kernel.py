"""The latency kernel (one mode per SM on eight warps) against the generic kernel with the same four
warps per mode: every sum keeps its order and every expression its form, so mixed-precision results
are equal bit for bit.  All-FP64 solves differ by the rounding of the pivots' reciprocals (1e-16, times
the condition of the tight-coupling head, about 1e5, over some thousand solves): 1e-9 of the result.
blocks_per_sm = 1 takes the latency kernel, 2 the generic one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

MODELS = {
    "n18 one-row tails": dict(lmax_gamma=3, lmax_nu=3, massive_nu=False),
    "n47": dict(lmax=5),
    "n96 functionals on a warp without rows": dict(lmax_gamma=20, lmax_nu=8, lmax_h=9, nx=4),
    "n97 functionals beside rows": dict(lmax_gamma=20, lmax_nu=9, lmax_h=9, nx=4),
    "n128 full slot": dict(lmax_gamma=30, lmax_nu=10, lmax_h=9, nx=5),
    "n129 one row in the second slot": dict(lmax_gamma=30, lmax_nu=11, lmax_h=9, nx=5),
    "32-row chains": dict(lmax_gamma=34, lmax_nu=31, lmax_h=4, nx=2),
    "33-row chain, generic": dict(lmax_gamma=35, lmax_nu=5, lmax_h=4, nx=2),
    "six momentum bins, generic": dict(lmax=5, nx=6),
}


@pytest.fixture(scope="module")
def S():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no GPU")
    import symboltz
    return symboltz


def _both(S, model, run, **kw):
    M = S.ΛCDM(**model)
    return [run(S.CosmologyProblem(M, S.parameters_Planck18(M), warps_per_mode=4, blocks_per_sm=b, **kw)) for b in (1, 2)]


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
@pytest.mark.parametrize("model", list(MODELS))
def test_same_bits_as_the_generic_kernel(S, model, precision):
    ks = np.array([0.3, 20.0, 200.0])
    a, b = _both(S, MODELS[model], lambda p: S.solvept(p, ks, lambda k: np.minimum(1e-2 / k, 1e-4), output="delta_m"),
                 precision=precision)
    assert np.all(a[1] == 0)
    if precision == "fp64":
        np.testing.assert_allclose(a[0], b[0], rtol=1e-9)
        return
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("output", ["sources", "sources4", "factors", "state"])
def test_saved_times(S, output):
    """Saved times before, at and after the start, several in one step, and the last one at τ0."""
    def run(p):
        t0 = p.solvebg().tau0[0]
        taus = np.concatenate([[5e-7, 1e-6], np.linspace(0.05, 0.08, 40), np.linspace(0.1, t0, 12)])
        return S.solvept(p, np.array([1.0, 60.0]), 1e-6, saveat=taus, output=output)
    a, b = _both(S, MODELS["n129 one row in the second slot"], run)
    assert np.all(a[1] == 0)
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)


def test_failed_and_skipped_modes(S):
    """Iteration limit, a mode that starts at τ0, NaN and zero wavenumbers, next to a good mode."""
    def run(p):
        t0 = p.solvebg().tau0[0]
        return S.solvept(p, np.array([50.0, 1.0, np.nan, 0.0, 2.0]), np.array([1e-5, 2 * t0, 1e-5, 1e-5, 0.9 * t0]), output="delta_m")
    a, b = _both(S, MODELS["n47"], run, maxiters=60)
    assert a[1][0] == 1 and a[1][1] == 0 and a[1][2] != 0 and a[1][4] == 0
    for x, y in zip(a, b):
        np.testing.assert_array_equal(x, y)
