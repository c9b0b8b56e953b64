"""The throughput kernel at every number of modes per SM, pinned by the shape that the library reports for the launch,
against the generic kernel with the same sums: equal bits in mixed precision.  All-FP64 solves differ by what the pivots'
reciprocals do (at most 1e-16, times the condition of the tight-coupling head, about 1e5, over some thousand solves):
1e-9 of the result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GENERIC, LATENCY, THROUGHPUT = 0, 1, 2
MODELS = {
    "n17 one-row tails": dict(lmax_gamma=3, lmax_nu=3, massive_nu=False),
    "n47": dict(lmax=5),
    "n98": dict(lmax_gamma=20, lmax_nu=10, lmax_h=9, nx=4),
    "n117 32-row chains": dict(lmax_gamma=34, lmax_nu=31, lmax_h=4, nx=2),
    "n128 full slots": dict(lmax_gamma=30, lmax_nu=10, lmax_h=9, nx=5),
    "n129": dict(lmax_gamma=30, lmax_nu=11, lmax_h=9, nx=5),
    "n181 eight momentum bins": dict(lmax_gamma=30, lmax_nu=17, lmax_h=11, nx=8),
}
PINNED = dict(warps_per_mode=4, blocks_per_sm=2)  # generic kernel, four-warp sums


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


def _shape(prob, ks, ntau=0):
    from symboltz import _lib as L
    out = L.i32(np.zeros(4))
    ks = L.f64(ks)
    L.check(L.lib().sbz_pt_launch_shape(prob._h, len(ks), L.dptr(ks), ntau, _sms(), L.iptr(out)))
    return tuple(int(v) for v in out)


def _both(S, model, ks, want, ti=lambda k: np.minimum(1e-2 / k, 1e-4), ntau=0, output="delta_m", exact=True, **kw):
    """The open shape (want) and the generic kernel on three cosmologies; ks: one wavenumber per mode."""
    M = S.ΛCDM(**model)
    base = S.parameters_Planck18(M)
    r = []
    for pin in ({}, PINNED):
        p = S.CosmologyProblem(M, [dict(base, h=0.66 + 0.01 * i) for i in range(3)], **pin, **kw)
        bg = p.solvebg()
        assert _shape(p, ks, ntau) == want if not pin else _shape(p, ks, ntau)[0] == GENERIC
        taus = np.stack([np.concatenate([[1e-6], np.linspace(0.05, t0, ntau - 1)]) for t0 in bg.tau0]) if ntau else None
        r.append(S.solvept(p, ks, 1e-6 if ntau else ti, saveat=taus, output=output, cosmo=np.arange(len(ks)) % 3))
    (a, sa, na), (b, sb, nb) = r
    np.testing.assert_array_equal(sa, sb)
    if exact:
        np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(na, nb)
    else:
        np.testing.assert_allclose(a, b, rtol=1e-9)
    return a, sa


def _modes(per_sm, kmax=2.0):
    n = int(per_sm * _sms()) - 3
    return np.geomspace(0.3, kmax, 40)[np.arange(n) % 40]


MIXED = {2.0: (2, 4), 2.8: (3, 4), 4.6: (4, 4), 12.0: (8, 2)}
FP64 = {2.0: (2, 4), 3.1: (3, 4), 5.0: (4, 4), 14.0: (8, 2)}


@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("per_sm", list(MIXED))
def test_mixed(S, model, per_sm):
    modes, warps = MIXED[per_sm]
    if model.startswith("n181") and modes == 8:
        modes, warps = 4, 4  # one block of four fits an SM
    _, st = _both(S, MODELS[model], _modes(per_sm), (THROUGHPUT, 4, modes, warps))
    assert np.all(st == 0)


@pytest.mark.parametrize("model", list(MODELS))
@pytest.mark.parametrize("per_sm", list(FP64))
def test_all_fp64(S, model, per_sm):
    modes, warps = FP64[per_sm]
    if int(model[1:].split()[0]) > 107 and modes > 3:
        modes, warps = 4, 2
    _, st = _both(S, MODELS[model], _modes(per_sm), (THROUGHPUT, 4, modes, warps), exact=False, precision="fp64")
    assert np.all(st == 0)


@pytest.mark.parametrize("output", ["sources", "sources4", "factors", "state"])
@pytest.mark.parametrize("precision,model,per_sm,modes,warps", [
    ("mixed", "n47", 2.0, 2, 4), ("mixed", "n129", 2.9, 3, 4), ("mixed", "n129", 4.0, 4, 4), ("mixed", "n47", 12.0, 8, 2),
    ("fp64", "n129", 2.0, 2, 4), ("fp64", "n47", 5.0, 4, 4), ("fp64", "n129", 14.0, 4, 2), ("fp64", "n47", 14.0, 8, 2)])
def test_saved_times(S, precision, model, per_sm, modes, warps, output):
    exact = precision == "mixed"
    if exact:
        a, st = _both(S, MODELS[model], _modes(per_sm), (THROUGHPUT, 4, modes, warps), ntau=9, output=output)
        assert np.all(st == 0) and np.isfinite(a[:, 1:-1]).all()
    else:  # entries that cancel: 1e-9 of the largest of their kind
        M = S.ΛCDM(**MODELS[model])
        ks = _modes(per_sm)
        r = []
        for pin in ({}, PINNED):
            p = S.CosmologyProblem(M, S.parameters_Planck18(M), precision=precision, **pin)
            taus = np.concatenate([[1e-6], np.linspace(0.05, 0.99 * p.solvebg().tau0[0], 8)])
            assert _shape(p, ks, 9) == (THROUGHPUT, 4, modes, warps) if not pin else _shape(p, ks, 9)[0] == GENERIC
            r.append(S.solvept(p, ks, 1e-6, saveat=taus, output=output))
        assert np.all(r[0][1] == 0)
        scale = np.abs(r[1][0]).max(axis=(0, 1), keepdims=True)
        assert np.all(np.abs(r[0][0] - r[1][0]) <= 1e-9 * scale)


# NaN and zero wavenumbers leave the modes' lengths unknown: a quarter of the longest each is assumed
@pytest.mark.parametrize("per_sm,modes,warps", [(8.0, 2, 4), (11.0, 3, 4), (16.0, 4, 4), (31.0, 8, 2)])
def test_failed_modes_beside_good_ones(S, per_sm, modes, warps):
    """NaN and zero wavenumbers, modes that reach the iteration limit, and modes that start at τ0."""
    ks = _modes(per_sm, 60.0)
    n = np.arange(len(ks))
    ks = np.where(n % 11 == 3, np.nan, np.where(n % 11 == 7, 0.0, ks))
    ti = np.where(n % 5 == 0, 100.0, 1e-5)
    _, st = _both(S, MODELS["n47"], ks, (THROUGHPUT, 4, modes, warps), ti=lambda k: ti, maxiters=60)
    good = ~((n % 11 == 3) | (n % 11 == 7))
    assert np.all(st[good & (n % 5 == 0)] == 0) and np.all(st[good & (n % 5 != 0) & (ks > 30)] == 1)
    assert np.all(st[(n % 11 == 3) & (n % 5 != 0)] != 0)
