"""Block fixed-point transforms (csrc/nlm_fx.cuh): the one-CTA kernels that run them, on every grid size they take,
against the oracle, and on fields at the ends of the double range.

Tolerance: the oracle's own rounding, a few 1e-16 per step of the field's norm and amplified by the medium's gain; the
media below have at most 40 steps and a gain below 10, so 1e-12 leaves a factor of ten over 40 x 1e-15 x 10 / 4."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu
TOL = 1e-12

PDC = dict(relativeLength=1, nlLength=0.5, beta2=1, beta2s=0.5, beta1s=2, beta3s=0.1, tMax=40, zPrecision=10,
           poling=np.ones(4))
SFGPDC = dict(relativeLength=1, nlLength=0.8, nlLengthOrig=1.2, beta2=0.5, beta2s=-0.3, beta2o=0.2, beta1s=1,
              beta1o=-0.5, diffBeta0=1.3, diffBeta0o=-0.4, tMax=10, zPrecision=10, poling=[1, 2, 1, 2])
ROWS = 160   # more rows than the cluster kernels take


def _media(nlm, oracle, name, n):
    kw = dict({"Chi2PDC": PDC, "Chi2SFGPDC": SFGPDC}[name], tPrecision=n)
    return getattr(nlm, name)(**kw), getattr(oracle, name)(**kw)


@pytest.mark.parametrize("in_time", [False, True])
@pytest.mark.parametrize("n", [128, 256, 512, 1024, 2048, 4096])
@pytest.mark.parametrize("name", ["Chi2PDC", "Chi2SFGPDC"])
def test_propagator_batches_match_oracle(nlm, oracle, name, n, in_time):
    med, ref = _media(nlm, oracle, name, n)
    modes = med._dims["nSignalModes"]
    # a smooth field of a few pulse lengths, so that no step amplifies the grid's edge frequencies
    t = np.fft.fftshift(np.linspace(-8, 8, n, endpoint=False))
    x = cases.noise(np.random.default_rng(n), 3 * n * modes, 0.1).reshape(3, modes, n) * np.exp(-t ** 2)
    x = x.reshape(3, -1)
    if in_time:
        x = np.fft.ifft(x.reshape(3, modes, n), axis=2).reshape(3, -1)
    want = ref.batch_signal_simulation(x, in_time)
    # few warps take half the points per thread up to 2048 points
    for rows in (ROWS, 1500):
        out = med.batchSignalSimulation(np.tile(x, (rows // 3, 1)), in_time)
        for k in range(3):
            assert cases.rel_l2(out[k], want[k]) < TOL
            assert np.array_equal(out[k], out[k + 3])


@pytest.mark.parametrize("n", [128, 512, 4096])
@pytest.mark.parametrize("name", [k for k in cases.CASES if k != "Chi3GNLSE"])
def test_every_solver_matches_oracle(nlm, oracle, name, n):
    """The DiffEq kernels (pump-driven solvers also with their propagator), in both domains."""
    kw = dict(cases.CASES[name], tPrecision=n)
    med, ref = getattr(nlm, name)(**kw), getattr(oracle, name)(**dict(cases.oracle_kwargs(name), tPrecision=n))
    fnl = name in cases.FULLY_NONLINEAR
    if not fnl:
        ref.run_pump_simulation()
    t = np.fft.fftshift(np.linspace(-8, 8, n, endpoint=False))
    modes = med._dims["nSignalModes"]
    x = cases.noise(np.random.default_rng(n), 2 * n * modes, 0.1).reshape(2, modes, n) * np.exp(-t ** 2)
    x = np.fft.ifft(x, axis=2).reshape(2, -1)
    want = ref.batch_signal_simulation(x, True) if fnl else ref.batch_signal_simulation(x, True, False)
    for use in ((-1,) if fnl else (0, 1)):
        med._set_schedule(use_propagator=use)
        rows = np.tile(x, (ROWS // 2, 1))
        out = med.batchSignalSimulation(rows, True)
        for k in range(2):
            assert cases.rel_l2(out[k], want[k]) < TOL
            assert np.array_equal(out[k], out[ROWS - 2 + k])


# every odd radix, alone and repeated, with each power-of-two part; then grids with a larger prime factor, in the
# convolution form (its smallest and largest L)
GENERAL = [70, 96, 100, 250, 294, 600, 1000, 1536, 2058, 4050, 66, 74, 502, 1022, 2042]


@pytest.mark.parametrize("n", GENERAL)
@pytest.mark.parametrize("name", ["Chi2PDC", "Chi2SFGPDC", "Chi2SHG", "Chi2SFGII", "Chi3GNLSE"])
def test_general_grids_match_oracle(nlm, oracle, name, n):
    """Grids that are not powers of two: batches (DiffEq and propagator) and full grids, in both domains."""
    kw = dict(cases.CASES[name], tPrecision=n)
    if name == "Chi3GNLSE":
        kw.update(zPrecision=2000, relativeLength=0.02, tMax=20)
    med, ref = getattr(nlm, name)(**kw), getattr(oracle, name)(**kw)
    fnl = name in cases.FULLY_NONLINEAR
    if not fnl:
        med.runPumpSimulation()
        ref.run_pump_simulation()
    modes = med._dims["nSignalModes"]
    t = np.fft.fftshift(np.linspace(-8, 8, n, endpoint=False))
    spec = cases.noise(np.random.default_rng(n), 2 * n * modes, 0.1).reshape(2, modes, n) * np.exp(-t ** 2)
    for in_time in (False, True):
        x = (np.fft.ifft(spec, axis=2) if in_time else spec).reshape(2, -1)
        want = ref.batch_signal_simulation(x, in_time) if fnl else ref.batch_signal_simulation(x, in_time, False)
        for use in ((-1,) if fnl else (0, 1)):
            med._set_schedule(use_propagator=use)
            out = med.batchSignalSimulation(x, in_time) if fnl else med.batchSignalSimulation(x, in_time, False)
            assert cases.rel_l2(out, want) < TOL
        med.runSignalSimulation(x[0], in_time)
        ref.run_signal_simulation(x[0], in_time)
        for m in range(modes):
            assert cases.rel_l2(med.signalTimes(m), ref.signal_time[m]) < TOL
            assert cases.rel_l2(med.signalFreqs(m), ref.signal_freq[m]) < TOL


@pytest.mark.parametrize("n", [66, 70, 250, 600, 1022, 1536, 2042, 4050])
def test_chi3_pump_march_on_general_grids(nlm, oracle, n):
    """The pump march (self-phase factor, dispersion pair per row) in the general and the convolution form."""
    kw = dict(relativeLength=1, nlLength=1, beta2=-1, beta3=0.1, pulseType=1, tMax=10, tPrecision=n, zPrecision=15)
    med, ref = nlm.Chi3(**kw), oracle.Chi3(**kw)
    med.runPumpSimulation()
    ref.run_pump_simulation()
    assert cases.rel_l2(med.pumpTime, ref.pump_time[0]) < TOL
    assert cases.rel_l2(med.pumpFreq, ref.pump_freq[0]) < TOL


@pytest.mark.parametrize("in_time", [False, True])
@pytest.mark.parametrize("n", [128, 256, 512, 1024, 2048, 4096])
def test_gnlse_matches_oracle(nlm, oracle, n, in_time):
    """One row per CTA (3 rows and the odd 100) and two rows per CTA (161 rows)."""
    kw = dict(cases.CASES["Chi3GNLSE"], tPrecision=n, zPrecision=2000, relativeLength=0.02, tMax=20)
    med, ref = nlm.Chi3GNLSE(**kw), oracle.Chi3GNLSE(**kw)
    med._set_cluster(0)
    t = np.fft.fftshift(np.linspace(-20, 20, n, endpoint=False))
    x = 1.5 / np.cosh(t)[None, :] + cases.noise(np.random.default_rng(n), 3 * n, 1e-3).reshape(3, n)
    x = x if in_time else np.fft.fft(x, axis=1)
    want = ref.batch_signal_simulation(x, in_time)
    for rows in (3, 161):
        out = med.batchSignalSimulation(np.tile(x, (54, 1))[:rows], in_time)
        for k in (0, 1, rows - 1):
            assert cases.rel_l2(out[k], want[k % 3]) < TOL


@pytest.mark.parametrize("n", [128, 256, 1024])
def test_one_step_media(nlm, oracle, n):
    """nZSteps = 1: no RK4 step, the dispersion pair alone."""
    kw = dict(relativeLength=1, nlLength=1, beta2=1, beta2s=0.5, beta1s=1, tMax=40, zPrecision=1, tPrecision=n)
    med, ref = nlm.Chi2PDC(**kw), oracle.Chi2PDC(**kw)
    assert med._dims["nZSteps"] == 1
    # dz is infinite for one step: the spectra of both are NaN in the same places
    x = cases.noise(np.random.default_rng(0), ROWS * n, 1.0).reshape(ROWS, n)
    for in_time in (False, True):
        with np.errstate(all="ignore"):
            want = ref.batch_signal_simulation(x[:2], in_time)
        out = med.batchSignalSimulation(x, in_time)[:2]
        assert np.array_equal(np.isnan(out), np.isnan(want))


@pytest.mark.parametrize("n", [128, 1024])
def test_ends_of_the_double_range(nlm, oracle, n):
    """Each row has its own exponent: rows near 1e-290 and 1e290, a zero row and rows with an infinite or a NaN
    value in one call."""
    med, ref = _media(nlm, oracle, "Chi2PDC", n)
    rng = np.random.default_rng(n)
    x = cases.noise(rng, ROWS * n, 1.0).reshape(ROWS, n)
    scale = np.ones(ROWS)
    scale[0], scale[1], scale[2], scale[3] = 1e-290, 1e290, 0.0, 2.0 ** -1000
    x *= scale[:, None]
    x[4, n // 3] = np.inf
    x[5, 1] = np.nan
    out = med.batchSignalSimulation(x)
    want = ref.batch_signal_simulation(x[6:9])
    for k in range(3):
        assert cases.rel_l2(out[6 + k], want[k]) < TOL
    for k in (0, 1, 3):
        one = ref.batch_signal_simulation((x[k] / scale[k])[None])[0]
        assert cases.rel_l2(out[k] / scale[k], one) < TOL
    assert np.all(out[2] == 0)
    assert not np.any(np.isfinite(out[4])) and np.all(np.isnan(out[5]))
