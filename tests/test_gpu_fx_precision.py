"""Rounding of the block fixed-point marches on powers of two against the same steps in extended precision (numpy's long
double: 80 bits or more), beside that of the numpy oracle's FP64 transforms.

The factor tables are the oracle's doubles on both sides, and the pump of Chi2PDC keeps its shape, so that what differs is
the rounding of transforms and RK4 steps.  The engine may be no further from the extended values than the FP64 oracle.
On other grids the products of the dispersion factors and 1/N, rounded in the tables of all the engine's kernels and the
same at every step, add to that (600 points, 100 steps: 8.8e-15 against the oracle's 7.4e-15).
"""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

C = np.clongdouble


def _fft(x):
    return np.fft.fft(x.astype(C), axis=-1)


def _ifft(x):
    return np.fft.ifft(x.astype(C), axis=-1)


def _pump_chi3(ref):
    """Rows of the pump march (solvers/Chi3.cpp:41-70) in extended precision, without an intensity profile."""
    step, d = ref.disp_step_pump[0].astype(C), ref.disp_pump[0]
    gain = C((ref.dzp / ref.dz) * ref.nl_step[0])
    row = _ifft(_fft(ref.envelope[0]) * np.exp((0.5j * ref.dzp) * d).astype(C))
    rows = [row]
    for _ in range(1, ref.n_z_steps_p):
        f = _fft(row * np.exp(gain * np.abs(row) ** 2)) * step
        row = _ifft(f)
        rows.append(row)
    rows[-1] = _ifft(f * np.exp((-0.5j * ref.dzp) * d).astype(C))
    return np.array(rows)


def _march(ref, x, rhs):
    """Last spectrum (src/_NonlinearMedium.hpp:160-239) of the input spectra x in extended precision; rhs(i, s, a): the
    derivative at sub-step s of step i."""
    d, step = ref.disp_sign[0], ref.disp_step_sign[0].astype(C)
    a = _ifft(x.astype(C) * np.exp((0.5j * ref.dz) * d).astype(C))
    for i in range(1, ref.n_z_steps):
        k1 = rhs(i, 0, a)
        k2 = rhs(i, 1, a + k1 / 2)
        k3 = rhs(i, 1, a + k2 / 2)
        k4 = rhs(i, 2, a + k3)
        f = _fft(a + (k1 + 2 * k2 + 2 * k3 + k4) / 6) * step
        a = _ifft(f)
    return f * np.exp((-0.5j * ref.dz) * d).astype(C)


def _off(y, exact):
    return float(np.linalg.norm((np.asarray(y) - exact).astype(complex)) / np.linalg.norm(exact.astype(complex)))


@pytest.mark.parametrize("n", [128, 512, 2048])
def test_chi3_pump_and_signal(nlm, oracle, n):
    kw = dict(relativeLength=1, nlLength=1, beta2=-1, pulseType=1, tMax=20, tPrecision=n, zPrecision=100,
              intensityProfile=1)
    med, ref = nlm.Chi3(**kw), oracle.Chi3(**kw)
    med.runPumpSimulation()
    ref.run_pump_simulation()
    pump = _pump_chi3(ref)
    assert _off(med.pumpTime, pump) <= _off(ref.pump_time[0], pump)
    x = cases.noise(np.random.default_rng(n), n, 1e-3)
    g = C(ref.nl_step[0])

    def rhs(i, s, a):
        p = pump[2 * i - 2 + s]
        return g * (2 * np.abs(p) ** 2 * a + p ** 2 * np.conj(a))

    exact = _march(ref, x, rhs)
    med.runSignalSimulation(x, False)
    ref.run_signal_simulation(x, False)
    assert _off(med.signalFreqs(0)[-1], exact) <= _off(ref.signal_freq[0][-1], exact)


@pytest.mark.parametrize("n", [128, 512, 1024])
def test_pdc_signal_and_rows(nlm, oracle, n):
    """One propagation with its grids (a cluster) and 40 rows (one CTA each, with the RK4
    matrices), two of which are compared."""
    t = np.fft.fftshift(np.linspace(-20, 20, n, endpoint=False))
    pump = np.exp(-t ** 2 / 2) * (1 + 0.3j)
    kw = dict(relativeLength=1, nlLength=0.5, beta2=0, beta2s=0.5, beta1s=2, tMax=20, tPrecision=n, zPrecision=50,
              customPump=pump, intensityProfile=1)
    med, ref = nlm.Chi2PDC(**kw), oracle.Chi2PDC(**kw)
    med.runPumpSimulation()
    ref.run_pump_simulation()
    x = cases.noise(np.random.default_rng(n), 40 * n, 1.0).reshape(40, n)
    p, g = pump.astype(C), C(ref.nl_step[0])
    exact = _march(ref, x[:2], lambda i, s, a: g * ref.pol(i)[s] * p * np.conj(a))
    want = ref.batch_signal_simulation(x[:2], False, False)
    med._set_cluster(0)
    out = med.batchSignalSimulation(x, False, False)[:2]
    assert _off(out, exact) <= _off(want, exact)
    med._set_cluster(1)
    med.runSignalSimulation(x[0], False)
    assert _off(med.signalFreqs(0)[-1], exact[0]) <= _off(want[0], exact[0])
