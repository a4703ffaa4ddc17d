"""Media, fields and calls at the edges of the block fixed-point kernels (csrc/nlm_fx.cuh, csrc/nlm_spread.cuh)."""
import numpy as np
import pytest

import cases

pytestmark = pytest.mark.gpu

GNLSE = dict(nlLength=1, selfSteepLength=5, fr=0.18, fb=0.21, tau1=0.0155, tau2=0.2165, tau3=0.4, beta2=-1, beta3=0.05)
PDC = dict(relativeLength=1, nlLength=0.5, beta2=1, beta2s=0.5, beta1s=2, tMax=40, zPrecision=10)
SFG = dict(relativeLength=1, nlLength=0.8, nlLengthOrig=1.2, beta2=0.5, beta2s=-0.3, beta2o=0.2, beta1s=1, tMax=20,
           zPrecision=10)


# ---- media without integer tables: FP64 kernels in every form -----------------------------------------------------

@pytest.mark.parametrize("n", [128, 512, 1024, 2048, 4096])
def test_one_step_gnlse(nlm, oracle, n):
    """One z step has an infinite step length, and no integer tables: full grids and few-row batches run the FP64
    kernels (never one point per thread), NaN where the oracle is."""
    kw = dict(GNLSE, relativeLength=1, tMax=10, tPrecision=n, zPrecision=1)
    med, ref = nlm.Chi3GNLSE(**kw), oracle.Chi3GNLSE(**kw)
    assert med._dims["nZSteps"] == 1
    x = cases.noise(np.random.default_rng(n), 3 * n, 1.0).reshape(3, n)
    for in_time in (False, True):
        med.runSignalSimulation(x[0], in_time)
        assert med._last_schedule()["R"] > 1
        out = med.batchSignalSimulation(x, in_time)
        assert med._last_schedule()["R"] > 1
        with np.errstate(all="ignore"):
            ref.run_signal_simulation(x[0], in_time)
            want = ref.batch_signal_simulation(x, in_time)
        assert np.array_equal(np.isnan(out), np.isnan(want))
        assert np.array_equal(np.isnan(med.signalFreq), np.isnan(ref.signal_freq[0]))
    import torch
    from multimodenonlinearoptics_gb300.autograd import propagate_gnlse
    with pytest.raises(ValueError):
        propagate_gnlse(med, torch.zeros((1, n), dtype=torch.complex128, device="cuda"))


@pytest.mark.parametrize("interval", [0, 4])
@pytest.mark.parametrize("n", [128, 1024, 2048, 4096])
@pytest.mark.parametrize("name", ["Chi2PDC", "Chi3GNLSE"])
def test_dispersion_that_is_not_finite(nlm, name, n, interval):
    """A NaN dispersion parameter (an optimiser's step) leaves no integer tables: full grids, batches and gradients come
    back NaN from the FP64 kernels."""
    import torch
    from multimodenonlinearoptics_gb300.autograd import propagate_gnlse, propagate_pdc
    nan = float("nan")
    if name == "Chi2PDC":
        med = nlm.Chi2PDC(**dict(PDC, beta2s=nan, tPrecision=n))
    else:
        med = nlm.Chi3GNLSE(**dict(GNLSE, relativeLength=1, beta2=nan, tMax=10, tPrecision=n, zPrecision=10))
    assert med._dims["nZSteps"] > 9
    x = cases.noise(np.random.default_rng(n), 2 * n, 0.1).reshape(2, n)
    med.runSignalSimulation(x[0])
    assert med._last_schedule()["R"] > 1 and np.all(np.isnan(med.signalFreq))
    out = med.batchSignalSimulation(x, True)
    assert med._last_schedule()["R"] > 1 and np.all(np.isnan(out))
    xt = torch.tensor(x, device="cuda").requires_grad_()
    if name == "Chi2PDC":
        pump = torch.ones(n, dtype=torch.complex128, device="cuda")
        y = propagate_pdc(med, xt, pump, torch.ones(med._dims["nZSteps"], dtype=torch.float64, device="cuda"), interval)
    else:
        y = propagate_gnlse(med, xt, interval)
    grad, = torch.autograd.grad(torch.sum(torch.abs(y) ** 2), xt)
    assert med._last_schedule()["R"] > 1
    assert torch.isnan(y).all() and torch.isnan(grad).all()


def test_ragged_set_with_a_medium_without_tables(nlm, oracle):
    """The planner gives a medium without integer tables no one-point-per-thread slot; its neighbours are unaffected."""
    media, refs, xs = [], [], []
    for k, n in enumerate((1024, 512, 1024, 2048)):
        kw = dict(SFG, tPrecision=n, beta2s=float("nan") if k in (0, 3) else -0.3)
        media.append(nlm.Chi2SFG(**kw))
        refs.append(oracle.Chi2SFG(**kw))
        xs.append(cases.noise(np.random.default_rng(k), n, 0.1))
        media[k].runPumpSimulation()
    out = nlm.ragged_batch(media, xs)
    for k in (0, 3):
        assert np.all(np.isnan(out[k]))
    for k in (1, 2):
        refs[k].run_pump_simulation()
        want = refs[k].batch_signal_simulation(xs[k][None], False, False)[0]
        assert cases.rel_l2(out[k].ravel(), want.ravel()) < 1e-12   # 20 steps, as in test_gpu_fx.py


# ---- rows that share a CTA ----------------------------------------------------------------------------------------

@pytest.mark.parametrize("in_time", [False, True])
@pytest.mark.parametrize("n", [128, 512, 1024, 4096])
def test_paired_rows_of_very_different_norm(nlm, oracle, n, in_time):
    """Two GNLSE rows per CTA, one ten decades below the other: each keeps its own exponent to the last step (a row
    rounded with its partner's would be off by 1e10 x 2^-60 = 1e-8), and repeated calls agree bit by bit.  40 steps:
    tolerance as in test_gpu_fx.py."""
    kw = dict(cases.CASES["Chi3GNLSE"], tPrecision=n, zPrecision=2000, relativeLength=0.02, tMax=20)
    med, ref = nlm.Chi3GNLSE(**kw), oracle.Chi3GNLSE(**kw)
    med._set_cluster(0)
    rows, rng = 331, np.random.default_rng(n)   # 165 pairs and a last row whose partner is idle
    t = np.fft.fftshift(np.linspace(-20, 20, n, endpoint=False))
    x = rng.uniform(0.5, 1.5, (rows, 1)) / np.cosh(t)[None, :] + cases.noise(rng, rows * n, 1e-3).reshape(rows, n)
    x[0:100:2] *= 1e-10   # the pair's first row, then its second
    x[101:200:2] *= 1e-10
    x = x if in_time else np.fft.fft(x, axis=1)
    out = med.batchSignalSimulation(x, in_time)
    pick = [0, 1, 2, 100, 101, 198, 199, 200, 329, 330]
    want = ref.batch_signal_simulation(x[pick], in_time)
    for k, p in enumerate(pick):
        assert cases.rel_l2(out[p], want[k]) < 1e-12
    for _ in range(4):
        assert np.array_equal(med.batchSignalSimulation(x, in_time), out)


# ---- spectra that no transform has rounded ------------------------------------------------------------------------

def _wide_spectrum(n, rows):
    """Bins from 1 down to 1e-25, far below the last bit of the row's norm."""
    rng = np.random.default_rng(n)
    phase = np.exp(2j * np.pi * rng.uniform(size=(rows, n)))
    return phase * 10.0 ** (-25 * np.abs(np.fft.fftfreq(n)) * 2)[None, :]


@pytest.mark.parametrize("n", [100, 128, 600, 1022, 1024, 4096])
@pytest.mark.parametrize("name", ["Chi2PDC", "Chi2SFG", "Chi3GNLSE"])
def test_first_row_of_a_spectrum_keeps_every_bin(nlm, name, n):
    """Row 0 of the spectrum grid is the input spectrum times a phase, bin by bin.  Modulus to 1.2e-15: the factor's
    parts (2.2e-16), its 1/N, the product (2.2e-16), the N, and the test's own two moduli (2.2e-16 each) and ratio."""
    kw = {"Chi2PDC": PDC, "Chi2SFG": SFG,
          "Chi3GNLSE": dict(GNLSE, relativeLength=1, tMax=10, zPrecision=10)}[name]
    med = getattr(nlm, name)(**dict(kw, tPrecision=n))
    x = _wide_spectrum(n, 1)[0]
    for cluster in (0, 1):
        med._set_cluster(cluster)
        med.runSignalSimulation(x, False)
        got = np.abs(med.signalFreqs(0)[0])
        assert np.max(np.abs(got / np.abs(x) - 1)) < 1.2e-15


@pytest.mark.parametrize("rows", [3, 161])
@pytest.mark.parametrize("n", [128, 600, 1022, 1024, 4096])
def test_gnlse_spectrum_keeps_every_bin(nlm, n, rows):
    """A nearly linear medium: the state's spectrum takes a phase per step and keeps every bin's modulus.  A step rounds
    its factor (3.3e-16 in all), sum, scaling and product (1.1, 1.1 and 2.2e-16), 41 times at most: 3.2e-14."""
    med = nlm.Chi3GNLSE(**dict(GNLSE, nlLength=1e30, selfSteepLength=1e30, relativeLength=1, tMax=10, tPrecision=n,
                               zPrecision=40))
    assert med._dims["nZSteps"] <= 41
    med._set_cluster(0)
    x = _wide_spectrum(n, rows)
    out = med.batchSignalSimulation(x)
    assert np.max(np.abs(np.abs(out) / np.abs(x) - 1)) < 3.2e-14


# ---- fields that a butterfly gathers in one point -----------------------------------------------------------------

@pytest.mark.parametrize("in_time", [False, True])
@pytest.mark.parametrize("n", [70, 80, 84, 98, 112, 140, 280, 294, 320, 336, 392, 448, 1120, 1280, 1344, 2058, 2240, 3920])
def test_single_bins_on_general_grids(nlm, oracle, n, in_time):
    """Plane waves (and single bins), whose transform is one point that sums all others, with norms just below powers of
    two and a mode of the other kind beside them: grids whose last odd pass runs at the highest norm, and others.
    Tolerance as in test_gpu_fx.py (20 steps)."""
    kw = dict(SFG, tPrecision=n)
    med, ref = nlm.Chi2SFG(**kw), oracle.Chi2SFG(**kw)
    med.runPumpSimulation()
    ref.run_pump_simulation()
    bins = sorted({0, 1, 2, 3, 5, 7, n // 7, n // 5, n // 4, n // 2, n - 1})
    t = np.arange(n)
    x = np.zeros((3 * len(bins), 2, n), complex)
    for i, k in enumerate(bins):
        for q, norm in enumerate((0.999, 0.71, 1.99)):
            x[3 * i + q, 0] = norm * np.exp(2j * np.pi * k * t / n) / np.sqrt(n)
            x[3 * i + q, 1, k] = norm
    x = x.reshape(len(x), -1)
    want = ref.batch_signal_simulation(x, in_time, False)
    for use in (0, 1):
        med._set_schedule(use_propagator=use)
        out = med.batchSignalSimulation(x, in_time, False)
        for k in range(len(x)):
            assert cases.rel_l2(out[k], want[k]) < 1e-12


@pytest.mark.parametrize("n", [70, 80, 294, 448])
def test_greens_functions_of_small_general_grids(nlm, oracle, n):
    """Impulses in every bin."""
    kw = dict(PDC, tPrecision=n)
    c, s = nlm.Chi2PDC(**kw).computeGreensFunction()
    cr, sr = oracle.Chi2PDC(**kw).compute_greens_function()
    assert cases.rel_l2_pair(c, s, cr, sr) < 1e-12


# ---- rounding of the convolution form -----------------------------------------------------------------------------

@pytest.mark.parametrize("n", [66, 134, 502, 662, 1018, 1022, 2038])
def test_convolution_form_rounds_like_fp64(nlm, n):
    """No pump and no dispersion: 1000 transform pairs leave the field where it is, and their errors, the same at every
    step, add up.  A pair of FP64 transforms rounds by 1.2e-16 of the norm, the factor 1/N by up to 1.1e-16: 2.3e-16 a
    step."""
    kw = dict(relativeLength=1, nlLength=1, beta2=0, beta2s=0, tMax=20, tPrecision=n, zPrecision=1001)
    med = nlm.Chi2PDC(customPump=np.zeros(n, complex), **kw)
    med.runPumpSimulation()
    for kind in ("noise", "peak"):
        x = cases.noise(np.random.default_rng(n), n, 1.0)
        if kind == "peak":
            x[n // 3] = 1e6
        med.runSignalSimulation(x, True)
        for row in (250, 999):
            assert cases.rel_l2(med.signalTime[row], x) < 2.3e-16 * row


@pytest.mark.parametrize("n", [600, 1536, 2646, 3402, 3750, 4050])
def test_mixed_radices_round_like_fp64(nlm, n):
    """The same on grids of many odd factors.  A pair of FP64 transforms in up to seven passes rounds by 2.5e-16 of the
    norm, the factor 1/N by up to 1.1e-16: 3.6e-16 a step."""
    kw = dict(relativeLength=1, nlLength=1, beta2=0, beta2s=0, tMax=20, tPrecision=n, zPrecision=401)
    med = nlm.Chi2PDC(customPump=np.zeros(n, complex), **kw)
    med.runPumpSimulation()
    x = cases.noise(np.random.default_rng(n), n, 1.0)
    med.runSignalSimulation(x, True)
    for row in (100, 399):
        assert cases.rel_l2(med.signalTime[row], x) < 3.6e-16 * row


# ---- tables of zeros ----------------------------------------------------------------------------------------------

@pytest.mark.parametrize("n", [128, 512, 600, 2048])
def test_gnlse_without_nonlinearity(nlm, oracle, n):
    """Infinite nonlinear and self-steepening lengths: a steepening table of zeros is a table, and few rows keep their
    one-point-per-thread clusters.  40 steps: tolerance as in test_gpu_fx.py."""
    kw = dict(GNLSE, nlLength=cases.INF, selfSteepLength=cases.INF, relativeLength=1, tMax=10, tPrecision=n,
              zPrecision=40)
    med, ref = nlm.Chi3GNLSE(**kw), oracle.Chi3GNLSE(**kw)
    x = cases.noise(np.random.default_rng(n), 3 * n, 1.0).reshape(3, n)
    out = med.batchSignalSimulation(x)
    if n in (512, 2048):
        assert med._last_schedule()["R"] == 1
    assert cases.rel_l2(out, ref.batch_signal_simulation(x, False)) < 1e-12


# ---- exchanges that do not arrive ---------------------------------------------------------------------------------

def _medium(nlm, name, n, cluster=1, **more):
    kw = {"Chi2PDC": PDC, "Chi2SFG": SFG, "Chi3": dict(relativeLength=1, nlLength=1, beta2=-1, tMax=20, zPrecision=15),
          "Chi3GNLSE": dict(GNLSE, relativeLength=1, tMax=10, zPrecision=10)}[name]
    med = getattr(nlm, name)(**dict(kw, tPrecision=n, **more))
    med._set_cluster(cluster)
    return med


def _signal(nlm, name, n, cluster=1):
    med = _medium(nlm, name, n, cluster)
    if name != "Chi3GNLSE":
        med.runPumpSimulation()
        assert np.all(np.isfinite(med.pumpTime))   # a deferred pump march runs now
    x = cases.noise(np.random.default_rng(n), n, 0.1)

    def call():
        med.runSignalSimulation(x)
        return np.concatenate([med.signalFreq.ravel(), med.signalTime.ravel()])
    return med, call


def _batch(nlm, name, n):
    med = _medium(nlm, name, n)
    x = cases.noise(np.random.default_rng(n), 3 * n, 0.1).reshape(3, n)
    if name == "Chi3GNLSE":
        return med, lambda: med.batchSignalSimulation(x).copy()
    med.runPumpSimulation()
    return med, lambda: med.batchSignalSimulation(x, False, False).copy()


def _pump(nlm, n, cluster):
    """The Chi3 pump march: deferred and read alone (cluster mode 1 on 512 points), or run at once."""
    med = _medium(nlm, "Chi3", n, cluster)

    def call():
        med.runPumpSimulation()
        return med.pumpTime.copy()
    return med, call


def _gradient(nlm, name, n, interval, part):
    """The forward or the backward pass of a gradient under the limit."""
    import torch
    from multimodenonlinearoptics_gb300.autograd import propagate_gnlse, propagate_pdc
    med = _medium(nlm, name, n)
    x = torch.tensor(cases.noise(np.random.default_rng(n), 2 * n, 0.1).reshape(2, n), device="cuda").requires_grad_()
    pump = torch.tensor(np.fft.fft(np.exp(-np.fft.fftshift(np.linspace(-8, 8, n)) ** 2)), device="cuda")
    poling = torch.ones(med._dims["nZSteps"], dtype=torch.float64, device="cuda")
    limit = [-1]

    def call():
        med._set_exchange_limit(limit[0] if part == "forward" else -1)
        y = propagate_gnlse(med, x, interval) if name == "Chi3GNLSE" else propagate_pdc(med, x, pump, poling, interval)
        med._set_exchange_limit(limit[0])
        grad, = torch.autograd.grad(torch.sum(torch.abs(y) ** 2), x)
        return torch.cat([y, grad]).detach().cpu().numpy()
    return med, call, limit


FORMS = [("signal", "Chi2PDC", 128, 1), ("signal", "Chi2PDC", 1024, 1), ("signal", "Chi2PDC", 2048, 1),
         ("signal", "Chi2PDC", 4096, 1), ("signal", "Chi2PDC", 4096, 3), ("signal", "Chi2SFG", 512, 1),
         ("signal", "Chi2SFG", 2048, 1), ("signal", "Chi3", 512, 1), ("signal", "Chi3", 512, 3),
         ("signal", "Chi3GNLSE", 512, 1), ("signal", "Chi3GNLSE", 4096, 1), ("batch", "Chi2PDC", 512, 1),
         ("batch", "Chi3GNLSE", 2048, 1), ("pump", "Chi3", 512, 1), ("pump", "Chi3", 2048, 3)]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: "-".join(map(str, f)))
def test_exchange_that_gives_up(nlm, form):
    """With a limit of no polls every exchange gives up at its first wait: the kernel still returns, the call raises, and
    the next call with the default limit gives what the one before gave, bit by bit."""
    kind, name, n, cluster = form
    med, call = (_signal(nlm, name, n, cluster) if kind == "signal" else
                 _batch(nlm, name, n) if kind == "batch" else _pump(nlm, n, cluster))
    want = call()
    for _ in range(2):
        med._set_exchange_limit(0)
        with pytest.raises(RuntimeError, match="exchange"):
            call()
        med._set_exchange_limit()
        assert np.array_equal(call(), want, equal_nan=True)


def test_deferred_pump_march_that_gives_up(nlm):
    """A pump march that runs beside a signal and fails with it stays deferred: the next signal runs it again."""
    med = _medium(nlm, "Chi3", 512)
    x = cases.noise(np.random.default_rng(1), 512, 0.1)
    med.runPumpSimulation()
    med.runSignalSimulation(x)
    assert med._last_schedule()["grid"] == 8
    want = np.concatenate([med.pumpTime.ravel(), med.signalFreq.ravel(), med.signalTime.ravel()])
    med.runPumpSimulation()
    med._set_exchange_limit(0)
    with pytest.raises(RuntimeError, match="exchange"):
        med.runSignalSimulation(x)
    med._set_exchange_limit()
    med.runSignalSimulation(x)
    assert med._last_schedule()["grid"] == 8
    assert np.array_equal(np.concatenate([med.pumpTime.ravel(), med.signalFreq.ravel(), med.signalTime.ravel()]), want)


@pytest.mark.parametrize("part", ["forward", "backward"])
@pytest.mark.parametrize("name,n,interval,ctas", [("Chi2PDC", 512, 0, 12), ("Chi2PDC", 512, 6, 8), ("Chi2PDC", 512, 6, 12),
                                                  ("Chi2PDC", 512, 6, 16), ("Chi2PDC", 2048, 6, 12),
                                                  ("Chi3GNLSE", 1024, 0, 12),
                                                  ("Chi3GNLSE", 4096, 0, 12)])
def test_gradient_whose_exchange_gives_up(nlm, monkeypatch, name, n, interval, ctas, part):
    """The same for the reverse sweeps; a forward pass that failed leaves nothing to differentiate."""
    if (n, interval, part) == (2048, 6, "forward"):
        pytest.skip("checkpointed forwards at 2048 points run four points per thread, without these exchanges")
    monkeypatch.setenv("NLM_ADJOINT_CTAS", str(ctas))
    med, call, limit = _gradient(nlm, name, n, interval, part)
    want = call()
    limit[0] = 0
    with pytest.raises(RuntimeError, match="exchange"):
        call()
    if part == "forward":
        import torch
        g = torch.zeros((2, n), dtype=torch.complex128, device="cuda")
        with pytest.raises(RuntimeError, match="no adjoint forward"):
            nlm._check(nlm._lib.nlm_adjoint_backward(med._h(), g.data_ptr(), g.data_ptr(), None, None))
    limit[0] = -1
    assert np.array_equal(call(), want, equal_nan=True)


def test_ragged_set_whose_exchange_gives_up(nlm):
    media = [_medium(nlm, "Chi2SFG", n) for n in (512, 1024, 2048, 512)]
    xs = [cases.noise(np.random.default_rng(k), m._dims["nFreqs"], 0.1) for k, m in enumerate(media)]
    for m in media:
        m.runPumpSimulation()
    want = [o.copy() for o in nlm.ragged_batch(media, xs)]
    media[2]._set_exchange_limit(0)
    with pytest.raises(RuntimeError, match="exchange"):
        nlm.ragged_batch(media, xs)
    media[2]._set_exchange_limit()
    for a, b in zip(nlm.ragged_batch(media, xs), want):
        assert cases.rel_l2(a, b) < 1e-12   # a repeated call may run with its matrices (test_gpu_ragged.py)


def test_each_medium_sees_its_own_failed_exchange(nlm):
    """Media on threads of their own, one of which gives up its exchanges: it raises on every call, and the others never
    do and keep their results bit by bit."""
    import threading
    media = [_signal(nlm, "Chi2PDC", n) for n in (512, 512, 128, 1024)]
    want = [call() for _, call in media]
    media[0][0]._set_exchange_limit(0)
    raised, wrong = [0] * len(media), []
    start = threading.Barrier(len(media))

    def work(k):
        start.wait()
        for _ in range(100):
            try:
                if not np.array_equal(media[k][1](), want[k]):
                    wrong.append(k)
            except RuntimeError:
                raised[k] += 1

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(media))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert raised == [100, 0, 0, 0] and not wrong
    media[0][0]._set_exchange_limit()
    assert np.array_equal(media[0][1](), want[0])


def test_failed_exchange_of_a_ragged_set_stays_with_it(nlm):
    """The flag of a set's medium is read and cleared by the set's call; a call of another medium after it succeeds, and
    so does the medium's own next call."""
    media = [_medium(nlm, "Chi2SFG", 512), _medium(nlm, "Chi2SFG", 512)]
    other, call = _signal(nlm, "Chi2PDC", 512)
    want = call()
    x = cases.noise(np.random.default_rng(0), 512, 0.1)
    for m in media:
        m.runPumpSimulation()
        m._set_exchange_limit(0)
    with pytest.raises(RuntimeError, match="exchange"):
        nlm.ragged_batch(media, [x, x])
    assert np.array_equal(call(), want, equal_nan=True)
    for m in media:
        m._set_exchange_limit()
        m.runSignalSimulation(x)


# ---- four modes in one transform ----------------------------------------------------------------------------------

@pytest.mark.parametrize("n", [128, 256, 512, 1024])
@pytest.mark.parametrize("name", ["Chi2SFGII", "Chi2SHGOPA"])
def test_four_modes_in_one_transform(nlm, oracle, name, n):
    """Clusters that transform four modes together, two at a time (four CTAs, and eight for full grids of 1024 points),
    with norms ten decades apart: every mode's field stays in its place and keeps its own exponent.  At most 111
    steps of two evaluations that round by about 1e-15 of the norm a step, times a growth of a few: 1e-12, per mode at
    the scale of the largest, which feeds the others."""
    kw = dict(cases.CASES[name], tPrecision=n, tMax=20)
    if name != "Chi2SFGII":   # whose keyword zPrecision binds to another slot (solvers/Chi2SFGII.cpp:98-106)
        kw["zPrecision"] = 10
    med, ref = getattr(nlm, name)(**kw), getattr(oracle, name)(**kw)
    fnl = name in cases.FULLY_NONLINEAR
    if not fnl:
        med.runPumpSimulation()
        ref.run_pump_simulation()
    assert med._dims["nSignalModes"] == 4 and med._dims["nZSteps"] == ref.n_z_steps
    x = cases.noise(np.random.default_rng(n), 8 * n, 0.3).reshape(2, 4, n)
    x[0, 1] *= 1e-5
    x[0, 3] *= 1e-10
    x[1, :2] *= 1e-10
    x = x.reshape(2, -1)
    for in_time in (False, True):
        args = (in_time,) if fnl else (in_time, False)
        out = med.batchSignalSimulation(x, *args)
        assert med._last_schedule()["R"] == 1 and med._last_schedule()["grid"] == 8
        want = ref.batch_signal_simulation(x, *args)
        for k in range(2):
            assert cases.rel_l2(out[k], want[k]) < 1e-12
        med.runSignalSimulation(x[0], in_time)
        ref.run_signal_simulation(x[0], in_time)
        assert med._last_schedule()["grid"] == (8 if n == 1024 else 4)
        size = max(np.linalg.norm(f) for f in ref.signal_freq)
        for m in range(4):
            assert np.linalg.norm(med.signalFreqs(m) - ref.signal_freq[m]) < 1e-12 * size
