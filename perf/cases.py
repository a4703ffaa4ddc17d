"""Performance cases of the engine: what its users have it compute, at the sizes they use.

The sizes come from the repository's workloads (multimodenonlinearoptics_gb300/workloads.py and the
benchmark): single propagations that keep their whole grids, Green's functions on power-of-two and on
other even grids, batches of realisations, ragged sets of media, gradients.  `prepare` builds the
media and inputs a program has before the call, `run` makes the calls, and `exact` evaluates the same
split-step equations with plain torch and numpy in double precision.
"""

import math

import numpy as np
import torch

from multimodenonlinearoptics_gb300 import nonlinearmedium as nlm
from multimodenonlinearoptics_gb300.autograd import propagate_gnlse, propagate_pdc


def listed():
    return [
        # smallest call: one signal through a PDC medium whose pump is kept, full grids read back (an interactive
        # parameter scan on a coarse grid)
        {"name": "pdc_signal_n128", "kind": "signal", "n": 128, "zp": 50},
        # soliton pump march and the noise signal riding on it, on the grid of the Chi3 benchmark workload
        {"name": "chi3_pump_signal_n512", "kind": "chi3", "n": 512, "zp": 200},
        # supercontinuum: one GNLSE propagation with its whole grids
        {"name": "gnlse_signal_n2048", "kind": "gnlse_signal", "n": 2048, "steps": 300},
        # Green's function of a coarse grid (design scans over poling patterns)
        {"name": "pdc_green_n128", "kind": "pdc_green", "n": 128, "zp": 100},
        # Green's function on an even grid that is not a power of two
        {"name": "pdc_green_n600", "kind": "pdc_green", "n": 600, "zp": 100},
        # the Green's-function benchmark workload: 2048 impulses, 1000 steps
        {"name": "pdc_green_n1024", "kind": "pdc_green", "n": 1024, "zp": 500},
        # two coupled modes: Green's function of simultaneous sum-frequency generation and amplification
        {"name": "sfgpdc_green_n256", "kind": "sfgpdc_green", "n": 256, "zp": 300},
        # a set of media of different grids and lengths with new pumps, one spectrum through each
        {"name": "sfg_ragged_24", "kind": "ragged", "n": 2048, "media": 24, "steps": 1200},
        # depleted-pump second-harmonic generation, a batch of noisy inputs (two modes)
        {"name": "shg_batch_256_n512", "kind": "shg_batch", "n": 512, "zp": 100, "rows": 256},
        # batch of supercontinuum realisations on the grid of the GNLSE benchmark workload
        {"name": "gnlse_batch_1024_n4096", "kind": "gnlse_batch", "n": 4096, "steps": 110, "rows": 1024},
        # gradient of a PDC medium in its input, pump spectrum and poling profile (inverse design)
        {"name": "pdc_grad_n512", "kind": "pdc_grad", "n": 512, "zp": 1000, "rows": 1},
        # gradient of a supercontinuum band energy for a few realisations
        {"name": "gnlse_grad_16_n1024", "kind": "gnlse_grad", "n": 1024, "steps": 110, "rows": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _even(rng, lo, hi):
    """An even grid: a power of two (the common choice) or any even size."""
    if rng.random() < 0.6:
        return 2 ** rng.randint(int(math.log2(lo)), int(math.log2(hi)))
    return 2 * _log_int(rng, lo // 2, hi // 2)


def draw(rng):
    kind = rng.choice(["signal", "chi3", "gnlse_signal", "pdc_green", "sfgpdc_green", "ragged", "shg_batch", "gnlse_batch",
                       "pdc_grad", "gnlse_grad"])
    if kind == "signal":
        return {"kind": kind, "n": _even(rng, 64, 4096), "zp": _log_int(rng, 20, 500)}
    if kind == "chi3":
        return {"kind": kind, "n": _even(rng, 64, 2048), "zp": _log_int(rng, 50, 400)}
    if kind == "gnlse_signal":
        return {"kind": kind, "n": _even(rng, 512, 4096), "steps": _log_int(rng, 40, 500)}
    if kind == "pdc_green":
        n = _even(rng, 64, 1024)
        return {"kind": kind, "n": n, "zp": _log_int(rng, 20, 120 if n & (n - 1) else 500)}
    if kind == "sfgpdc_green":
        n = _even(rng, 64, 512)
        return {"kind": kind, "n": n, "zp": _log_int(rng, 20, 120 if n & (n - 1) else 300)}
    if kind == "ragged":
        return {"kind": kind, "n": 2 ** rng.randint(8, 11), "media": _log_int(rng, 2, 32), "steps": _log_int(rng, 100, 1200)}
    if kind == "shg_batch":
        return {"kind": kind, "n": _even(rng, 64, 1024), "zp": _log_int(rng, 20, 100), "rows": _log_int(rng, 1, 512)}
    if kind == "gnlse_batch":
        return {"kind": kind, "n": 2 ** rng.randint(9, 12), "steps": _log_int(rng, 30, 110), "rows": _log_int(rng, 8, 1024)}
    if kind == "pdc_grad":
        return {"kind": kind, "n": 2 ** rng.randint(7, 11), "zp": _log_int(rng, 50, 500), "rows": _log_int(rng, 1, 16)}
    return {"kind": kind, "n": 2 ** rng.randint(10, 12), "steps": _log_int(rng, 30, 110), "rows": _log_int(rng, 1, 200)}


# ------------------------------------------------------------------------------------------------
# Inputs, all from the seed: host arrays and constructor keywords
# ------------------------------------------------------------------------------------------------

def _tau(n, t_max):
    return np.fft.fftshift(np.linspace(-t_max, t_max, n, endpoint=False))


def _noise(rng, shape, sigma):
    return (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)) * sigma / np.sqrt(2)


def _pdc_medium(rng, n, zp, poled=True):
    """Degenerate parametric amplification with a chirped Gaussian pump; 2 zp steps."""
    kw = dict(relativeLength=1, nlLength=0.5, beta2=1, beta2s=0.5, beta1=0, beta1s=2, beta3=0, beta3s=0.1, diffBeta0=0,
              tMax=40, tPrecision=n, zPrecision=zp)
    t = _tau(n, 40)
    pump = np.exp(-t ** 2 * (0.5 + 0.1j * rng.uniform(-1, 1)) / rng.uniform(0.6, 2) ** 2)
    doms = rng.uniform(0.8, 1.2, max(2, 2 * zp // 10)) if poled else None
    return kw, pump, doms


def _sfg_medium(rng, n, steps):
    """A random sum-frequency medium (the distribution of the ragged workload) of about `steps` steps."""
    b1s, b2, b2s, b3s = rng.uniform(-3, 3), rng.uniform(-1, 1), rng.uniform(-1, 1), rng.uniform(-0.2, 0.2)
    zp = int(math.ceil(steps * min(1.0, 1.0 / max(abs(b1s), abs(b2), abs(b2s), abs(b3s)))))
    kw = dict(relativeLength=1, nlLength=1, nlLengthOrig=1, beta2=b2, beta2s=b2s, beta2o=0, beta1=0, beta1s=b1s, beta1o=0,
              beta3=0, beta3s=b3s, beta3o=0, diffBeta0=0, tMax=10, tPrecision=n, zPrecision=zp)
    pump = np.exp(-_tau(n, 10) ** 2 / (2 * rng.uniform(0.5, 3) ** 2)) + 0j
    doms = rng.uniform(5, 50, max(2, steps // 27))
    return kw, pump, doms


# the GNLSE workload's medium; a shorter length at its step size, so that a pass is a part of its 9999 steps
_GNLSE = dict(nlLength=1.0 / 9, selfSteepLength=6.5, fr=0.18, fb=0.21, tau1=0.244, tau2=0.64, tau3=1.92,
              beta2=-1, beta3=0.05, tMax=50)


def _gnlse_rows(rng, rows, n):
    return 3 / np.cosh(_tau(n, 50))[None, :] * rng.uniform(0.8, 1.1, (rows, 1)) + _noise(rng, (rows, n), 1e-4)


def _inputs(case, seed):
    """{"media": [(constructor keywords, pump, poling), ...], and the arrays of the call}, on the host."""
    rng = np.random.default_rng(seed)
    kind, n = case["kind"], case["n"]
    if kind == "signal":
        return {"media": [_pdc_medium(rng, n, case["zp"])], "x": _noise(rng, n, 0.1)}
    if kind == "chi3":
        kw = dict(relativeLength=1, nlLength=1, beta2=-1, beta3=0, tMax=20, tPrecision=n, zPrecision=case["zp"])
        return {"media": [(kw, rng.uniform(0.9, 1.1) / np.cosh(_tau(n, 20)) + 0j, None)], "x": _noise(rng, n, 1e-3)}
    if kind in ("gnlse_signal", "gnlse_batch", "gnlse_grad"):
        kw = dict(_GNLSE, relativeLength=(case["steps"] + 0.5) / 9999, tPrecision=n, zPrecision=1111)
        return {"media": [(kw, None, None)], "x": _gnlse_rows(rng, case.get("rows", 1), n)}
    if kind == "pdc_green":
        return {"media": [_pdc_medium(rng, n, case["zp"])]}
    if kind == "sfgpdc_green":
        kw, pump, doms = _sfg_medium(rng, n, case["zp"])
        return {"media": [(dict(kw, diffBeta0=rng.uniform(-2, 2), diffBeta0o=rng.uniform(-2, 2)), pump, doms)]}
    if kind == "ragged":
        media, xs = [], []
        for k in range(case["media"]):
            nk = max(64, n >> (k % 5))
            media.append(_sfg_medium(rng, nk, int(rng.integers(max(20, case["steps"] // 4), case["steps"] + 1))))
            xs.append(_noise(rng, nk, 1e-3))
        return {"media": media, "x": xs}
    if kind == "shg_batch":
        kw = dict(relativeLength=1, nlLengthH=0.9, nlLengthP=1.0, beta2h=0.3, beta2p=-0.2, beta1h=0.5, beta1p=0,
                  diffBeta0=0.4, tMax=20, tPrecision=n, zPrecision=case["zp"])
        x = 1.5 * np.exp(-_tau(n, 20) ** 2 / 2)[None, :] * rng.uniform(0.8, 1.2, (case["rows"], 1))
        return {"media": [(kw, None, rng.uniform(0.8, 1.2, 10))],
                "x": np.concatenate([x + _noise(rng, x.shape, 1e-3), _noise(rng, x.shape, 1e-3)], axis=1)}
    if kind == "pdc_grad":
        kw, pump, _ = _pdc_medium(rng, n, case["zp"], poled=False)
        nz = _steps(kw)
        target = _noise(rng, (case["rows"], n), 1.0)
        return {"media": [(kw, None, None)], "x": _noise(rng, (case["rows"], n), 1e-3), "pump": np.fft.fft(pump),
                "poling": rng.uniform(-1, 1, nz), "target": target / np.linalg.norm(target)}
    raise ValueError("unknown kind %r" % kind)


_SOLVER = {"signal": "Chi2PDC", "chi3": "Chi3", "gnlse_signal": "Chi3GNLSE", "gnlse_batch": "Chi3GNLSE",
           "gnlse_grad": "Chi3GNLSE", "pdc_green": "Chi2PDC", "sfgpdc_green": "Chi2SFGPDC", "ragged": "Chi2SFG",
           "shg_batch": "Chi2SHG", "pdc_grad": "Chi2PDC"}


def prepare(case, seed):
    inputs = _inputs(case, seed)
    media = []
    for kw, pump, doms in inputs["media"]:
        more = {}
        if pump is not None:
            more["customPump"] = pump
        if doms is not None:
            more["poling"] = doms
        media.append(getattr(nlm, _SOLVER[case["kind"]])(**more, **kw))
    state = {"kind": case["kind"], "media": media, "x": inputs.get("x")}
    if case["kind"] == "signal":
        media[0].runPumpSimulation()
    if case["kind"] == "pdc_grad":
        dev = {"x": inputs["x"], "pump": inputs["pump"], "poling": inputs["poling"]}
        for k, v in dev.items():
            state[k] = torch.tensor(v, device="cuda").requires_grad_()
        state["target"] = torch.tensor(inputs["target"], device="cuda")
    if case["kind"] == "gnlse_grad":
        state["x"] = torch.fft.fft(torch.tensor(inputs["x"], device="cuda"), dim=1).requires_grad_()
        state["band"] = _band(torch.tensor(media[0].omega.copy(), device="cuda"))
    return state


def _band(omega):
    return ((omega >= 2) & (omega <= 4)).to(torch.float64)


class _Grid(np.ndarray):
    """A grid property's view of its medium's host memory, with the medium kept alive."""

    medium = None


def _grid(view, medium):
    grid = view.view(_Grid)
    grid.medium = medium
    return grid


def run(state):
    kind, m = state["kind"], state["media"][0]
    if kind == "signal":
        m.runSignalSimulation(state["x"])
        return {"freq": _grid(m.signalFreq, m), "time": _grid(m.signalTime, m)}
    if kind == "chi3":
        m.runPumpSimulation()
        m.runSignalSimulation(state["x"])
        return {"pump": _grid(m.pumpTime, m), "freq": _grid(m.signalFreq, m), "time": _grid(m.signalTime, m)}
    if kind == "gnlse_signal":
        m.runSignalSimulation(state["x"][0])
        return {"freq": _grid(m.signalFreq, m), "time": _grid(m.signalTime, m)}
    if kind in ("pdc_green", "sfgpdc_green"):
        c, s = m.computeGreensFunction()
        return {"C": c, "S": s}
    if kind == "ragged":
        for medium in state["media"]:
            medium.runPumpSimulation()
        return nlm.ragged_batch(state["media"], state["x"])
    if kind == "shg_batch":
        return m.batchSignalSimulation(state["x"], inTimeDomain=True)
    if kind == "gnlse_batch":
        return m.batchSignalSimulation(state["x"], inTimeDomain=True)
    if kind == "pdc_grad":
        leaves = [state["x"], state["pump"], state["poling"]]
        out = propagate_pdc(m, *leaves)
        loss = torch.sum(torch.abs(out - state["target"]) ** 2)
        return {"out": out.detach(), "grads": list(torch.autograd.grad(loss, leaves))}
    out = propagate_gnlse(m, state["x"])
    loss = torch.sum(torch.abs(out) ** 2 * state["band"])
    return {"out": out.detach(), "grad": torch.autograd.grad(loss, state["x"])[0]}


# ------------------------------------------------------------------------------------------------
# Work of one pass
# ------------------------------------------------------------------------------------------------

def _steps(kw):
    """z steps of a medium (step length: the shortest of the unit, dispersion and nonlinear lengths)."""
    disp = max(abs(v) for k, v in kw.items() if k.startswith("beta"))
    nl = min(v for k, v in kw.items() if k.startswith("nlLength") or k == "selfSteepLength")
    return int(kw["zPrecision"] * kw["relativeLength"] / min(1.0, 1.0 / disp if disp else math.inf, nl))


def work(case):
    """Field values in and out at 16 bytes each, and the flops of the split-step algorithm: 5 N log2 N for a
    transform (two a step and mode; 18 a GNLSE step) and the point-wise RK4 step."""
    inputs = _inputs(case, 0)
    kind, flops, values = case["kind"], 0.0, 0
    for kw, _, _ in inputs["media"]:
        n, nz = kw["tPrecision"], _steps(kw)
        fft = 5 * n * math.log2(n)
        modes = 2 if kind in ("sfgpdc_green", "ragged", "shg_batch") else 1
        rows = case.get("rows", 1)
        if kind in ("pdc_green", "sfgpdc_green"):
            rows = 2 * n * modes
            values += n + 2 * (n * modes) ** 2
        elif kind in ("signal", "chi3", "gnlse_signal"):
            values += n + 2 * nz * n + ((2 * nz - 1) * n if kind == "chi3" else 0)
        elif kind == "ragged":
            values += n + n * (1 + modes)
        elif kind == "pdc_grad":
            values += 4 * rows * n + 2 * n + nz
        else:
            values += 2 * rows * n * modes * (2 if kind == "gnlse_grad" else 1)
        step = (18 * fft + 120 * n) if kind.startswith("gnlse") else modes * (2 * fft + 80 * n)
        flops += rows * (nz - 1) * step * (2 if kind.endswith("grad") else 1)
        if kind == "chi3":
            flops += (2 * nz - 2) * (2 * fft + 20 * n)
    return {"bytes": 16 * values, "flops": flops}


# ------------------------------------------------------------------------------------------------
# The same results from plain torch / numpy in double precision
# ------------------------------------------------------------------------------------------------

class _Axes:
    """Grids, dispersion phases and poling of a medium."""

    def __init__(self, kw, doms, signal, pump=None, device="cpu"):
        n, t_max = kw["tPrecision"], kw["tMax"]
        self.n, self.nz, self.z = n, _steps(kw), kw["relativeLength"]
        self.dz = self.z / (self.nz - 1)
        self.dzp = self.z / (2 * self.nz - 2)
        w = np.fft.fftshift(np.arange(-n // 2, n // 2) * (-math.pi / t_max))
        self.omega = torch.tensor(w, device=device)
        phase = lambda b: w * (b[0] + w * (0.5 * b[1] + w * b[2] / 6))  # noqa: E731
        self.disp = torch.tensor(np.stack([phase(b) for b in signal]), device=device)
        self.disp_pump = None if pump is None else torch.tensor(phase(pump), device=device)
        self.poling = np.ones(self.nz)
        if doms is not None and len(doms) > 1:
            edges = np.cumsum(doms) * (self.nz / np.cumsum(doms)[-1])
            prev, sign = 0, 1.0
            for edge in edges:
                cell = int(edge)
                self.poling[prev:cell] = sign
                if cell < self.nz:
                    self.poling[cell] = sign * (2 * (edge % 1) - 1)
                sign, prev = -sign, cell + 1

    def factor(self, length):
        return torch.exp(1j * length * self.disp)

    def pump_rows(self, spectrum):
        rows = torch.arange(2 * self.nz - 1, dtype=torch.float64, device=self.omega.device) * self.dzp
        return torch.fft.ifft(spectrum[None, :] * torch.exp(1j * rows[:, None] * self.disp_pump[None, :]))


def _march(ax, x, deriv, in_time, grids=False):
    """Split-step march of the fields x (..., modes, N): `deriv(step, sub-step 0..2, fields)` is dz times the nonlinear
    derivative.  Returns the last spectra and fields, or every row."""
    step, back = ax.factor(ax.dz), ax.factor(-0.5 * ax.dz)
    f = (torch.fft.fft(x) if in_time else x) * ax.factor(0.5 * ax.dz)
    a = torch.fft.ifft(f)
    rows_f, rows_a = [f], [a]
    for i in range(1, ax.nz):
        k1 = deriv(i, 0, a)
        k2 = deriv(i, 1, a + 0.5 * k1)
        k3 = deriv(i, 1, a + 0.5 * k2)
        k4 = deriv(i, 2, a + k3)
        f = torch.fft.fft(a + (k1 + 2 * k2 + 2 * k3 + k4) / 6) * step
        a = torch.fft.ifft(f)
        if grids:
            rows_f.append(f)
            rows_a.append(a)
    f = f * back
    a = torch.fft.ifft(f)
    if grids:
        rows_f[-1], rows_a[-1] = f, a
        return torch.stack(rows_f), torch.stack(rows_a)
    return f, a


def _pdc_deriv(ax, kw, rows, poling):
    g = 1j * ax.dz / kw["nlLength"]
    mid = 0.5 * (poling[:-1] + poling[1:])
    drive = lambda i, s: (poling[i - 1], mid[i - 1], poling[i])[s] * g * rows[2 * i - 2 + s]  # noqa: E731
    return lambda i, s, a: drive(i, s) * torch.conj(a)


def _sfg_deriv(ax, kw, rows, gain=False):
    """Sum-frequency generation; gain: the second mode is also amplified (Chi2SFGPDC)."""
    p = ax.poling
    g0, g1 = 1j * ax.dz / kw["nlLength"], 1j * ax.dz / kw["nlLengthOrig"]

    def deriv(i, s, a):
        sign = (p[i - 1], 0.5 * (p[i - 1] + p[i]), p[i])[s]
        row = rows[2 * i - 2 + s]
        m, mo = (complex(np.exp(1j * kw.get(k, 0) * (i - 1 + 0.5 * s) * ax.dz)) for k in ("diffBeta0", "diffBeta0o"))
        other = torch.conj(row) * a[..., 0, :] / m
        if gain:
            other = other + mo * row * torch.conj(a[..., 1, :])
        return torch.stack([sign * g0 * m * row * a[..., 1, :], sign * g1 * other], dim=-2)
    return deriv


def _shg_deriv(ax, kw):
    p, db = ax.poling, kw["diffBeta0"]
    gp, gh = 1j * ax.dz / kw["nlLengthP"], 1j * ax.dz / kw["nlLengthH"]

    def deriv(i, s, a):
        sign = (p[i - 1], 0.5 * (p[i - 1] + p[i]), p[i])[s]
        m = complex(np.exp(1j * db * (i - 1 + 0.5 * s) * ax.dz))
        y, h = a[..., 0, :], a[..., 1, :]
        return torch.stack([sign * gp * m * torch.conj(y) * h, sign * gh / m * 0.5 * y * y], dim=-2)
    return deriv


def _gnlse_deriv(ax, kw):
    n, dev = ax.n, ax.omega.device
    t = np.arange(n // 2) * (2 * kw["tMax"] / n)
    fr, fb, t1, t2, t3 = (kw[k] for k in ("fr", "fb", "tau1", "tau2", "tau3"))
    r = np.zeros(n)
    r[:n // 2] = fr * (1 - fb) * (t1 / t2 ** 2 + 1 / t1) * np.exp(-t / t2) * np.sin(t / t1) \
        + fr * fb / t3 ** 2 * np.exp(-t / t3) * (2 * t3 - t)
    r[0] += 1 - fr
    raman = torch.fft.fft(torch.tensor(r + 0j, device=dev))
    steep = 1j * ax.dz * (1 / kw["nlLength"] + ax.omega / kw["selfSteepLength"])

    def deriv(i, s, y):
        conv = torch.fft.ifft(torch.fft.fft((y * torch.conj(y))) * raman)
        return torch.fft.ifft(torch.fft.fft(conv * y) * steep)
    return deriv


def _green_exact(ax, modes, deriv):
    """C and S from the responses to 1 and i in every bin, output modes and bins in rows, axes centred."""
    n = ax.n
    out_c, out_s = [], []
    for m in range(modes):
        x = torch.zeros(2 * n, modes, n, dtype=torch.complex128, device=ax.omega.device)
        k = torch.arange(n, device=x.device)
        x[k, m, k] = 1
        x[n + k, m, k] = 1j
        f = torch.fft.fftshift(_march(ax, x, deriv, False)[0], dim=-1)
        one = torch.fft.fftshift(f[:n], dim=0).permute(1, 2, 0).reshape(modes * n, n)
        im = torch.fft.fftshift(f[n:], dim=0).permute(1, 2, 0).reshape(modes * n, n)
        out_c.append(0.5 * (one - 1j * im))
        out_s.append(0.5 * (one + 1j * im))
    return torch.cat(out_c, dim=1), torch.cat(out_s, dim=1)


def exact(case, seed):
    inputs = _inputs(case, seed)
    kind = case["kind"]
    kw, pump, doms = inputs["media"][0]
    gpu = "cuda" if torch.cuda.is_available() else "cpu"
    betas = lambda k, s: (k.get("beta1" + s, 0), k.get("beta2" + s, 0), k.get("beta3" + s, 0))  # noqa: E731
    host = lambda v: torch.tensor(v)  # noqa: E731
    if kind == "signal":
        ax = _Axes(kw, doms, [betas(kw, "s")], betas(kw, ""))
        deriv = _pdc_deriv(ax, kw, ax.pump_rows(torch.fft.fft(host(pump))), ax.poling)
        f, a = _march(ax, host(inputs["x"])[None], deriv, True, grids=True)
        return {"freq": f[:, 0], "time": a[:, 0]}
    if kind == "chi3":
        ax = _Axes(kw, None, [betas(kw, "")], betas(kw, ""))
        env = np.fft.ifft(np.fft.fft(pump) * np.exp(0.5j * ax.dzp * ax.disp_pump.numpy()))
        full = np.exp(1j * ax.dzp * ax.disp_pump.numpy())
        rows = [env]
        g = 0.5j * ax.dz / kw["nlLength"]
        for _ in range(2 * ax.nz - 2):
            a = rows[-1]
            spec = np.fft.fft(a * np.exp(g * np.abs(a) ** 2)) * full
            rows.append(np.fft.ifft(spec))
        rows[-1] = np.fft.ifft(spec * np.exp(-0.5j * ax.dzp * ax.disp_pump.numpy()))
        rows = host(np.stack(rows))
        h = 1j * ax.dz / kw["nlLength"]

        def deriv(i, s, a):
            p = rows[2 * i - 2 + s]
            return h * (2 * torch.abs(p) ** 2 * a + p * p * torch.conj(a))
        f, a = _march(ax, host(inputs["x"])[None], deriv, True, grids=True)
        return {"pump": rows, "freq": f[:, 0], "time": a[:, 0]}
    if kind == "gnlse_signal":
        ax = _Axes(kw, None, [betas(kw, "")])
        f, a = _march(ax, host(inputs["x"]), _gnlse_deriv(ax, kw), True, grids=True)
        return {"freq": f[:, 0], "time": a[:, 0]}
    if kind == "pdc_green":
        ax = _Axes(kw, doms, [betas(kw, "s")], betas(kw, ""), gpu)
        rows = ax.pump_rows(torch.fft.fft(torch.tensor(pump, device=gpu)))
        c, s = _green_exact(ax, 1, _pdc_deriv(ax, kw, rows, ax.poling))
        return {"C": c, "S": s}
    if kind == "sfgpdc_green":
        ax = _Axes(kw, doms, [betas(kw, "s"), betas(kw, "o")], betas(kw, ""), gpu)
        rows = ax.pump_rows(torch.fft.fft(torch.tensor(pump, device=gpu)))
        c, s = _green_exact(ax, 2, _sfg_deriv(ax, kw, rows, gain=True))
        return {"C": c, "S": s}
    if kind == "ragged":
        if case["media"] * case["steps"] > 30000:
            return None
        outs = []
        for (kw, pump, doms), x in zip(inputs["media"], inputs["x"]):
            ax = _Axes(kw, doms, [betas(kw, "s"), betas(kw, "o")], betas(kw, ""))
            both = np.stack([x, np.zeros_like(x)])
            outs.append(_march(ax, host(both), _sfg_deriv(ax, kw, ax.pump_rows(torch.fft.fft(host(pump)))), False)[0])
        return outs
    if kind == "shg_batch":
        ax = _Axes(kw, doms, [betas(kw, "p"), betas(kw, "h")], None, gpu)
        x = torch.tensor(inputs["x"].reshape(case["rows"], 2, -1), device=gpu)
        return _march(ax, x, _shg_deriv(ax, kw), True)[1].reshape(case["rows"], -1)
    if kind == "gnlse_batch":
        ax = _Axes(kw, None, [betas(kw, "")], None, gpu)
        return _march(ax, torch.tensor(inputs["x"], device=gpu), _gnlse_deriv(ax, kw), True)[1]
    if kind == "pdc_grad":
        ax = _Axes(kw, None, [betas(kw, "s")], betas(kw, ""))
        leaves = [host(inputs[k]).requires_grad_() for k in ("x", "pump", "poling")]
        deriv = _pdc_deriv(ax, kw, ax.pump_rows(leaves[1]), leaves[2])
        out = _march(ax, leaves[0], deriv, False)[0]
        loss = torch.sum(torch.abs(out - host(inputs["target"])) ** 2)
        return {"out": out.detach(), "grads": list(torch.autograd.grad(loss, leaves))}
    ax = _Axes(kw, None, [betas(kw, "")], None, gpu)
    x = torch.fft.fft(torch.tensor(inputs["x"], device=gpu), dim=1).requires_grad_()
    out = _march(ax, x, _gnlse_deriv(ax, kw), False)[0]
    loss = torch.sum(torch.abs(out) ** 2 * _band(ax.omega))
    return {"out": out.detach(), "grad": torch.autograd.grad(loss, x)[0]}
