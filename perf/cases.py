"""Performance cases: the work that users of this package have it do, through its public entry points.

Each case is one of the package's paths at a size it meets in use:

* "td"     one time-domain waveform (``InterpolatedModeSum``), forward or with gradients;
* "batch"  many uneven waveforms in one persistent launch (``BatchedInterpolatedModeSum``);
* "fd"     one frequency-domain waveform (``FDInterpolatedModeSum``);
* "aak"    one AAK waveform (``AAKSummation``);
* "direct" the direct sum over dense amplitudes (``DirectModeSum``);
* "spline" many cubic splines built and evaluated (``CubicSplineInterpolant``);
* "select" amplitudes from B-spline grids, harmonics and the power-threshold mode selection
           (``AmpInterp2D``, ``GetYlms``, ``ModeSelector``), the producers of the sum's inputs.

Amplitudes, harmonics, phases and coefficient grids are in GPU memory before a call; the knot times
and mode numbers are host arrays, as a trajectory integrator and a mode list leave them.  ``exact``
restates each path in plain torch and numpy in 64 bits.
"""
import math

import numpy as np
import torch

from fastemriwaveforms_b200 import (AAKSummation, AmpInterp2D, CubicSplineInterpolant, DirectModeSum,
                                    FDInterpolatedModeSum, GetYlms, InterpolatedModeSum, ModeSelector)
from fastemriwaveforms_b200 import synthetic as S
from fastemriwaveforms_b200.batched import BatchedInterpolatedModeSum

DT = 10.0
MTSUN = 4.9254909491978065e-06  # solar mass in seconds
DEV = "cuda"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a first look at a source: few modes, eleven days; host work and launches count
        {"name": "td_small", "kind": "td", "modes": "lmn", "K": 200, "N": 100, "T": 100_001, "precision": "faithful",
         "backward": ""},
        # the headline: one year, every mode, the reference's rounding
        {"name": "td_year", "kind": "td", "modes": "lmn", "K": 3843, "N": 1000, "T": 3_150_001,
         "precision": "faithful", "backward": ""},
        # a generic (inclined) orbit, whose k != 0 modes make many (m, k) rows; an odd, ragged length
        {"name": "td_generic", "kind": "td", "modes": "lmkn", "K": 363, "N": 437, "T": 700_003, "precision": "exact",
         "backward": ""},
        # the year again for a search, where 1e-5 of the amplitude is enough
        {"name": "td_year_mixed", "kind": "td", "modes": "lmn", "K": 3843, "N": 1000, "T": 3_150_001,
         "precision": "mixed", "backward": ""},
        # a likelihood gradient (amplitudes and phases), four months, FP64 throughout
        {"name": "grad_fp64", "kind": "td", "modes": "lmn", "K": 1000, "N": 500, "T": 1_000_000,
         "precision": "faithful", "backward": "fp64"},
        # the same gradient on the tensor cores
        {"name": "grad_mixed", "kind": "td", "modes": "lmn", "K": 1000, "N": 500, "T": 1_000_000,
         "precision": "mixed", "backward": "mixed"},
        # a population: waveforms of uneven length, knot and mode counts at once
        {"name": "batch", "kind": "batch", "count": 12, "T_lo": 100_000, "T_hi": 3_150_000, "N_lo": 50,
         "N_hi": 2000, "K_lo": 200, "K_hi": 3843, "precision": "mixed"},
        # the frequency-domain year
        {"name": "fd_year", "kind": "fd", "K": 3843, "N": 1000, "T": 3_150_001, "spin": 0.5, "mask_positive": False},
        # the AAK year, the 18 harmonics of the int(30 e0) rule at e0 = 0.6
        {"name": "aak_year", "kind": "aak", "N": 1000, "T": 3_150_001, "nmodes": 18, "mich": False},
        # dense amplitudes and phases of a few modes, summed as they are
        {"name": "direct", "kind": "direct", "T": 100_001, "K": 200},
        # a set of trajectory quantities splined and sampled on a dense grid, values and first derivatives
        {"name": "spline", "kind": "spline", "series": 256, "N": 1000, "points": 10_000, "own_knots": False},
        # what comes before a year's sum: the amplitude grids at the knots, harmonics, the modes that matter
        {"name": "select", "kind": "select", "lmax": 10, "nmax": 30, "N": 1000, "grid": 40, "threshold": 1e-5},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["td", "td", "grad", "batch", "fd", "aak", "direct", "spline", "select"])
    if kind in ("td", "grad"):
        c = {"kind": "td", "modes": rng.choice(["lmn", "lmn", "lmkn"]), "K": _log(rng, 100, 3843),
             "N": _log(rng, 20, 2000), "T": _log(rng, 4000, 3_150_001),
             "precision": rng.choice(["faithful", "faithful", "exact", "mixed"]), "backward": ""}
        if c["modes"] == "lmkn":
            c["K"] = min(c["K"], 1260)  # m = 0..6, k = -1..1, n = -30..30 and a little less
        if kind == "grad":
            c["T"] = _log(rng, 4000, 1_000_000)
            c["backward"] = "mixed" if c["precision"] == "mixed" else "fp64"
        c["N"] = min(c["N"], c["T"] // 8)
        return c
    if kind == "batch":
        hi = _log(rng, 200_000, 3_150_000)
        return {"kind": "batch", "count": rng.randint(2, 12), "T_lo": 100_000, "T_hi": hi, "N_lo": 50,
                "N_hi": _log(rng, 100, 2000), "K_lo": 200, "K_hi": _log(rng, 400, 3843), "precision": "mixed"}
    if kind == "fd":
        return {"kind": "fd", "K": _log(rng, 100, 3843), "N": _log(rng, 20, 1000), "T": _log(rng, 50_000, 3_150_001),
                "spin": round(rng.uniform(0.0, 0.8), 3), "mask_positive": rng.random() < 0.5}
    if kind == "aak":
        return {"kind": "aak", "N": _log(rng, 20, 1000), "T": _log(rng, 4000, 3_150_001),
                "nmodes": rng.randint(4, 24), "mich": rng.random() < 0.5}
    if kind == "direct":
        K = _log(rng, 8, 400)
        return {"kind": "direct", "T": _log(rng, 1000, 400_000 if K < 100 else 100_000), "K": K}
    if kind == "spline":
        own = rng.random() < 0.3
        n = _log(rng, 3, 256 if own else 2048)
        return {"kind": "spline", "series": n, "N": _log(rng, 5, 2000),
                "points": min(_log(rng, 1, 100_000), 4_000_000 // n), "own_knots": own}
    return {"kind": "select", "lmax": rng.randint(3, 10), "nmax": rng.randint(4, 30), "N": _log(rng, 20, 2000),
            "grid": rng.randint(12, 50), "threshold": 10.0 ** rng.uniform(-6, -2)}


# ------------------------------------------------------------------ inputs
def _gen(seed, salt=0):
    g = torch.Generator(device=DEV)
    g.manual_seed((int(seed) * 1000003 + salt) % (1 << 62))
    return g


def _normal(g, *shape):
    return torch.randn(*shape, generator=g, device=DEV, dtype=torch.float64)


def _cnormal(g, *shape):
    return torch.complex(_normal(g, *shape), _normal(g, *shape)) / math.sqrt(2.0)


def _dev(x):
    return torch.as_tensor(np.ascontiguousarray(x), device=DEV)


def _mode_numbers(modes, K):
    if modes == "lmn":
        return S.mode_list(10, 30, K)
    # inclined orbits: m = 0..10 and |k| <= 1 first with |n| <= 5 (363 modes), then wider n
    nmax = 5 if K <= 363 else 30
    rows = [(max(2, m), m, k, n) for m in range(11 if K <= 363 else 7) for k in (-1, 0, 1)
            for n in range(-nmax, nmax + 1)][:K]
    a = np.asarray(rows, dtype=np.int32)
    return tuple(np.ascontiguousarray(a[:, i]) for i in range(4))


def _trajectory_inputs(modes, K, N, T, seed, t=None):
    """Knots, phases and mode numbers on the host; amplitudes and harmonics on the GPU."""
    rng = np.random.default_rng(seed)
    span = (T - 1) * DT
    if t is None:
        t = S.knot_times(rng, N, span, 0.099 * span / (N - 1))
    l, m, k, n = _mode_numbers(modes, K)
    K = len(l)
    phi, phr = S.phase_values(t, 1.02 * span, span)
    theta = 0.93 * phi if modes == "lmkn" else np.zeros_like(phi)
    pc = S.phase_basis_from_knots(t, np.stack([phi, theta, phr]))
    g = _gen(seed)
    a = _cnormal(g, K) * _dev(np.exp(-np.abs(n) / 4.0) / l.astype(np.float64) ** 2)
    omega = torch.rand(K, generator=g, device=DEV, dtype=torch.float64) * 1e-6
    td = _dev(t)
    ang = td[:, None] * omega[None, :]
    teuk = a[None, :] * (1.0 + 0.5 * td[:, None] / span) * torch.complex(torch.cos(ang), torch.sin(ang))
    lm, inv = np.unique(np.stack([l, m]), axis=1, return_inverse=True)
    pairs = _cnormal(g, 2, lm.shape[1])
    inv = _dev(np.asarray(inv).reshape(-1))
    ylms = torch.cat([pairs[0][inv], pairs[1][inv]])
    return {"t": t, "teuk": teuk.contiguous(), "ylms": ylms, "pc": _dev(pc), "l": l, "m": m, "k": k, "n": n,
            "T": (span + DT) / S.YRSID_SI, "K": K, "N": N, "span": span}


def _td_inputs(case, seed):
    x = _trajectory_inputs(case["modes"], case["K"], case["N"], case["T"], seed)
    if case["backward"]:
        num = S.output_length(x["t"], x["T"], DT)[0]
        x["upstream"] = _cnormal(_gen(seed, 1), num)
    return x


def _batch_shapes(case, seed):
    # the sizes belong to the case, not to the seed of the inputs
    rng = np.random.default_rng(case["count"] * 7 + 5)
    out = []
    for w in range(case["count"]):
        T = int(np.exp(rng.uniform(np.log(case["T_lo"]), np.log(case["T_hi"]))))
        out.append((int(rng.integers(case["K_lo"], case["K_hi"] + 1)), int(rng.integers(case["N_lo"], case["N_hi"] + 1)),
                    T, int(seed) * 100 + w))
    return out


def _frequencies(M, a, p, e):
    """Azimuthal and radial frequencies (Hz) of prograde equatorial Kerr geodesics, by quadrature
    of the radial motion (trapezoid rule on the periodic integrands)."""
    p, e = np.asarray(p, float)[:, None], np.asarray(e, float)[:, None]
    r1, r2 = p / (1 - e), p / (1 + e)
    # x = L - a E and E from R(r1) = R(r2) = 0, by Newton from the Schwarzschild values
    E = np.sqrt(((p - 2) ** 2 - 4 * e**2) / (p * (p - 3 - e**2)))
    x = p / np.sqrt(p - 3 - e**2) - a * E
    for _ in range(30):
        rows = []
        for r in (r1, r2):
            D = r * r - 2 * r + a * a
            u = E * r * r - a * x
            rows.append((u * u - D * (r * r + x * x), 2 * u * r * r, -2 * u * a - 2 * D * x))
        (f1, a1, b1), (f2, a2, b2) = rows
        det = a1 * b2 - a2 * b1
        E, x = E - (f1 * b2 - f2 * b1) / det, x - (a1 * f2 - a2 * f1) / det
    L = x + a * E
    r3 = 2 / (1 - E * E) - (r1 + r2)
    psi = (np.arange(128) + 0.5) * (np.pi / 128)
    r = p / (1 + e * np.cos(psi))
    # dlambda/dpsi from R = (1 - E^2)(r1 - r)(r - r2)(r - r3) r, its zeros at r1 and r2 divided out
    rate = r / p * np.sqrt((1 - e * e) / ((1 - E * E) * (r - r3) * r))
    D = r * r - 2 * r + a * a
    tdot = E * ((r * r + a * a) ** 2 / D - a * a) + a * L * (1 - (r * r + a * a) / D)
    pdot = L - a * E + a / D * (E * (r * r + a * a) - a * L)
    period, advance = (tdot * rate).mean(axis=1), (pdot * rate).mean(axis=1)  # over 2 pi
    den = 2 * np.pi * M * MTSUN
    return advance / period / den, 1.0 / period / den


def _orbit(case, u):
    return 12.0 + (7.4 - 12.0) * (1.0 - (1.0 - u) ** 0.8), 0.4 + (0.2 - 0.4) * u


def _fd_inputs(case, seed):
    # knots that close in on the plunge, as an adaptive integrator sets them: with knots at random a mode's
    # frequency spline can turn twice in a segment, which the sum refuses as the reference does
    t = (case["T"] - 1) * DT * (1.0 - np.linspace(1.0, 0.0, case["N"]) ** 1.3)
    x = _trajectory_inputs("lmn", case["K"], case["N"], case["T"], seed, t)
    u = x["t"] / x["span"]
    x["M"], x["a"] = 1e6, case["spin"]
    x["p"], x["e"] = _orbit(case, u)
    x["xI"] = np.ones_like(u)
    ud = np.linspace(0.0, 1.0, 20 * case["N"])
    fphi, fr = _frequencies(x["M"], x["a"], *_orbit(case, ud))
    knots = S.phase_knots_from_frequencies(x["t"], ud * x["span"], np.stack([fphi, np.zeros_like(fphi), fr]))
    x["pc"] = _dev(S.phase_basis_from_knots(x["t"], knots))
    return x


def _aak_inputs(case, seed):
    span = (case["T"] - 1) * DT
    rng = np.random.default_rng(seed)
    e0 = float(rng.uniform(0.5, 0.65))
    inp = S.aak_case(N=case["N"], span=span, seed=seed, e_range=(e0, e0 - 0.25), nmodes=case["nmodes"])
    return inp, _dev(inp.interp_coeffs)


def _direct_inputs(case, seed):
    T, K = case["T"], case["K"]
    rng = np.random.default_rng(seed)
    g = _gen(seed)
    t = np.linspace(0.0, (T - 1) * DT, T)
    td = _dev(t)
    lo, hi = _cnormal(g, K), _cnormal(g, K)
    teuk = lo[None, :] + (hi - lo)[None, :] * (td / td[-1])[:, None]
    rates = torch.tensor([12e-3, 2e-3, 9e-3], device=DEV, dtype=torch.float64)
    phases = rates[:, None] * td[None, :] * (1.0 + 0.1 * td / td[-1])[None, :] + 0.5
    l = rng.integers(2, 6, K)
    m, k, n = rng.integers(0, 5, K), rng.integers(-1, 2, K), rng.integers(-5, 6, K)
    return {"t": t, "teuk": teuk.contiguous(), "phases": phases.contiguous(), "ylms": _cnormal(g, 2 * K),
            "l": l, "m": m, "k": k, "n": n}


def _spline_inputs(case, seed):
    rng = np.random.default_rng(seed)
    n, N, M = case["series"], case["N"], case["points"]
    span = 1e7
    if case["own_knots"]:
        gaps = rng.uniform(0.2, 1.0, (n, N - 1))
        t = np.concatenate([np.zeros((n, 1)), np.cumsum(gaps, axis=1)], axis=1)
        t *= span / t[:, -1:]
        t[:, -1] = span
    else:
        t = S.knot_times(rng, N, span, 0.099 * span / (N - 1))
    td = _dev(t)
    g = _gen(seed)
    w = torch.rand(n, 1, generator=g, device=DEV, dtype=torch.float64) * 6 + 1
    y = torch.sin(w * td / span + 6 * _normal(g, n, 1)) * (1 + 0.5 * td / span)
    return {"t": td, "y": y.contiguous(), "tnew": _dev(np.linspace(0.0, span, M) if M > 1 else np.array([0.37 * span]))}


class GridAmplitudes:
    """An amplitude generator as ``ModeSelector`` calls it: B-spline grids in (w, u), with the mode
    bookkeeping of the reference's amplitude modules (m = 0 modes first)."""

    def __init__(self, lmax, nmax, grid, seed):
        book = S.FixedAmplitudes(lmax=lmax, nmax=nmax, N=2, seed=1)
        for name in ("l_arr_no_mask", "m_arr_no_mask", "k_arr_no_mask", "n_arr_no_mask", "unique_l", "unique_m",
                     "inverse_lm", "index_map_arr"):
            setattr(self, name, getattr(book, name))
        K = len(self.l_arr_no_mask)
        inner = np.linspace(0, 1, grid - 6)[1:-1]
        self.knots = np.concatenate([np.zeros(4), inner, np.ones(4)])
        # a mode's power is the mode list's own, its phase the seed's: the selection keeps the same modes
        # for every seed
        mag = np.exp(-np.abs(self.n_arr_no_mask) / 1.5) / self.l_arr_no_mask.astype(np.float64) ** 3
        mag *= np.random.default_rng(K).uniform(0.5, 1.0, K)
        shape = np.random.default_rng(grid).uniform(0.7, 1.3, (grid - 4) ** 2)
        phase = torch.rand(K, generator=_gen(seed), device=DEV, dtype=torch.float64) * (2 * math.pi)
        part = torch.stack([torch.cos(phase), torch.sin(phase)], dim=1) * _dev(mag)[:, None]
        self.coeff = (part[:, :, None] * _dev(shape)).contiguous()
        self.amp = AmpInterp2D(self.knots, self.knots, self.coeff, self.l_arr_no_mask, self.m_arr_no_mask,
                               self.k_arr_no_mask, self.n_arr_no_mask)

    def __call__(self, a, p, e, xI, specific_modes=None):
        return self.amp(p, e, mode_indexes=specific_modes)


def _select_points(case, seed):
    rng = np.random.default_rng(seed)
    s = np.linspace(0.0, 1.0, case["N"])
    t = S.knot_times(rng, case["N"], 3.15e7, 0.099 * 3.15e7 / (case["N"] - 1))
    return t, 0.05 + 0.9 * s**1.5, 0.5 + 0.4 * np.sin(2.0 * np.pi * s) * (1.0 - s), 1.1, rng.uniform(0, 6.2)


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    if kind == "td":
        x = _td_inputs(case, seed)
        x["sum"] = InterpolatedModeSum(precision=case["precision"])
        if case["backward"]:
            x["teuk"].requires_grad_(True)
            x["pc"].requires_grad_(True)
    elif kind == "batch":
        waves = []
        for K, N, T, s in _batch_shapes(case, seed):
            w = _trajectory_inputs("lmn", K, N, T, s)
            waves.append({"t": w["t"], "teuk_modes": w["teuk"], "ylms": w["ylms"], "phase_interp_t": w["t"],
                          "phase_interp_coeffs": w["pc"], "l_arr": w["l"], "m_arr": w["m"], "k_arr": w["k"],
                          "n_arr": w["n"], "T": w["T"], "dt": DT})
        x = {"sum": BatchedInterpolatedModeSum(precision=case["precision"], autotune=False).setup(waves)}
    elif kind == "fd":
        x = _fd_inputs(case, seed)
        x["sum"] = FDInterpolatedModeSum()
        x["mask_positive"] = case["mask_positive"]
    elif kind == "aak":
        inp, coeffs = _aak_inputs(case, seed)
        args = list(inp.call_args())
        args[11] = coeffs
        x = {"sum": AAKSummation(), "args": args, "mich": case["mich"], "T": inp.T}
    elif kind == "direct":
        x = _direct_inputs(case, seed)
        x["T"] = (x["t"][-1] + DT) / S.YRSID_SI
        x["sum"] = DirectModeSum()
    elif kind == "spline":
        x = _spline_inputs(case, seed)
    else:
        t, w, u, theta, phi = _select_points(case, seed)
        gen = GridAmplitudes(case["lmax"], case["nmax"], case["grid"], seed)
        x = {"t": t, "w": w, "u": u, "theta": theta, "phi": phi,
             "sel": ModeSelector(gen, ylm_generator=GetYlms(), mode_selection_threshold=case["threshold"])}
    x["kind"] = kind
    return x


def run(x):
    kind = x["kind"]
    if kind == "td":
        h = x["sum"](x["t"], x["teuk"], x["ylms"], x["t"], x["pc"], x["l"], x["m"], x["k"], x["n"], T=x["T"], dt=DT)
        if "upstream" not in x:
            return {"h": h}
        g_teuk, g_pc = torch.autograd.grad(h, (x["teuk"], x["pc"]), grad_outputs=x["upstream"])
        return {"h": h, "g_teuk": g_teuk, "g_pc": g_pc}
    if kind == "batch":
        return list(x["sum"].forward())
    if kind == "fd":
        h = x["sum"](x["t"], x["teuk"], x["ylms"], x["t"], x["pc"], x["l"], x["m"], x["k"], x["n"], x["M"], x["a"],
                     x["p"], x["e"], x["xI"], T=x["T"], dt=DT, mask_positive=x["mask_positive"])
        return {"h": h, "f": x["sum"].frequency}
    if kind == "aak":
        return {"h": x["sum"](*x["args"], mich=x["mich"], T=x["T"], dt=DT)}
    if kind == "direct":
        return {"h": x["sum"](x["t"], x["teuk"], x["ylms"], x["t"], x["phases"], x["l"], x["m"], x["k"], x["n"],
                              T=x["T"], dt=DT)}
    if kind == "spline":
        s = CubicSplineInterpolant(x["t"], x["y"])
        return {"coeffs": s.interp_array, "value": s(x["tnew"]), "rate": s(x["tnew"], deriv_order=1)}
    teuk, ylms, l, m, k, n = x["sel"](x["t"], 0.5, x["w"], x["u"], None, x["theta"], x["phi"])
    return {"teuk": teuk, "ylms": ylms, "l": l, "m": m, "k": k, "n": n}


# ------------------------------------------------------------------ the work of one pass
def _keys(modes, K):
    l, m, k, n = _mode_numbers(modes, K)
    rows = set(zip(m.tolist(), k.tolist())) | {(-a, -b) for a, b in zip(m.tolist(), k.tolist())}
    top = int(np.abs(n).max())
    return len(rows) * (2 * top + 1), len(l)


def work(case):
    kind = case["kind"]
    if kind == "td":
        keys, K = _keys(case["modes"], case["K"])
        N, T = case["N"], case["T"]
        b = 16 * N * K + 192 * N + 16 * T
        # a cubic and a complex product per (key, sample); twice again for the two gradients
        f = 20.0 * keys * T
        return {"bytes": b * (3 if case["backward"] else 1), "flops": f * (3 if case["backward"] else 1)}
    if kind == "batch":
        b = f = 0.0
        for K, N, T, _ in _batch_shapes(case, 0):
            keys, K = _keys("lmn", K)
            b += 16 * N * K + 192 * N + 16 * T
            f += 20.0 * keys * T
        return {"bytes": b, "flops": f}
    if kind == "fd":
        l, m, k, n = _mode_numbers("lmn", case["K"])
        fphi, fr = _frequencies(1e6, case["spin"], *_orbit(case, np.linspace(0, 1, 33)))
        f = np.outer(fphi, m) + np.outer(fr, n)
        bins = np.abs(np.diff(f, axis=0)).sum() * case["T"] * DT
        # per (mode, bin): a cubic's root, the amplitude, phase and frequency derivatives there, one phasor
        return {"bytes": 16 * case["N"] * len(l) + 32 * case["T"], "flops": 200.0 * float(bins)}
    if kind == "aak":
        # per sample the orbit and its geometry, per harmonic a phasor and three amplitudes
        return {"bytes": 16 * case["T"] + 384 * case["N"], "flops": case["T"] * (400.0 + 100.0 * case["nmodes"])}
    if kind == "direct":
        return {"bytes": 16 * case["T"] * (case["K"] + 2.5), "flops": 60.0 * case["T"] * case["K"]}
    if kind == "spline":
        n, N, M = case["series"], case["N"], case["points"]
        return {"bytes": 8.0 * n * (5 * N + 2 * M), "flops": n * (30.0 * N + 12.0 * M)}
    K = (2 * case["nmax"] + 1) * sum(l + 1 for l in range(2, case["lmax"] + 1))
    return {"bytes": 16.0 * K * ((case["grid"] - 4) ** 2 + case["N"]), "flops": 80.0 * K * case["N"]}


# ------------------------------------------------------------------ 64-bit restatements
def _spline_coeffs(t, y):
    """Not-a-knot cubic coefficients (4, N - 1, ...) of y (N, ...) on knots t (N,), by a dense solve."""
    N = t.numel()
    h = t[1:] - t[:-1]
    A = torch.zeros(N, N, dtype=torch.float64, device=t.device)
    B = torch.zeros(N, N - 1, dtype=torch.float64, device=t.device)  # right-hand side from the slopes
    i = torch.arange(1, N - 1, device=t.device)
    A[i, i - 1], A[i, i], A[i, i + 1] = h[1:], 2 * (h[:-1] + h[1:]), h[:-1]
    B[i, i - 1], B[i, i] = 3 * h[1:], 3 * h[:-1]
    d, g = h[0] + h[1], h[-1] + h[-2]
    A[0, 0], A[0, 1] = h[1], d
    B[0, 0], B[0, 1] = (h[0] + 2 * d) * h[1] / d, h[0] ** 2 / d
    A[N - 1, N - 1], A[N - 1, N - 2] = h[-2], g
    B[N - 1, N - 2], B[N - 1, N - 3] = (2 * g + h[-1]) * h[-2] / g, h[-1] ** 2 / g
    shape = (-1,) + (1,) * (y.ndim - 1)
    hh = h.reshape(shape)
    slope = (y[1:] - y[:-1]) / hh
    s = torch.linalg.solve(A, (B @ slope.reshape(N - 1, -1))).reshape(y.shape)
    q = (s[:-1] + s[1:] - 2 * slope) / hh
    return torch.stack([y[:-1], s[:-1], (slope - s[:-1]) / hh - q, q / hh])


def _phase(c, s):
    s1 = 1.0 - s
    return c[0] + s * (c[1] + s1 * (c[2] + s * (c[3] + s1 * (c[4] + s * (c[5] + s1 * (c[6] + s * c[7]))))))


def _basis(s):
    s1 = 1.0 - s
    return torch.stack([torch.ones_like(s), s, s * s1, s * s * s1, s * s * s1 * s1, s**3 * s1**2, s**3 * s1**3,
                        s**4 * s1**3], dim=1)


def _td_exact(x, backward):
    """The interpolated mode sum, its terms of equal (m, k, n) added first, every term at its rounded phase."""
    t, teuk, K, N = _dev(x["t"]), x["teuk"].detach(), x["K"], x["N"]
    num = S.output_length(x["t"], x["T"], DT)[0]
    sign = _dev(np.where(x["l"] % 2 == 0, 1.0, -1.0))
    yp, ym = x["ylms"][:K], x["ylms"][K:] * sign
    y = torch.view_as_real(teuk).reshape(N, 2 * K).clone().requires_grad_(bool(backward))
    coeffs = _spline_coeffs(t, y)
    c = torch.view_as_complex(coeffs.detach().reshape(4, N - 1, K, 2).contiguous())
    mkn = np.stack([x["m"], x["k"], x["n"]], axis=1)
    nz = np.nonzero(x["m"])[0]
    keys, inv = np.unique(np.concatenate([mkn, -mkn[nz]]), axis=0, return_inverse=True)
    inv = _dev(np.asarray(inv).reshape(-1))
    nzd = _dev(nz)
    Q = len(keys)
    W = torch.zeros(4, N - 1, Q, dtype=torch.complex128, device=DEV)
    W.index_add_(2, inv[:K], c * yp)
    W.index_add_(2, inv[K:], c[:, :, nzd].conj() * ym[nzd])
    km, kk, kn = (_dev(keys[:, q].astype(np.float64)) for q in range(3))
    starts = np.ceil(x["t"] / DT).astype(np.int64).clip(0, num)
    starts[0], starts[-1] = 0, num
    out = torch.zeros(num, dtype=torch.complex128, device=DEV)
    if backward:
        gW = torch.zeros_like(W)
        gpc = torch.zeros(N - 1, 3, 8, dtype=torch.float64, device=DEV)
        up = x["upstream"].conj()
    pc, h = x["pc"].detach(), np.diff(x["t"])
    step = max(1, (1 << 25) // Q)
    for j in range(N - 1):
        for a in range(int(starts[j]), int(starts[j + 1]), step):
            b = min(a + step, int(starts[j + 1]))
            tt = torch.arange(a, b, device=DEV, dtype=torch.float64) * DT
            xx, s = tt - x["t"][j], (tt - x["t"][j]) / h[j]
            P = [_phase(pc[j, q], s)[:, None] for q in range(3)]
            ph = km * P[0] + kk * P[1]
            ph = ph + kn * P[2]
            E = torch.complex(torch.cos(ph), -torch.sin(ph))
            x1 = xx[:, None]
            F = E * (W[0, j] + x1 * (W[1, j] + x1 * (W[2, j] + x1 * W[3, j])))
            out[a:b] = F.sum(dim=1)
            if backward:
                g = up[a:b]
                for q in range(4):
                    gW[q, j] += ((g * xx**q)[:, None] * E).sum(dim=0).conj()
                Bs = _basis(s)
                for q, w in enumerate((km, kk, kn)):
                    gpc[j, q] += (g * (-1j) * (F * w).sum(dim=1)).real @ Bs
    if not backward:
        return {"h": out}
    gc = gW[:, :, inv[:K]] * yp.conj()
    gc[:, :, nzd] += ym[nzd] * gW[:, :, inv[K:]].conj()
    gy, = torch.autograd.grad(coeffs, y, torch.view_as_real(gc).reshape(4, N - 1, 2 * K))
    return {"h": out, "g_teuk": torch.view_as_complex(gy.reshape(N, K, 2).contiguous()), "g_pc": gpc}


_E23, _E13 = complex(math.cos(2 * math.pi / 3), -math.sin(2 * math.pi / 3)), complex(0.5, -math.sqrt(3) / 2)


def _spa(z):
    """i sqrt(z) e^{-iz} K_{1/3}(-iz): the power series for |z| <= 7, else nine asymptotic terms."""
    small = z.abs() <= 7.0
    zs = torch.where(small, z, torch.ones_like(z))
    z2 = zs * zs
    s1, s2 = torch.zeros_like(z), torch.zeros_like(z)
    c1, c2 = [0.5], [1.0]
    for j in range(13):
        c1.append(c1[-1] * -0.25 / ((j + 1) * (j + 4 / 3)))
        c2.append(c2[-1] * -0.25 / ((j + 1) * (j + 2 / 3)))
    for u, v in zip(reversed(c1), reversed(c2)):
        s1, s2 = u + z2 * s1, v + z2 * s2
    r = torch.exp(torch.log(zs.abs()) / 6)
    arg = torch.where(zs < 0, math.pi / 6, 0.0)
    p6 = torch.complex(r * torch.cos(arg), r * torch.sin(arg))
    small_v = torch.complex(torch.cos(zs), -torch.sin(zs)) * (
        _E23 * p6**5 * (s1 * (math.gamma(-1 / 3) / 2 ** (1 / 3))) + _E13 * p6 * (s2 * (math.gamma(1 / 3) / 2 ** (2 / 3))))
    inv = 1.0 / torch.where(small, torch.full_like(z, 8.0), z)
    a, big = 1.0, torch.zeros_like(small_v)
    terms = []
    for j in range(9):
        terms.append(a * 1j ** (j + 1))
        a *= (4 / 9 - (2 * j + 1) ** 2) / (8.0 * (j + 1))
    for v in reversed(terms):
        big = v + inv * big
    big = big * (complex(-math.sqrt(0.5), -math.sqrt(0.5)) * math.sqrt(0.5 * math.pi))
    return torch.where(small, small_v, big)


def _fd_exact(case, seed):
    """The stationary-phase sum over (mode, segment, bin), equatorial orbits and k = 0.  A turnover between
    knots widens a segment only when there is exactly one in the whole mode list; that is left out."""
    x = _fd_inputs(case, seed)
    K, N = x["K"], x["N"]
    num = S.output_length(x["t"], x["T"], DT)[0]
    L = num + (num + 1) % 2
    z0 = L // 2
    f = torch.arange(-z0, L - z0, device=DEV, dtype=torch.float64) / (L * DT)
    t = _dev(x["t"])
    fphi, fr = _frequencies(x["M"], x["a"], x["p"], x["e"])
    fk = torch.stack([_dev(fphi), _dev(fr)], dim=1)
    fc = _spline_coeffs(t, fk)  # (4, N-1, 2)
    ac = _spline_coeffs(t, torch.view_as_real(x["teuk"]).reshape(N, 2 * K)).reshape(4, N - 1, K, 2)
    sign = _dev(np.where(x["l"] % 2 == 0, 1.0, -1.0))
    yp, ym = x["ylms"][:K], x["ylms"][K:] * sign
    m, n = _dev(x["m"].astype(np.float64)), _dev(x["n"].astype(np.float64))
    fm = fk @ torch.stack([m, n])  # (N, K)
    lo, hi = torch.minimum(fm[1:], fm[:-1]).T, torch.maximum(fm[1:], fm[:-1]).T  # (K, N-1)
    f0, df = f[0].item(), (f[1] - f[0]).item()
    start = (((lo - f0) / df).abs().long() + 1).clamp(min=0)
    end = ((hi - f0) / df).abs().long().clamp(max=L - 1)
    count = (end - start + 1).clamp(min=0).reshape(-1)
    pre = torch.cat([count.new_zeros(1), count.cumsum(0)])
    start = start.reshape(-1)
    out = torch.zeros(L, dtype=torch.complex128, device=DEV)
    pc = x["pc"]
    h = t[1:] - t[:-1]
    xi = complex(-0.5, math.sqrt(3) / 2)
    total = int(pre[-1])
    for b0 in range(0, total, 1 << 23):
        bins = torch.arange(b0, min(b0 + (1 << 23), total), device=DEV)
        ent = torch.searchsorted(pre, bins, right=True) - 1
        i = start[ent] + bins - pre[ent]
        mode, seg = ent // (N - 1), ent % (N - 1)
        mm, nn = m[mode], n[mode]
        d, c, b, a = (mm * fc[q, seg, 0] + nn * fc[q, seg, 1] for q in range(4))
        fi = f[i]
        d = d - fi
        D0 = b * b - 3 * a * c
        D1 = 2 * b**3 - 9 * a * b * c + 27 * a * a * d
        C = ((torch.sqrt((D1 * D1 - 4 * D0**3).to(torch.complex128)) + D1) / 2)
        C = torch.exp(torch.log(C) / 3)
        del D1, c, d
        for q in range(3):
            u = C * xi**q
            root = (-(b + u + D0 / u) / (3 * a)).real
            tt = t[seg] + root
            ok = torch.nonzero((tt < t[seg + 1]) & (tt >= t[seg])).reshape(-1)
            if ok.numel() == 0:
                continue
            r, sg, mo, tr, fr_ = root[ok], seg[ok], mode[ok], tt[ok], fi[ok]
            hh = h[sg]
            s = (tr - t[sg]) / hh
            A = ac[0, sg, mo] + r[:, None] * (ac[1, sg, mo] + r[:, None] * (ac[2, sg, mo] + r[:, None] * ac[3, sg, mo]))
            A = torch.view_as_complex(A.contiguous())
            phase, fd, fdd = 0.0, 0.0, 0.0
            for field, mult in ((0, mm[ok]), (2, nn[ok])):
                cc = [pc[sg, field, w] for w in range(8)]
                phase = phase + mult * _phase(cc, s)
                s2, s3, s4, s5 = s * s, s**3, s**4, s**5
                d2 = (-2 * cc[2] + cc[3] * (2 - 6 * s) + cc[4] * (2 - 12 * s + 12 * s2) + cc[5] * (6 * s - 24 * s2 + 20 * s3)
                      + cc[6] * (6 * s - 36 * s2 + 60 * s3 - 30 * s4) + cc[7] * (12 * s2 - 60 * s3 + 90 * s4 - 42 * s5))
                d3 = (-6 * cc[3] + cc[4] * (-12 + 24 * s) + cc[5] * (6 - 48 * s + 60 * s2)
                      + cc[6] * (6 - 72 * s + 180 * s2 - 120 * s3) + cc[7] * (24 * s - 180 * s2 + 360 * s3 - 210 * s4))
                fd, fdd = fd + mult * d2 / (2 * math.pi * hh**2), fdd + mult * d3 / (2 * math.pi * hh**3)
            z = 2 * math.pi * fd**3 / (3 * fdd**2)
            amp = _spa(z) * (-fd / fdd.abs() * 2 / math.sqrt(3)) / torch.sqrt(z.to(torch.complex128))
            w = 2 * math.pi * fr_ * tr - phase
            term = A * amp * torch.complex(torch.cos(w), torch.sin(w))
            out.index_add_(0, i[ok], yp[mo] * term)
            im = 2 * z0 - i[ok]
            neg = torch.nonzero((mm[ok] != 0) & (im >= 0) & (im < L)).reshape(-1)
            out.index_add_(0, im[neg], ym[mo[neg]] * term[neg].conj())
    s, sf = -out.flip(0), -out
    p, q = s + sf, s - sf
    hp, hc = torch.complex(p.real / 2, q.imag / 2), torch.complex(-p.imag / 2, q.real / 2)
    res = torch.stack([hp, hc])
    return {"h": res[:, z0:].contiguous() if case["mask_positive"] else res, "f": f}


def _aak_exact(case, seed):
    inp, coeffs = _aak_inputs(case, seed)
    num = S.output_length(inp.t, inp.T, DT)[0]
    t = torch.arange(num, device=DEV, dtype=torch.float64) * DT
    kn = _dev(inp.t)
    out = torch.zeros(num, dtype=torch.complex128, device=DEV)
    pi, sin, cos = math.pi, torch.sin, torch.cos
    qS, qK, phiS, phiK = inp.qS, inp.qK, inp.phiS, inp.phiK
    sqS, cqS, sqK, cqK = math.sin(qS), math.cos(qS), math.sin(qK), math.cos(qK)
    sin_d, cos_d = math.sin(phiK - phiS), math.cos(phiK - phiS)
    hs3 = math.sqrt(3.0) / 2
    zeta = inp.m2 * 4.9254909491978065e-06 / inp.dist / 1.02927125054339e17
    n_s = (sqS * math.cos(phiS), sqS * math.sin(phiS), cqS)
    S_s = (sqK * math.cos(phiK), sqK * math.sin(phiK), cqK)
    cross = lambda u, v: (u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0])  # noqa: E731
    dot = lambda u, v: u[0] * v[0] + u[1] * v[1] + u[2] * v[2]  # noqa: E731
    for a0 in range(0, num, 1 << 17):
        tt = t[a0:a0 + (1 << 17)]
        j = (torch.searchsorted(kn, tt, right=True) - 1).clamp(0, len(inp.t) - 2)
        h = kn[j + 1] - kn[j]
        s = (tt - kn[j]) / h
        c = coeffs[j]  # (samples, 6, 8)

        def val(q):
            return _phase([c[:, q, w] for w in range(8)], s)

        def rate(q):
            w = [c[:, q, i] for i in range(8)]
            s2, s3, s4, s5, s6 = s * s, s**3, s**4, s**5, s**6
            return (w[1] + w[2] * (1 - 2 * s) + w[3] * (2 * s - 3 * s2) + w[4] * (2 * s - 6 * s2 + 4 * s3)
                    + w[5] * (3 * s2 - 8 * s3 + 5 * s4) + w[6] * (3 * s2 - 12 * s3 + 15 * s4 - 6 * s5)
                    + w[7] * (4 * s3 - 15 * s4 + 18 * s5 - 7 * s6)) / h

        e, Y = val(1), val(2)
        Pp, Pt, Pr = val(3), val(4), val(5)
        Op, Ot, Or = rate(3), rate(4), rate(5)
        gim, alp, nu, gimdot = Pt - Pr, Pp - Pt, Or / (2 * pi), Ot - Or
        lam = torch.acos(Y)
        sl, cl, sa, ca = sin(lam), cos(lam), sin(alp), cos(alp)
        cqL = cqK * cl + sqK * sl * ca
        sqL = torch.sqrt(1 - cqL**2)
        phiL = torch.atan2(sqK * math.sin(phiK) * cl - math.cos(phiK) * sl * sa - cqK * math.sin(phiK) * sl * ca,
                           sqK * math.cos(phiK) * cl + math.sin(phiK) * sl * sa - cqK * math.cos(phiK) * sl * ca)
        Ln = cqL * cqS + sqL * sqS * cos(phiL - phiS)
        Sn = cqK * cqS + sqK * sqS * cos_d
        beta = torch.atan2(-Sn + cl * Ln, sqS * sin_d * sl * ca + (cqK * Sn - cqS) / sqK * sl * sa)
        s2g, c2g = sin(2 * (gim + beta)), cos(2 * (gim + beta))
        F = (1.0, 0.0, 0.0, 1.0)
        cosorb = None
        if case["mich"]:
            orb = 2 * pi * tt / 31558149.763545595
            cosorb = cos(orb - phiS)
            cq = 0.5 * cqS - hs3 * sqS * cosorb
            phw = orb + torch.atan2(hs3 * cqS + 0.5 * sqS * cosorb, sqS * sin(orb - phiS))
            up = 0.5 * cqK - hs3 * sqK * cos(orb - phiK) - cq * (cqK * cqS + sqK * sqS * cos_d)
            dn = (0.5 * sqK * sqS * sin_d - hs3 * cos(orb) * (cqK * sqS * math.sin(phiS) - cqS * sqK * math.sin(phiK))
                  - hs3 * sin(orb) * (cqS * sqK * math.cos(phiK) - cqK * sqS * math.cos(phiS)))
            psi = torch.atan2(up, dn)
            c1 = 0.5 * (1 + cq * cq)
            sp, cp, ss, cs = sin(2 * phw), cos(2 * phw), sin(2 * psi), cos(2 * psi)
            F = (c1 * cp * cs - cq * sp * ss, c1 * cp * ss + cq * sp * cs, c1 * sp * cs + cq * cp * ss,
                 c1 * sp * ss - cq * cp * cs)
        Amp = (Op.abs() * inp.m1 * 4.9254909491978065e-06) ** (2.0 / 3.0) * zeta
        Lv = (cl * sqK * math.cos(phiK) + sl * (sa * math.sin(phiK) - ca * cqK * math.cos(phiK)),
              cl * sqK * math.sin(phiK) - sl * (sa * math.cos(phiK) + ca * cqK * math.sin(phiK)), cl * cqK + sl * ca * sqK)
        nL, nS = cross(n_s, Lv), cross(n_s, S_s)
        norm = (torch.sqrt(dot(nL, nL)) * math.sqrt(dot(nS, nS))).clamp(min=1e-6)
        cr = dot(nL, nS) / norm
        sr = (dot(Lv, nS) - dot(S_s, nL)) / norm
        r0, r1 = 2 * cr * cr - 1, cr * sr
        hI = hII = 0.0
        for n in range(1, case["nmodes"] + 1):
            nPhi = n * Pr
            if case["mich"]:
                nPhi = nPhi + 2 * pi * (n * nu + gimdot / pi) * 499.00478383615643 * sqS * cosorb
            nodes = (n + 2 + n + 40) // 2
            tau = np.arange(nodes + 1) * (pi / nodes)
            wt = np.full(nodes + 1, 1.0 / nodes)
            wt[0] = wt[-1] = 0.5 / nodes
            J = [0.0] * 5
            for tv, w in zip(tau, wt):
                y = n * e * math.sin(tv)
                cy, sy = cos(y), sin(y)
                for q in range(5):
                    k = n - 2 + q
                    J[q] = J[q] + (w * math.cos(k * tv)) * cy + (w * math.sin(k * tv)) * sy
            a = -n * Amp * (J[0] - 2 * e * J[1] + 2 / n * J[2] + 2 * e * J[3] - J[4]) * cos(nPhi)
            b = -n * Amp * torch.sqrt(1 - e * e) * (J[0] - 2 * J[2] + J[4]) * sin(nPhi)
            cc = 2 * Amp * J[2] * cos(nPhi)
            Ap0 = -(1 + Ln * Ln) * (a * c2g - b * s2g) + cc * (1 - Ln * Ln)
            Ac0 = 2 * Ln * (b * c2g + a * s2g)
            Ap, Ac = Ap0 * r0 + Ac0 * r1, -Ap0 * r1 + Ac0 * r0
            k = hs3 if case["mich"] else 1.0
            hI, hII = hI + k * (F[0] * Ap + F[1] * Ac), hII + k * (F[2] * Ap + F[3] * Ac)
        out[a0:a0 + tt.numel()] = torch.complex(hI, -hII)
    return {"h": out}


def _direct_exact(case, seed):
    x = _direct_inputs(case, seed)
    K = case["K"]
    m, k, n = (_dev(x[q].astype(np.float64)) for q in "mkn")
    sign = _dev(np.where(x["l"] % 2 == 0, 1.0, -1.0))
    yp, ym = x["ylms"][:K], x["ylms"][K:] * sign * (m > 0)
    out = []
    for a in range(0, case["T"], 1 << 14):
        P = x["phases"][:, a:a + (1 << 14), None]
        ph = (m * P[0] + k * P[1]) + n * P[2]
        E = torch.complex(torch.cos(ph), -torch.sin(ph))
        A = x["teuk"][a:a + (1 << 14)]
        out.append((yp * A * E).sum(dim=1) + (ym * A.conj() * E.conj()).sum(dim=1))
    return {"h": torch.cat(out)}


def _spline_exact(case, seed):
    x = _spline_inputs(case, seed)
    n, N = x["y"].shape
    tn = x["tnew"]
    coeffs = torch.zeros(4, N, n, dtype=torch.float64, device=DEV)
    value = torch.zeros(n, tn.numel(), dtype=torch.float64, device=DEV)
    rate = torch.zeros_like(value)
    shared = x["t"].ndim == 1
    for p in range(1 if shared else n):
        cols = slice(None) if shared else slice(p, p + 1)
        t = x["t"] if shared else x["t"][p]
        c = _spline_coeffs(t, x["y"][cols].T.contiguous())
        hl = t[-1] - t[-2]
        y, c1, c2, c3 = c[0, -1], c[1, -1], c[2, -1], c[3, -1]
        end = torch.stack([x["y"][cols, -1], c1 + 2 * c2 * hl + 3 * c3 * hl**2, c2 + 3 * c3 * hl, c3])
        coeffs[:, :, cols] = torch.cat([c, end[:, None, :]], dim=1)
        j = (torch.searchsorted(t, tn, right=True) - 1).clamp(0, N - 2)
        xx = (tn - t[j])[:, None]
        value[cols] = (c[0, j] + xx * (c[1, j] + xx * (c[2, j] + xx * c[3, j]))).T
        rate[cols] = (c[1, j] + xx * (2 * c[2, j] + xx * 3 * c[3, j])).T
    return {"coeffs": coeffs.reshape(-1), "value": value.squeeze(), "rate": rate.squeeze()}


def _bspline_matrix(knots, x):
    """Cubic B-splines on the knots at the points x: (points, len(knots) - 4), by Cox and de Boor."""
    k, x = np.asarray(knots), np.asarray(x)[:, None]
    last = np.max(np.nonzero(k[:-1] < k[1:])[0])
    B = ((x >= k[:-1]) & (x < k[1:])).astype(float)
    B[:, last] += (x[:, 0] >= k[last + 1])
    for d in range(1, 4):
        n = B.shape[1] - 1
        l, r = k[d:d + n] - k[:n], k[d + 1:d + 1 + n] - k[1:1 + n]
        with np.errstate(divide="ignore", invalid="ignore"):
            u = np.where(l > 0, (x - k[:n]) / l, 0.0)
            v = np.where(r > 0, (k[d + 1:d + 1 + n] - x) / r, 0.0)
        B = u * B[:, :-1] + v * B[:, 1:]
    return B


def _ylm(l, m, theta, phi):
    c, s = math.cos(theta / 2), math.sin(theta / 2)
    tot = 0.0
    for r in range(max(0, m + 2), min(l + 2, l + m) + 1):
        ec = 2 * r - 2 - m
        tot += (-1) ** (l - r + 2) * math.comb(l + 2, r) * math.comb(l - 2, r - 2 - m) * c**ec * s ** (2 * l - ec)
    f = math.factorial
    norm = math.sqrt(f(l + m) * f(l - m) * (2 * l + 1) / (4 * math.pi * f(l - 2) * f(l + 2)))
    return (-1) ** m * norm * tot * complex(math.cos(m * phi), math.sin(m * phi))


def _select_exact(case, seed):
    t, w, u, theta, phi = _select_points(case, seed)
    g = GridAmplitudes(case["lmax"], case["nmax"], case["grid"], seed)
    q = case["grid"] - 4
    Bw, Bu = _dev(_bspline_matrix(g.knots, w)), _dev(_bspline_matrix(g.knots, u))
    l, m, k, n = (np.asarray(v).astype(np.int64) for v in (g.l_arr_no_mask, g.m_arr_no_mask, g.k_arr_no_mask,
                                                            g.n_arr_no_mask))
    K = len(l)
    parts = [torch.einsum("pi,kij,pj->pk", Bw, g.coeff[:, c].reshape(K, q, q), Bu) for c in (0, 1)]
    teuk = torch.complex(parts[0], parts[1])
    table = {(a, b): _ylm(a, b, theta, phi) for a, b in set(zip(l.tolist(), m.tolist())) | set(zip(l.tolist(), (-m).tolist()))}
    yp = _dev(np.array([table[a, b] for a, b in zip(l.tolist(), m.tolist())]))
    ym = _dev(np.array([table[a, -b] for a, b in zip(l.tolist(), m.tolist())]))
    md = _dev(m)
    power = (teuk * yp).abs() ** 2 + torch.where(md != 0, (teuk.conj() * ym).abs() ** 2, 0.0)
    snr = (power[:-1] * _dev(np.diff(t))[:, None]).sum(dim=0)
    vals, order = torch.sort(snr, descending=True, stable=True)
    cs = vals.cumsum(0)
    keep = torch.ones(K, dtype=torch.bool, device=DEV)
    keep[1:] = cs[:-1] < cs[-1] * (1 - case["threshold"]) ** 2
    kept = torch.sort(order[keep])[0]
    pick = [_dev(v)[kept] for v in (l, m, k, n)]
    return {"teuk": teuk[:, kept].contiguous(), "ylms": torch.cat([yp[kept], ym[kept]]), "l": pick[0], "m": pick[1],
            "k": pick[2], "n": pick[3]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "td":
        return _td_exact(_td_inputs(case, seed), case["backward"])
    if kind == "batch":
        return [_td_exact(_trajectory_inputs("lmn", K, N, T, s), "")["h"] for K, N, T, s in _batch_shapes(case, seed)]
    return {"fd": _fd_exact, "aak": _aak_exact, "direct": _direct_exact, "spline": _spline_exact,
            "select": _select_exact}[kind](case, seed)
