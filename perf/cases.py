"""The propagator's workloads: what a program that uses this library has it do, through the public
Python API (``pySWE``), over the sizes the configurations, tests and benchmark use.

A case is one of

* ``solve``: a set-up propagation taken back to its equilibrium and run over the whole pulse, and its
  current read (a repeated solve; ``rho`` reads the propagated density matrix too);
* ``new``: the reference's polarisation-scan loop for one angle: settings, setup, run, current and
  spectrum of a solve that did not exist before;
* ``scan``: several angles of one or more models as one batch;
* ``spectrum``: the post-processing alone, spectra and harmonic intensities of recorded currents.

Models are synthetic tight-binding files made from the seed (``tbgen``); so are the pulse's intensity and
phases.  ``exact`` restates the propagation in complex128 torch: separable structure, tables and layouts of
the library are not used, only the equations.
"""
import ctypes
import math
import os
import sys
import tempfile

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hhg-solids_b200"))
import tbgen  # noqa: E402
from pySWE import pyswe  # noqa: E402

DT = 21.97e-3  # fs
A_LAT = 2.5    # Angstrom


def _solve(name, nw, n1, n2, nt, pol, window=7, precision="fp64", solver="rspace", kind="solve", rho=False, count=1,
           lam=3000.0):
    c = dict(kind=kind, nw=nw, window=window, n1=n1, n2=n2, nt=nt, pol=pol, precision=precision, solver=solver, rho=rho,
             count=count, lam=lam)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # The 2-orbital model under the full pulse: the small grid a user starts with, where a step is a
        # chain of dependent operations on few warps, and the converged grid.
        _solve("two_band_60", 2, 60, 60, 4096, 90.0, window=5),
        _solve("two_band_200", 2, 200, 200, 4096, 90.0, window=5),
        # The same converged grid with the k-space (interpolating) solver.
        _solve("two_band_200_kspace", 2, 200, 200, 4096, 90.0, window=5, solver="kspace"),
        # The 11-orbital benchmark configuration in both precisions.
        _solve("tmd11_150", 11, 150, 150, 4096, 90.0),
        _solve("tmd11_150_mixed", 11, 150, 150, 4096, 90.0, precision="mixed"),
        # An off-axis angle of a polarisation scan (two field components) on a 6-orbital model.
        _solve("tmd6_100_angle", 6, 100, 100, 4096, 30.0),
        # 12 orbitals, k-space solver, few-cycle pulse, off-axis.
        _solve("tmd12_64_kspace_angle", 12, 64, 64, 1024, 45.0, solver="kspace"),
        # A model whose shape nothing is compiled for, on a ragged grid, with its final density matrix.
        _solve("tmd5_46x38", 5, 46, 38, 1024, 63.0, window=5, rho=True),
        # A batch of angles over the three model sizes, mixed form (the scan workload).
        _solve("scan_9_mixed", 0, 60, 60, 1024, 0.0, precision="mixed", kind="scan", count=9),
        # One angle of the reference's scan loop from nothing: parse, setup, run, current, spectrum.
        _solve("new_tmd6_40", 6, 40, 40, 512, 15.0, kind="new"),
        # Spectra and harmonic intensities of one solve's current, and of a scan's.
        _solve("spectrum_1", 0, 0, 0, 4096, 0.0, kind="spectrum", count=1),
        _solve("spectrum_64", 0, 0, 0, 4096, 0.0, kind="spectrum", count=64),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["solve"] * 7 + ["new", "scan", "spectrum"])
    if kind == "spectrum":
        return _solve(None, 0, 0, 0, int(_log(rng, 512, 8192)), 0.0, kind=kind, count=int(_log(rng, 1, 100)))
    nt = int(_log(rng, 256, 4096))
    pol = round(rng.choice([0.0, 90.0, rng.uniform(1.0, 179.0)]), 1)
    lam = rng.choice([2000.0, 3000.0])
    if kind == "scan":
        n = 2 * int(_log(rng, 10, 40))
        return _solve(None, 0, n, n, min(nt, 1024), 0.0, precision="mixed", kind=kind, count=rng.randint(3, 12), lam=lam)
    nw = rng.choice([2, 2, 3, 4, 5, 6, 6, 8, 10, 11, 11, 12])
    solver = rng.choice(["rspace", "rspace", "kspace"])
    precision = "mixed" if nw in (6, 11, 12) and rng.random() < 0.3 else "fp64"
    # the largest costs no more than the 11-orbital benchmark grid under the full pulse
    side = min(200.0, math.sqrt(3.5e9 / (nt * max(nw, 4) ** 2)))
    n1 = 2 * max(7, int(_log(rng, 14, side) / 2))
    n2 = n1 if solver == "kspace" else 2 * max(7, int(n1 * rng.uniform(0.7, 1.0) / 2))
    return _solve(None, nw, n1, n2, nt if kind == "solve" else min(nt, 1024), pol, window=rng.choice([5, 7]) if nw > 2 else 5,
                  precision=precision, solver=solver, kind=kind, rho=rng.random() < 0.3 and kind == "solve", lam=lam)


# ---------------------------------------------------------------------------------------- inputs

_TMP = None


def _model(nw, window, seed):
    """A model file of its own for this seed; 2 orbitals: the Haldane-like model, else a random TMD-like one."""
    global _TMP
    if _TMP is None:
        _TMP = tempfile.mkdtemp(prefix="hhg_cases_")
    path = os.path.join(_TMP, f"m{nw}_{window}_{seed}_tb.dat")
    if nw == 2:
        u = np.random.default_rng(seed).uniform(-1, 1, 3)
        tbgen.haldane(path, a=A_LAT, onsite=0.8 * (1 + 0.1 * u[0]), t1=-2.7 * (1 + 0.05 * u[1]), t2=0.1 * (1 + 0.2 * u[2]))
    else:
        tbgen.random_tmd(path, nw=nw, seed=seed, window=window, a=A_LAT)
    return path


def _param(case, seed, nw=None, pol=None):
    nw = case["nw"] if nw is None else nw
    pol = math.radians(case["pol"] if pol is None else pol)
    vec = np.array([math.cos(pol), math.sin(pol), 0.0])
    vec[np.abs(vec) < 1e-12] = 0.0
    u = np.random.default_rng(seed + 77).uniform(0, 1, 3)
    tmax = (case["nt"] + 0.5) * DT
    return {"path_tb": _model(nw, 5 if nw == 2 else case["window"], seed), "nr1": case["n1"], "nr2": case["n2"], "nr3": 1,
            "tmax": tmax, "dt": DT, "intensity": 0.5e12 * (1 + 3 * u[0]), "lambda": case["lam"],
            "tmax_field": tmax * 8.0 / 9.0, "pol_vec": vec, "phi_vec": np.array([0.3 * u[1], 0.3 * u[2], 0.0])}


def _scan_params(case, seed):
    """The batch's solves: models of 2, 6 and 11 orbitals in turn, angles spread over the half circle."""
    n = case["count"]
    return [_param(case, seed, nw=(2, 6, 11)[i % 3], pol=180.0 * i / n) for i in range(n)]


def _signals(case, seed):
    """Recorded currents [3 count, nt] in host memory, as scans keep them: harmonics under an envelope."""
    rng = np.random.default_rng(seed)
    n, rows = case["nt"], 3 * case["count"]
    t = np.arange(n) * DT
    env = np.sin(np.pi * np.arange(n) / n) ** 2
    w0 = 2.0 * np.pi * 300.0 / case["lam"]
    J = np.zeros((rows, n), dtype=np.complex128)
    for h in (1, 3, 5, 7, 9, 15):
        J += (rng.standard_normal((rows, 1)) * np.exp(-0.4 * h)) * np.cos(h * w0 * t + rng.uniform(0, 6.28, (rows, 1)))
    return (J + 1e-6j * rng.standard_normal((rows, n))) * env * 1e-3


def _swe(case, param):
    return pyswe.SWE(pyswe.Settings(param), precision=case["precision"], solver=case["solver"])


def _harmonics(case):
    return 25 if case["lam"] > 2500 else 15


def prepare(case, seed):
    if case["kind"] == "spectrum":
        return {"case": case, "J": _signals(case, seed)}
    if case["kind"] == "scan":
        solves = [_swe(case, p) for p in _scan_params(case, seed)]
        return {"case": case, "solves": solves, "batch": pyswe.SWEBatch(solves)}
    param = _param(case, seed)
    if case["kind"] == "new":
        return {"case": case, "param": param}
    return {"case": case, "swe": _swe(case, param)}


def _current(swe):
    t, jx, jy, jz = swe.get_current()
    return {"t": t.real, "jx": jx, "jy": jy, "jz": jz}


def run(state):
    case = state["case"]
    if case["kind"] == "spectrum":
        S = pyswe.spectrum(state["J"], DT)
        return {"spectrum": S, "harmonics": pyswe.harmonic_intensities(S, case["nt"] * DT, case["lam"], _harmonics(case))}
    if case["kind"] == "scan":
        state["batch"].run()
        return [_current(s) for s in state["solves"]]
    if case["kind"] == "new":
        swe = _swe(case, state["param"])
        swe.run_simulation()
        out = _current(swe)
        out["spectrum"] = swe.get_spectrum()
        swe.delete()
        return out
    swe = state["swe"]
    swe.reset()
    swe.run_simulation()
    out = _current(swe)
    if case["rho"]:
        out["rho"] = swe.get_rho_k()
    return out


# ---------------------------------------------------------------------------------------- work


def _solve_work(case, nw, naxes):
    """Minimal operations of a k-point step (Hermitian commutators, separable Wannier sums, windowed
    current) and the state and current once in and out."""
    W = 5 if nw == 2 else case["window"]
    points = 2 if case["solver"] == "kspace" else 1
    flops = 32.0 * nw**3 + points * 8.0 * nw * nw * (1 + naxes) * W * (1 + W / case["n1"])
    flops += 2 * 8.0 * nw * nw * (4 * (1 + 4.0 / case["n1"]) + 1) + 12.0 * nw * nw
    nk = case["n1"] * case["n2"]
    nbytes = 2 * 16.0 * nk * nw * nw + 16.0 * 3 * case["nt"] + 16.0 * (1 + naxes) * W * W * nw * nw
    return nbytes, flops * nk * case["nt"]


def work(case):
    n = case["nt"]
    if case["kind"] == "spectrum":
        rows = 3 * case["count"]
        return {"bytes": 2 * 16.0 * rows * n + 8.0 * rows * _harmonics(case), "flops": rows * (5.0 * n * math.log2(n) + 7.0 * n)}
    if case["kind"] == "scan":
        parts = [_solve_work(case, (2, 6, 11)[i % 3], 1 if (180.0 * i / case["count"]) % 90.0 == 0 else 2)
                 for i in range(case["count"])]
    else:
        parts = [_solve_work(case, case["nw"], 1 if case["pol"] % 90.0 == 0 else 2)]
    b, f = (sum(p[q] for p in parts) for q in (0, 1))
    if case["kind"] == "new":
        f += 3 * 5.0 * n * math.log2(n)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------------------- exact values

EV2HA, A2BOHR, FS2AU = 1.0 / 27.2114, 1.0 / 0.5291772, 1.0 / 0.02418884


def _read_tb(path):
    """(lattice, [(n1, n2)], stored H [cells, nw, nw], stored x [3, cells, nw, nw]) of a model file."""
    with open(path) as f:
        lines = f.read().split("\n")
    lat = np.array([[float(v) for v in lines[1 + i].split()] for i in range(3)])
    nw, nc = int(lines[4]), int(lines[5])
    at = 6 + (nc + 14) // 15 + 1
    cells, H, X = [], np.zeros((nc, nw, nw), complex), np.zeros((3, nc, nw, nw), complex)
    for part in range(2):
        for c in range(nc):
            if part == 0:
                cells.append(tuple(int(v) for v in lines[at].split()[:2]))
            v = np.array([ln.split()[2:] for ln in lines[at + 1:at + 1 + nw * nw]], dtype=float).reshape(nw, nw, -1)
            if part == 0:
                H[c] = v[..., 0] + 1j * v[..., 1]
            else:
                for a in range(3):
                    X[a, c] = v[..., 2 * a] + 1j * v[..., 2 * a + 1]
            at += nw * nw + 2
    return lat, cells, H, X


_SINF = ctypes.CDLL("libm.so.6").sinf
_SINF.argtypes, _SINF.restype = [ctypes.c_float], ctypes.c_float


def _field(param, nt):
    """t, E, A in atomic units; the method's carrier is the C library's single-precision sine, its peak a
    single-precision square root."""
    t = np.arange(nt) * param["dt"] * FS2AU
    omega = 2.0 * np.pi * 2997.025 / (param["lambda"] * 10.0) / FS2AU
    tf = param["tmax_field"] * FS2AU
    peak = float(np.sqrt(np.float32(param["intensity"] / 3.56e16)))
    env = np.where(t < tf, np.sin(np.pi * t / tf) ** 2, 0.0)
    E = np.zeros((3, nt))
    for a in range(3):
        carrier = np.array([_SINF(x) for x in omega * t + param["phi_vec"][a]])
        E[a] = param["pol_vec"][a] * peak * env * carrier
    A = np.zeros((3, nt))
    A[:, 1:] = -np.cumsum(E[:, :-1], axis=1) * (t[1] - t[0])
    return t, E, A


def _exact_solve(case, param):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n1g, n2g, nt, kspace = case["n1"], case["n2"], case["nt"], case["solver"] == "kspace"
    lat, cells, Hm, Xm = _read_tb(param["path_tb"])
    nw, nw2, nk = Hm.shape[1], Hm.shape[1] ** 2, n1g * n2g
    t, E, A = _field(param, nt)
    dt = t[1] - t[0]
    axes = [a for a in range(3) if param["pol_vec"][a] != 0.0]
    # Placement on the grid: the method truncates each cell's fractional coordinates, which on this lattice
    # reads the blocks of the corner cells (3, 2) and (-3, -2) from the cells beside them.
    index = {c: i for i, c in enumerate(cells)}
    moved = {(3, 2): (3, 1), (-3, -2): (-3, -1)}
    where = {c: index[moved.get(c, c)] for c in cells
             if -n1g // 2 <= c[0] < n1g // 2 and -n2g // 2 <= c[1] < n2g // 2}
    pos = list(where)
    src = [where[c] for c in pos]
    h0, r = Hm[src] * EV2HA, -Xm[:, src] * A2BOHR
    # Velocity i [H, r] plus the intracell part on the 4 x 4 window, in eV and Angstrom as the method has it.
    win = [(a, b) for a in range(-2, 2) for b in range(-2, 2)]
    vel = np.zeros((3, 16, nw, nw), complex)
    for w, (a, b) in enumerate(win):
        s = where.get((a, b))
        for ax in range(3):
            acc = np.zeros((nw, nw), complex)
            for q in pos:
                d = ((a - q[0] + n1g // 2) % n1g - n1g // 2, (b - q[1] + n2g // 2) % n2g - n2g // 2)
                if d in where:
                    iq, idd = where[q], where[d]
                    acc += -Xm[ax, iq] @ Hm[idd] + Hm[iq] @ Xm[ax, idd]
            Rw = a * lat[0, ax] + b * lat[1, ax]
            vel[ax, w] = 1j * ((Rw * Hm[s] if s is not None else 0.0) - acc)
    jax = [a for a in range(3) if np.any(vel[a] != 0)]

    c128 = dict(dtype=torch.complex128, device=dev)
    m1, m2 = np.divmod(np.arange(nk), n2g)

    def waves(ns):  # e^{-i k.R} of every k-point and cell
        x = np.array([n[0] for n in ns]), np.array([n[1] for n in ns])
        ang = -2.0 * np.pi * ((m1[:, None] * x[0][None]) % n1g / n1g + (m2[:, None] * x[1][None]) % n2g / n2g)
        return torch.polar(torch.ones(ang.shape, dtype=torch.float64, device=dev), torch.tensor(ang, device=dev))

    # The k-space solver reads the grid with its two indices exchanged (square grids).
    eval_pos = [(c[1], c[0]) for c in pos] if kspace else pos
    wk, ww = waves(eval_pos), waves(win)
    ops = torch.tensor(np.stack([h0] + [r[a] for a in axes], axis=1).reshape(len(pos), -1), **c128)
    vop = torch.tensor(np.stack([vel[a] for a in jax], axis=1).reshape(16, -1), **c128)
    Rc, Rw = (np.array([[n[0] * lat[0, a] + n[1] * lat[1, a] for a in range(3)] for n in ns]) * A2BOHR for ns in (pos, win))

    def interp_factors():
        """[2 nt + 1, cells]: the Catmull-Rom interpolation at k - A acts on a cell as one factor per direction."""
        B = np.zeros((3, 3))
        vol = np.dot(lat[0], np.cross(lat[1], lat[2]))
        for i in range(3):
            B[i] = 2 * np.pi * np.cross(lat[(i + 1) % 3], lat[(i + 2) % 3]) / vol / A2BOHR
        pts = np.zeros((2 * nt + 1, 3))
        pts[0:2 * nt:2] = A.T
        pts[1:2 * nt - 1:2] = 0.5 * (A.T[:-1] + A.T[1:])
        pts[2 * nt - 1] = pts[2 * nt] = A[:, -1]
        u = np.linalg.solve(B.T, pts.T).T
        out = np.ones((2 * nt + 1, len(pos)), complex)
        for d in range(2):
            x = -u[:, d] * n1g
            o = np.floor(x)
            f = x - o
            taps = [((-0.5 * f + 1.0) * f - 0.5) * f, (1.5 * f - 2.5) * f * f + 1.0, ((-1.5 * f + 2.0) * f + 0.5) * f,
                    (0.5 * f - 0.5) * f * f]
            n = np.array([c[d] for c in eval_pos])
            out *= sum(taps[i][:, None] * np.exp(-2j * np.pi * (((o + i - 1)[:, None] * n[None]) % n1g) / n1g) for i in range(4))
        return out

    ph = interp_factors() if kspace else np.exp(1j * (A.T @ Rc.T))
    pw = np.ones((nt, 16), complex) if kspace else np.exp(1j * (A.T @ Rw.T))
    ph, pw = torch.tensor(ph, **c128), torch.tensor(pw, **c128)

    h = (waves(pos) @ torch.tensor(h0.reshape(len(pos), -1), **c128)).reshape(nk, nw, nw)
    low = torch.tril(h)
    _, U = torch.linalg.eigh((low + torch.tril(h, -1).mH).cpu())  # (the lower triangle)
    U = U.to(dev)
    occ = (torch.einsum("kpn,kpq,kqn->kn", U.conj(), h, U).real < 0).to(torch.complex128)
    rho = (U * occ[:, None, :]) @ U.mH

    def product(a, b):
        if nw > 4:
            return a @ b
        return sum(a[:, :, q, None] * b[:, None, q, :] for q in range(nw))

    def matrices(p):
        return (wk @ (ph[p][:, None] * ops)).reshape(nk, 1 + len(axes), nw, nw)

    def field_h(m, e):
        hh = m[:, 0]
        for q, a in enumerate(axes):
            hh = hh + e[a] * m[:, 1 + q]
        return hh

    J = torch.zeros((3, nt), **c128)
    m_next = matrices(0) if kspace else None
    wnow = (ww @ vop).reshape(nk, len(jax), nw, nw) if kspace else None
    for i in range(nt):
        e0 = E[:, i]
        e2 = E[:, min(i + 1, nt - 1)]
        e1 = 0.5 * e0 + 0.5 * e2
        if kspace:
            ma, mb, mc = m_next, matrices(2 * i + 1), matrices(2 * i + 2)
            m_next = mc
        else:
            ma = mb = mc = matrices(i)
            wnow = (ww @ (pw[i][:, None] * vop)).reshape(nk, len(jax), nw, nw)
        ha, hb, hc = field_h(ma, e0), field_h(mb, e1), field_h(mc, e2)
        acc, k = None, None
        for hs, cs, wt in ((ha, 0.0, 1.0), (hb, 0.5 * dt, 2.0), (hb, 0.5 * dt, 2.0), (hc, dt, 1.0)):
            x = rho if k is None else rho + cs * k
            k = -1j * (product(hs, x) - product(x, hs))
            acc = wt * k if acc is None else acc + wt * k
        rho = rho + (0.1666666666666 * dt) * acc
        J[jax, i] = (wnow * rho.conj()[:, None]).sum(dim=(0, 2, 3)) / nk
    J = J.cpu().numpy()
    return {"t": t, "jx": J[0], "jy": J[1], "jz": J[2]}, rho.reshape(nk, nw2).cpu().numpy()


def _spectrum(J, spacing):
    g = np.gradient(J, spacing, axis=-1)
    return np.fft.fftshift(np.fft.fft(np.fft.ifftshift(g, axes=-1), axis=-1), axes=-1)


def _exact_seconds(case, nw):
    nk = case["n1"] * case["n2"]
    return case["nt"] * (2.5e-3 + nk * nw * nw * (8e-10 if case["solver"] == "rspace" else 1.2e-9))


def exact(case, seed):
    if case["kind"] == "spectrum":
        S = _spectrum(_signals(case, seed), DT)
        n, tmax, nh = case["nt"], case["nt"] * DT, _harmonics(case)
        order = np.linspace(-n * np.pi / tmax, n * np.pi / tmax, n) / (2.0 * np.pi * 300.0 / case["lam"])
        P = np.abs(S) ** 2
        I = np.stack([P[:, (order > h - 0.5) & (order < h + 0.5)].sum(axis=1) for h in range(1, 2 * nh, 2)], axis=1)
        return {"spectrum": S, "harmonics": I}
    if case["kind"] == "scan":
        if sum(_exact_seconds(case, (2, 6, 11)[i % 3]) for i in range(case["count"])) > 18.0:
            return None
        return [_exact_solve(case, p)[0] for p in _scan_params(case, seed)]
    if _exact_seconds(case, case["nw"]) > 18.0:
        return None
    out, rho = _exact_solve(case, _param(case, seed))
    if case["kind"] == "new":
        out["spectrum"] = [_spectrum(out[j], DT) for j in ("jx", "jy", "jz")]
    elif case["rho"]:
        out["rho"] = rho
    return out
