"""Performance cases of tbplas_b200: the calls that a TBPM program makes, over the sizes it makes them at.

Every case is one call of a driver of `tbplas_b200.fortran.f2py` (what `Solver.calc_*` calls) on a graphene
sample: small and ordinary samples hand over a host CSR matrix, as `Solver` does with a `LatticeSample`, large
ones the handle of a `DeviceSample`, which the call assembles on the GPU.  Sizes follow the benchmark
configurations, scaled down where a full run takes minutes; lattices that are no powers of two, odd numbers of
states, vacancies, open boundaries and a magnetic field stand for the samples of real studies.

`exact` evaluates each driver's definition by plain time stepping in 64 bits with torch.
"""

import math
import random

import numpy as np
import torch

from tbplas_b200.builder import make_graphene_sample, pack_samples
from tbplas_b200.fortran import f2py
from tbplas_b200.supercell import make_graphene_device_sample

RESCALE = 9.0          # eV: above 3 * 2.7 + 0.5, the largest row sum at W = 1 eV
BETA = 1.0 / (8.617333262145e-5 * 300) * RESCALE
CHECK = (128, 1.0e-9)  # Config.generic: wfn_check_steps, wfn_check_thr
NR_FERMI, FERMI_EPS = 2 ** 15, 1.0e-12
A_CC = 0.246           # lattice constant, nm


def listed():
    d = {"prec": "fp64", "disorder": 1.0, "vacancy": 0.0, "field": 0.0, "pbc": True}
    return [
        # the documented first run: a clean 100 x 100 supercell, one state, 256 steps; every launch counts
        {**d, "name": "dos_100x100", "kind": "dos", "nx": 100, "ny": 100, "states": 1, "steps": 256, "disorder": 0.0},
        # an ordinary study: a ragged flake with vacancies and open edges, an odd number of states
        {**d, "name": "dos_flake", "kind": "dos", "nx": 251, "ny": 190, "states": 5, "steps": 300, "vacancy": 0.01,
         "pbc": False},
        # a large disordered sample, 16 states as one block
        {**d, "name": "dos_large", "kind": "dos", "nx": 1600, "ny": 1500, "states": 16, "steps": 64},
        # single-precision states, as for the training curves of the tail extrapolator
        {**d, "name": "dos_fp32", "kind": "dos", "nx": 1024, "ny": 1000, "states": 16, "steps": 128, "prec": "fp32"},
        # a batch of uneven disorder realisations propagated together
        {**d, "name": "dos_batch", "kind": "seg", "segments": 20, "lo": 96, "hi": 280, "states": 4, "steps": 128,
         "vacancy": 0.01},
        # optical conductivity
        {**d, "name": "ac", "kind": "ac", "nx": 512, "ny": 500, "states": 8, "steps": 256},
        # DC conductivity in a field, single-precision states, the default energy window
        {**d, "name": "dc_field", "kind": "dc", "nx": 384, "ny": 400, "states": 4, "steps": 512, "field": 77.06,
         "prec": "fp32"},
        # dynamical polarisation of one state at two q-points
        {**d, "name": "dyn_pol", "kind": "dynpol", "nx": 800, "ny": 600, "states": 1, "steps": 256, "n_q": 2},
        # quasi-eigenstates around the Dirac point
        {**d, "name": "quasi_eigenstates", "kind": "qe", "nx": 320, "ny": 301, "states": 2, "steps": 256, "n_en": 7},
        # Kubo-Bastin moments for the Hall conductivity
        {**d, "name": "hall_moments", "kind": "kbdc", "nx": 200, "ny": 180, "states": 1, "n_kernel": 768},
        # local DOS of a site by the Haydock recursion
        {**d, "name": "ldos_haydock", "kind": "haydock", "nx": 512, "ny": 512, "states": 1, "steps": 256, "depth": 500},
        # a wave packet's propagation with a few frames kept
        {**d, "name": "psi_t", "kind": "psi_t", "nx": 512, "ny": 480, "states": 1, "steps": 256, "frames": 5},
    ]


def draw(rng: random.Random):
    """A call of the same kinds and ranges, no costlier than the largest listed one."""
    limit = max(_stepping_bytes(c) for c in listed())

    def between(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["dos", "dos", "dos", "seg", "ac", "dc", "dynpol", "qe", "kbdc", "haydock", "psi_t"])
    while True:
        big = {"dos": 1800, "ac": 600, "dc": 400, "dynpol": 900, "qe": 400, "kbdc": 240, "haydock": 700, "psi_t": 700,
               "seg": 300}[kind]
        c = {"kind": kind, "prec": rng.choice(["fp64", "fp64", "fp32"]), "nx": between(64, big), "ny": between(64, big),
             "disorder": round(rng.uniform(0.0, 1.0), 3), "vacancy": rng.choice([0.0, 0.0, 0.01]),
             "field": rng.choice([0.0, 0.0, 40.0]), "pbc": rng.random() < 0.8, "states": 1}
        if kind in ("dos", "ac", "dc"):
            c["states"] = between(1, {"dos": 16, "ac": 8, "dc": 6}[kind])
        if kind in ("dynpol", "qe", "seg"):
            c["states"] = rng.randint(1, 4)
        if kind not in ("kbdc",):
            c["steps"] = between(64, 512)
        if kind == "seg":
            del c["nx"], c["ny"], c["field"], c["pbc"]
            c["segments"], c["lo"] = rng.randint(4, 24), between(48, 120)
            c["hi"] = c["lo"] + between(16, 180)
        if kind == "dynpol":
            c["n_q"] = rng.randint(1, 3)
        if kind == "qe":
            c["n_en"] = rng.randint(3, 16)
        if kind == "kbdc":
            c["n_kernel"] = between(128, 768)
        if kind in ("haydock", "psi_t"):
            c["prec"] = "fp64"
        if kind == "haydock":
            c["depth"] = between(100, max(101, min(c["nx"], c["ny"])))  # below the sample's linear size
        if kind == "psi_t":
            c["frames"] = rng.randint(2, 9)
        if _stepping_bytes(c) <= limit:
            return c


# ---- what a program has before the call -----------------------------------------------------------------------

def _bessel(z: float):
    """J_k(z) down to 1e-14 (the integral of cos(k t - z sin t) over a period, exact at 512 points)."""
    t = 2 * np.pi * np.arange(512) / 512
    b = [float(np.mean(np.cos(k * t - z * np.sin(t)))) for k in range(60)]
    n = max(k for k in range(60) if abs(b[k]) > 1e-14)
    return np.array(b[:n + 1])


def _energies(steps: int):
    """The energy grid and window of the DC conductivity (Config.DC_conductivity's default limits)."""
    e = np.array([0.5 * i * 2 * RESCALE / steps - RESCALE for i in range(2 * steps)])
    return e, np.where((e >= -0.5) & (e <= 0.5))[0]


def _frames(c):
    return np.unique(np.round(np.linspace(0, c["steps"], c["frames"])).astype(np.int64))


def _q_points(c):
    return np.array([[0.7 * (k + 1), 0.4 * k, 0.0] for k in range(c["n_q"])])


def _qe_energies(c):
    return np.linspace(-0.3, 0.3, c["n_en"])


def _segment_dims(c):
    r = random.Random(7)
    return [(r.randint(c["lo"], c["hi"]), r.randint(c["lo"], c["hi"])) for _ in range(c["segments"])]


def prepare(case, seed):
    c = dict(case)
    seed = int(seed) % (1 << 15) + 1
    s = {"case": c, "seed": seed, "bes": _bessel(math.pi if c["kind"] not in ("ac", "dynpol") else math.pi / 2)}
    if c["kind"] == "seg":
        packed = pack_samples([make_graphene_sample(nx, ny, rescale=RESCALE, disorder=c["disorder"],
                                                    vacancy_rate=c["vacancy"], seed=seed + i)
                               for i, (nx, ny) in enumerate(_segment_dims(c))])
        s["ham"] = (packed.indptr, packed.indices, packed.data)
        s["offsets"] = packed.offsets
        return s
    make = make_graphene_sample if c["nx"] * c["ny"] < 60000 else make_graphene_device_sample
    sample = make(c["nx"], c["ny"], rescale=RESCALE, pbc=c["pbc"], disorder=c["disorder"], vacancy_rate=c["vacancy"],
                  b_field=c["field"], seed=seed)
    if c["kind"] in ("ac", "dc", "dynpol", "kbdc"):
        ip, ix, hop, dx, dy = sample.build_ham_dxy()
        s["ham"], s["dxy"] = (ip, ix, hop), (dx, dy)
    else:
        h = sample.build_ham_csr()
        s["ham"] = (h.indptr, h.indices, h.data)
    if c["kind"] == "dynpol":
        s["sites"] = [np.ascontiguousarray(sample.orb_pos[:, k]) for k in range(3)]
    if c["kind"] == "psi_t":
        r = np.random.default_rng(seed)
        p = r.standard_normal(sample.num_orb) + 1j * r.standard_normal(sample.num_orb)
        s["psi0"] = p / np.linalg.norm(p)
    return s


def run(s):
    c, seed, bes = s["case"], s["seed"], s["bes"]
    f2py.set_backend(precision=c["prec"], batch=16)
    n = c["states"]
    kind = c["kind"]
    if kind == "dos":
        out = f2py.tbpm_dos(bes, *s["ham"], seed, c["steps"], n, "", 0, *CHECK)
    elif kind == "seg":
        out = f2py.tbpm_dos_segmented(bes, *s["ham"], s["offsets"], n, seed, c["steps"], *CHECK)
    elif kind == "ac":
        out = f2py.tbpm_accond(bes, BETA, 0.0, *s["ham"], RESCALE, *s["dxy"], seed, c["steps"], n, NR_FERMI,
                               FERMI_EPS, "", 0, *CHECK)
    elif kind == "dc":
        e, sel = _energies(c["steps"])
        out = f2py.tbpm_dccond(bes, BETA, 0.0, *s["ham"], RESCALE, *s["dxy"], seed, c["steps"], n,
                               math.pi / RESCALE, e, sel, "", "", 0, *CHECK)
    elif kind == "dynpol":
        out = f2py.tbpm_dyn_pol(bes, BETA, 0.0, *s["ham"], RESCALE, *s["dxy"], *s["sites"], seed, c["steps"], n,
                                NR_FERMI, FERMI_EPS, _q_points(c), "", 0, *CHECK)
    elif kind == "qe":
        out = f2py.tbpm_eigenstates(bes, *s["ham"], seed, c["steps"], n, math.pi / RESCALE, _qe_energies(c), 0, *CHECK)
    elif kind == "kbdc":
        out = f2py.tbpm_kbdc(seed, *s["ham"], RESCALE, *s["dxy"], n, c["n_kernel"], 1, 0)
    elif kind == "haydock":
        out = f2py.ldos_haydock([0], 0.01, 2 * RESCALE, *s["ham"], RESCALE, seed, c["depth"], c["steps"], n, "")
    else:
        out = f2py.tbpm_psi_t(bes, *s["ham"], s["psi0"], _frames(c), c["steps"], *CHECK)
    if c["prec"] == "fp32":
        # results of single-precision states are kept in single precision (as learned.curves_to_xy does)
        single = {np.dtype("complex128"): np.complex64, np.dtype("float64"): np.float32}
        cast = lambda x: x.astype(single[x.dtype])  # noqa: E731
        out = tuple(map(cast, out)) if isinstance(out, tuple) else cast(out)
    return out


# ---- what a pass cannot do without ------------------------------------------------------------------------------

def _rows(c):
    if c["kind"] == "seg":
        return sum(2 * nx * ny for nx, ny in _segment_dims(c))
    return 2 * c["nx"] * c["ny"]


def _block(c):
    """Bytes of one pass over the matrix, and over the state block."""
    v = 16 if c["prec"] == "fp64" else 8
    cols = c["states"] * {"ac": 3, "dynpol": 1 + c.get("n_q", 0)}.get(c["kind"], 1)
    return _rows(c) * (3 * (4 + v) + v + 4), _rows(c) * cols * v, cols


def _stepping_bytes(c):
    """Bytes of the same call by plain time stepping, the yardstick of a case's cost."""
    mat, vec, _ = _block(c)
    if c["kind"] == "kbdc":
        return 2 * c["n_kernel"] * (mat + 3 * vec) + c["n_kernel"] ** 2 * _rows(c) / 2
    if c["kind"] == "haydock":
        return c["depth"] * (mat + 9 * vec)
    terms = c["steps"] * (15 if c["kind"] in ("ac", "dynpol") else 20)
    terms += 3061 if c["kind"] in ("ac", "dynpol") else 0
    both = 4 if c["kind"] == "dc" else 2 if c["kind"] == "qe" else 1
    qe = c["steps"] * c.get("n_en", c["steps"] / 9) * vec if both > 1 else 0
    return terms * (mat + 4 * vec * both) + qe


def work(case):
    """The Hamiltonian is applied as often as the degree of the call's polynomials asks for (a moment sum of T steps
    of phase z needs z T / 2 applications: two moments each); an application reads the matrix and the two last
    blocks and writes one."""
    c = dict(case)
    mat, vec, cols = _block(c)
    n, v = _rows(c), 16 if c["prec"] == "fp64" else 8
    apply_flops = n * cols * (3 * 8 + 8)
    steps = c.get("steps", 0)
    extra_b = extra_f = 0.0
    if c["kind"] in ("dos", "seg"):
        terms = 0.5 * math.pi * steps
    elif c["kind"] in ("ac", "dynpol"):
        terms = 3061 + 0.5 * math.pi * steps
        extra_b, extra_f = steps * (mat + vec), steps * n * cols * 60.0
    elif c["kind"] in ("dc", "qe"):
        n_en = c["n_en"] if c["kind"] == "qe" else len(_energies(steps)[1])
        terms = math.pi * steps * (3 if c["kind"] == "dc" else 1)
        extra_f = steps * n * c["states"] * n_en * 8.0 * (3 if c["kind"] == "dc" else 1)
        extra_b = n * c["states"] * n_en * v * 2.0
    elif c["kind"] == "kbdc":
        terms = 2 * c["n_kernel"]
        extra_f, extra_b = 8.0 * c["n_kernel"] ** 2 * n, 2.0 * c["n_kernel"] * n * v
    elif c["kind"] == "haydock":
        terms = c["depth"]
    else:
        terms = math.pi * steps
        extra_b = len(_frames(c)) * n * 16.0
    return {"bytes": terms * (mat + 3 * vec) + extra_b, "flops": terms * apply_flops + extra_f}


# ---- the definitions, in 64 bits ---------------------------------------------------------------------------------

class _Graphene:
    """Rows of up to three neighbours and a diagonal, from the lattice's geometry and the sample's random draws."""

    def __init__(self, nx, ny, pbc, disorder, vacancy, field, seed, cutoff=0.0):
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        full = 2 * nx * ny
        r = np.random.default_rng(seed)
        keep = np.ones(full, dtype=bool)
        if vacancy > 0:
            keep[r.choice(full, size=int(round(vacancy * full)), replace=False)] = False
        n = int(keep.sum())
        eng = r.uniform(-0.5 * disorder, 0.5 * disorder, n) if disorder > 0 else np.zeros(n)
        eng[np.abs(eng / RESCALE) < cutoff] = 0.0  # on-site terms that build_ham_dxy drops
        keep = torch.from_numpy(keep).to(dev)
        new = torch.cumsum(keep.long(), 0) - 1
        i = torch.arange(full, device=dev)
        o, ib, ia = i % 2, (i // 2) % ny, i // 2 // ny
        a1 = np.array([A_CC, 0.0])
        a2 = np.array([A_CC * 0.5, A_CC * math.sqrt(0.75)])
        fa, fb = ia.double() + o.double() / 3.0, ib.double() + o.double() / 3.0
        x = fa * a1[0] + fb * a2[0]
        y = fb * a2[1]
        cols, vals, dxs, dys = [], [], [], []
        for da, db in ((0, 0), (1, 0), (0, 1)):
            # orbital 0 couples to orbital 1 of the cells (0, 0), (-1, 0), (0, -1), orbital 1 back
            sgn = 2 * o - 1
            ja, jb = ia + sgn * da, ib + sgn * db
            ok = torch.ones_like(keep) if pbc else (ja >= 0) & (ja < nx) & (jb >= 0) & (jb < ny)
            j = ((ja % nx) * ny + jb % ny) * 2 + 1 - o
            tau = (a1 + a2) / 3.0 - da * a1 - db * a2  # from orbital 0 to orbital 1
            dx, dy = -sgn.double() * tau[0], -sgn.double() * tau[1]
            phase = math.pi / 4135.666734 * field * dx * (y + y[j])
            ok = ok & keep[j]
            v = torch.polar(torch.full_like(y, 1.0), phase) * (-2.7 / RESCALE) * ok
            cols.append(torch.where(ok, new[j], 0)[keep])
            vals.append(v[keep])
            dxs.append(dx[keep])
            dys.append(dy[keep])
        self.n, self.dev = n, dev
        self.cols, self.vals = cols, vals
        self.diag = torch.from_numpy(eng / RESCALE).to(dev)[:, None]
        self.pos = (x[keep], y[keep])
        self.cur = [[1j * RESCALE * v * d for v, d in zip(vals, ds)] for ds in (dxs, dys)]

    def h(self, p):
        q = self.diag * p
        for c, v in zip(self.cols, self.vals):
            q += v[:, None] * p[c]
        return q

    def j(self, d, p):
        q = torch.zeros_like(p)
        for c, v in zip(self.cols, self.cur[d]):
            q += v[:, None] * p[c]
        return q

    def series(self, coef, p):
        """sum_k coef[k] T_k(H) p"""
        a, b = p, self.h(p)
        out = coef[0] * a + coef[1] * b
        for k in range(2, len(coef)):
            a, b = b, 2 * self.h(b) - a
            out += coef[k] * b
        return out

    def step(self, z, p, forward=True):
        b = _bessel(z)
        s = -1j if forward else 1j
        return self.series([(2 if k else 1) * b[k] * s ** k for k in range(len(b))], p)

    def states(self, seed, count, first=1):
        return torch.stack([_random_state(self.n, seed * (first + k) * 49741, self.dev) for k in range(count)], 1)


def _random_state(n, key, dev):
    """|z|^2 ~ Exp(1), uniform phase, from the Philox4x32-10 stream of the key; normalised."""
    mask = 0xffffffff
    j = torch.arange(n, device=dev, dtype=torch.int64)
    c = [j & mask, j >> 32, torch.full_like(j, 0x5442504D), torch.zeros_like(j)]
    k0, k1 = key & mask, (key >> 32) & mask

    def mul(a, m):
        p0, p1 = (a & 0xffff) * m, (a >> 16) * m  # below 2^48
        low = p0 + ((p1 & 0xffff) << 16)
        return (p1 >> 16) + (low >> 32), low & mask

    for _ in range(10):
        hi0, lo0 = mul(c[0], 0xD2511F53)
        hi1, lo1 = mul(c[2], 0xCD9E8D57)
        c = [hi1 ^ c[1] ^ k0, lo1, hi0 ^ c[3] ^ k1, lo0]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    f = ((c[0] >> 5).double() * 67108864.0 + (c[1] >> 6).double()) / 9007199254740992.0
    g = ((c[2] >> 5).double() * 67108864.0 + (c[3] >> 6).double()) / 9007199254740992.0
    r = torch.sqrt(-torch.log(1.0 - f))
    z = torch.polar(r, 2 * math.pi * g)
    return z / torch.linalg.vector_norm(z)


def _dots(a, b):
    return torch.sum(a.conj() * b, 0)


def _fermi_coef(one_minus):
    """Chebyshev coefficients of the (1 -) Fermi operator with the Jackson kernel, cut at FERMI_EPS."""
    e = np.cos(2 * np.pi * np.arange(NR_FERMI) / NR_FERMI)
    x = np.exp(-BETA * np.abs(e))
    f = np.where(e >= 0, x / (1 + x), 1 / (1 + x))
    re = np.fft.fft(1 - f if one_minus else f).real
    m = NR_FERMI // 2
    k = np.arange(m)
    q = np.pi / m
    g = ((m - k) * np.cos(q * k) + np.sin(q * k) / np.tan(q)) / m
    g[0] = 0.5
    c = g * re[:m] / m
    small = np.abs(c) < FERMI_EPS
    cut = np.nonzero(small[:-1] & small[1:])[0]
    return c[:cut[0] + 1] if cut.size else c


def _np(t):
    return t.cpu().numpy()


def _dos_curve(g, wf0, steps):
    p, out = wf0, [_dots(wf0, wf0).mean()]
    for _ in range(steps):
        p = g.step(math.pi, p)
        out.append(_dots(wf0, p).mean())
    return _np(torch.stack(out))


def exact(case, seed):
    c = dict(case)
    seed = int(seed) % (1 << 15) + 1
    if c["kind"] == "seg":
        out = []
        for i, (nx, ny) in enumerate(_segment_dims(c)):
            g = _Graphene(nx, ny, True, c["disorder"], c["vacancy"], 0.0, seed + i)
            out.append(_dos_curve(g, g.states(seed, c["states"], 1 + i * c["states"]), c["steps"]))
        return np.stack(out)
    if _stepping_bytes(c) > 1.5 * max(_stepping_bytes(x) for x in listed()):
        return None
    g = _Graphene(c["nx"], c["ny"], c["pbc"], c["disorder"], c["vacancy"], c["field"], seed,
                  1.0e-5 if c["kind"] in ("ac", "dc", "dynpol", "kbdc") else 0.0)
    kind, steps, ns = c["kind"], c.get("steps", 0), c["states"]
    if kind == "psi_t":
        r = np.random.default_rng(seed)
        p = r.standard_normal(g.n) + 1j * r.standard_normal(g.n)
        p = torch.from_numpy(p / np.linalg.norm(p)).to(g.dev)[:, None]
        want, out = set(_frames(c).tolist()), []
        for t in range(steps + 1):
            if t in want:
                out.append(_np(p[:, 0]))
            p = g.step(math.pi, p)
        return np.stack(out, 1)
    if kind == "haydock":
        v = torch.zeros(g.n, 1, dtype=torch.complex128, device=g.dev)
        v[0] = _random_state(1, seed * 49741, g.dev)
        a, b, prev = [], [], torch.zeros_like(v)
        for d in range(c["depth"]):
            w = RESCALE * g.h(v) - (b[-1] * prev if b else 0)
            a.append(complex(_dots(v, w)[0]))
            w -= a[-1] * v
            b.append(float(torch.linalg.vector_norm(w)))
            prev, v = v, w / b[-1]
        e = np.array([0.5 * i * 2 * RESCALE / steps for i in range(-steps, steps + 1)])
        z, gr = e + 0.01j, 0.0
        for d in range(c["depth"] - 1, -1, -1):
            gr = 1.0 / (z - a[d] - b[d] ** 2 * gr)
        return e, -gr.imag / np.pi
    wf0 = g.states(seed, ns)
    if kind == "dos":
        return _dos_curve(g, wf0, steps)
    if kind in ("ac", "dynpol"):
        f, nf = _fermi_coef(False), _fermi_coef(True)
        p2 = g.series(f, wf0)
        if kind == "ac":
            p1 = [g.series(nf, g.j(d, wf0)) for d in (0, 1)]
            out = torch.zeros(4, steps, dtype=torch.complex128, device=g.dev)
        else:
            q = _q_points(c)
            wave = [torch.polar(torch.ones_like(g.pos[0]), k[0] * g.pos[0] + k[1] * g.pos[1])[:, None] for k in q]
            p1 = [g.series(nf, w.conj() * wf0) for w in wave]
            out = torch.zeros(len(q), steps, dtype=torch.float64, device=g.dev)
        for t in range(steps):
            if t:
                moved = g.step(math.pi / 2, torch.cat(p1 + [p2], 1))
                p1, p2 = list(moved.split(ns, 1)[:-1]), moved[:, -ns:]
            if kind == "dynpol":
                for k, w in enumerate(wave):
                    out[k, t] = _dots(p2, w * p1[k]).mean().imag
            elif t:
                for a in (0, 1):
                    for b in (0, 1):
                        out[2 * a + b, t] = _dots(p2, g.j(b, p1[a])).mean()
        return np.asfortranarray(_np(out))
    if kind == "kbdc":
        m = c["n_kernel"]
        k = np.arange(m)
        w = ((m - k) * np.cos(np.pi * k / m) + np.sin(np.pi * k / m) / np.tan(np.pi / m)) / m
        w[0] = 0.5
        mu = 0
        for s in range(ns):
            def chain(p, last):
                rows = [p, g.h(p)]
                for _ in range(2, m):
                    rows.append(2 * g.h(rows[-1]) - rows[-2])
                return torch.cat([last(x) for x in rows], 1)
            bra = chain(g.j(0, wf0[:, s:s + 1]), lambda x: x)
            ket = chain(wf0[:, s:s + 1], lambda x: g.j(0, x))
            mu = mu + _np(bra.conj().T @ ket) / ns
            del bra, ket
        return np.asfortranarray(mu * w[:, None] * w[None, :])
    # quasi-eigenstates, Hanning window
    e, sel = _energies(steps) if kind == "dc" else (_qe_energies(c), np.arange(c["n_en"]))
    en = torch.from_numpy(e[sel]).to(g.dev)
    qe = wf0[:, None, :].repeat(1, len(sel), 1)
    fw = bw = wf0
    dos = []
    for t in range(1, steps + 1):
        fw, bw = g.step(math.pi, fw), g.step(math.pi, bw, False)
        dos.append(_dots(wf0, fw).mean())
        w = torch.polar(torch.full_like(en, 0.5 * (1 + math.cos(math.pi * t / steps))), en * t * math.pi / RESCALE)
        qe += w[None, :, None] * fw[:, None, :]
        qe += w.conj()[None, :, None] * bw[:, None, :]
    if kind == "qe":
        dens = qe.abs() ** 2
        return np.asfortranarray(_np((dens / dens.sum(0)).mean(2)).T)
    amp = torch.einsum("rb,rib->ib", wf0.conj(), qe).abs()
    dc = torch.zeros(2, len(e), steps, dtype=torch.complex128, device=g.dev)
    for d in (0, 1):
        p = g.j(d, wf0)
        for t in range(steps):
            u = g.j(d, p)
            for b in range(ns):
                dc[d, :len(sel), t] += (u[:, b].conj() @ qe[:, :, b]) / amp[:, b] / ns
            p = g.step(math.pi, p)
    return _np(torch.stack(dos)), np.asfortranarray(_np(dc))
