"""The work that users of the framework have it do, as measurable cases.

A fit spends its time in NLL + gradient evaluations (``FCN.nll_grad``), so
most cases are single evaluations: in each precision form (plain FP64, the
default; the column cache of fixed lineshapes; the floating-shape cache; the
FP32 amplitudes of a polarised parent), for the shipped configurations and
from sample sizes where latency counts to the largest that the benchmark
holds.  The others are what surrounds a fit: its exact Hessian (the errors),
its set-up (MC Gram matrix and column cache), the kinematics of a new
dataset, and one round of the many-fit service.

Events are made here with torch from the seed alone: three-body phase space
(with the D*(2007) decaying on, in the four-body model), the data resampled
by sum |A|^2.  The same FP64 torch amplitude gives ``exact``'s values.
"""
import math
import os
from fractions import Fraction
from functools import lru_cache

import numpy as np
import torch

# The tuner picks the cached kernel's variant by timing, and the variants
# round FP32 sums in different orders: off, so that a run can be repeated.
os.environ.setdefault("PWA_AUTOTUNE", "0")

import __graft_entry__  # noqa: E402

__graft_entry__._pkg()
from tf_pwa_b200.api import ConfigLoader, EventData  # noqa: E402
from tf_pwa_b200.serving import FitJob, FitServer  # noqa: E402
from tf_pwa_b200.workload import config_path  # noqa: E402

DEV = "cuda"
CHUNK = 1 << 17          # events per step of the FP64 torch amplitude
BG_WEIGHT = 0.1          # background rows enter the NLL with weight -0.1
H = Fraction(1, 2)

# name: spin, parity, mass[, width] of every particle, the top one, the three
# bodies of its phase space, the chains (resonance, its daughters, bachelor;
# the top's first daughter in the configuration first), the decays that break
# parity, and the events' momenta in the configuration's order
_KPP = dict(
    particles=dict(A=(0, -1, 1.865), B=(0, -1, 0.4937), C=(0, -1, 0.1396), D=(0, -1, 0.1396),
                   R1=(1, -1, 0.892, 0.050), R2=(0, 1, 0.98, 0.10)),
    top="A", bodies=("B", "C", "D"), order=("B", "C", "D"), weak=(),
    chains=[("R1", ("B", "C"), ("R1", "D")), ("R2", ("C", "D"), ("R2", "B"))])
_LC = dict(
    particles=dict(Lc=(H, 1, 2.28646), p=(H, 1, 0.938272), K=(0, -1, 0.493677), pi=(0, -1, 0.13957),
                   L1520=(3 * H, -1, 1.5195, 0.016), Kstar=(1, -1, 0.8955, 0.047),
                   D1232=(3 * H, 1, 1.232, 0.117)),
    top="Lc", bodies=("p", "K", "pi"), order=("p", "K", "pi"), weak=("Lc",),
    chains=[("L1520", ("p", "K"), ("L1520", "pi")), ("Kstar", ("K", "pi"), ("Kstar", "p")),
            ("D1232", ("p", "pi"), ("D1232", "K"))])
_B4 = dict(
    particles=dict(B=(0, -1, 5.279), D=(0, -1, 1.865), pis=(0, -1, 0.135), K=(0, -1, 0.4937),
                   pi=(0, -1, 0.1396), Dst=(1, -1, 2.007),
                   RDstK0=(0, -1, 3.0945, 0.2481), RDstK1=(1, 1, 2.62, 0.1575),
                   RDstK2=(2, -1, 2.93, 0.0315), RDstK3=(3, 1, 2.71, 0.3717),
                   RDstpi0=(0, -1, 2.2891, 0.2756), RDstpi1=(1, 1, 2.2964, 0.1242),
                   RDstpi2=(2, -1, 2.25, 0.1119), RDstpi3=(3, 1, 2.8705, 0.2095),
                   RKpi0=(0, 1, 1.0808, 0.274), RKpi1=(1, -1, 1.2151, 0.3766),
                   RKpi2=(2, 1, 1.0835, 0.1569), RKpi3=(3, -1, 2.9826, 0.2302)),
    top="B", bodies=("Dst", "K", "pi"), order=("D", "pis", "K", "pi"),
    weak=("B",) + tuple(f"RDst{q}{j}" for q in ("K", "pi") for j in range(4)),
    chains=[(f"RDstK{j}", ("Dst", "K"), (f"RDstK{j}", "pi")) for j in range(4)]
    + [(f"RDstpi{j}", ("Dst", "pi"), (f"RDstpi{j}", "K")) for j in range(4)]
    + [(f"RKpi{j}", ("K", "pi"), ("Dst", f"RKpi{j}")) for j in range(4)])
MODELS = {"d2kpipi": _KPP, "d2kpipi_float": _KPP, "lc2pkpi": _LC, "lc2pkpi_float": _LC,
          "lc2pkpi_pol": _LC, "b2dstkpi": _B4}
# (column, helicity) pairs with a value, columns, helicity sums, masses and
# angles per event, forward operations per event
SIZES = {"d2kpipi": (2, 2, 1, 2, 8, 400), "lc2pkpi": (32, 8, 4, 3, 18, 1850),
         "b2dstkpi": (30, 30, 1, 4, 18, 7850)}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a first look at a Dalitz plot in the default form, the D -> K pi pi
        # sample size of the tests: launches and host work count
        dict(name="plain_kpipi_1e4", kind="fit", model="d2kpipi", precision="plain",
             n_data=10_000, n_bg=0, n_mc=100_000),
        # the benchmark's Lambda_c sample in the default (all-FP64) form
        dict(name="plain_lc_1e6", kind="fit", model="lc2pkpi", precision="plain",
             n_data=1_000_000, n_bg=100_000, n_mc=1_000_000),
        # a four-body fit in the default form: twelve resonances, ragged sizes
        dict(name="plain_4body", kind="fit", model="b2dstkpi", precision="plain",
             n_data=200_003, n_bg=0, n_mc=800_009),
        # a small fit with fixed lineshapes (the usual size of a real sample)
        dict(name="cached_lc_5e3", kind="fit", model="lc2pkpi", precision="mixed",
             n_data=5_011, n_bg=499, n_mc=100_003),
        # the benchmark's headline: Lambda_c with fixed lineshapes
        dict(name="cached_lc_1e6", kind="fit", model="lc2pkpi", precision="mixed",
             n_data=1_000_000, n_bg=100_000, n_mc=1_000_000),
        # the benchmark's four-body model with fixed lineshapes
        dict(name="cached_4body_1e6", kind="fit", model="b2dstkpi", precision="mixed",
             n_data=1_000_000, n_bg=0, n_mc=4_000_000),
        # masses and widths floating, the benchmark's D -> K pi pi sample
        dict(name="float_kpipi_1e6", kind="fit", model="d2kpipi_float", precision="mixed",
             n_data=1_000_000, n_bg=0, n_mc=1_000_000),
        # a polarised Lambda_c: the form that recomputes amplitudes in FP32
        dict(name="polarised_lc", kind="fit", model="lc2pkpi_pol", precision="mixed",
             n_data=100_000, n_bg=0, n_mc=500_001),
        # the errors of a fit: the exact Hessian in the couplings
        dict(name="hessian_lc", kind="hessian", model="lc2pkpi", precision="mixed",
             n_data=200_000, n_bg=20_000, n_mc=200_003),
        # a fit's set-up, again whenever a fixed mass or width is changed
        dict(name="setup_4body", kind="setup", model="b2dstkpi", precision="mixed",
             n_data=300_001, n_bg=0, n_mc=1_200_000),
        # a new dataset: momenta to masses and angles
        dict(name="kinematics_4body", kind="kinematics", model="b2dstkpi", precision="plain",
             n_data=1_000_003, n_bg=0, n_mc=0),
        # a toy study: one round of the fit service over many uneven fits
        dict(name="service_256_fits", kind="service", model="d2kpipi", precision="mixed",
             n_data=16_000_000, n_bg=0, n_mc=500_000, fits=256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind, model, precision, data, mc = rng.choice([
        ("fit", "d2kpipi", "plain", (2_000, 1_000_000), (20_000, 1_000_000)),
        ("fit", "lc2pkpi", "plain", (2_000, 1_100_000), (20_000, 1_000_000)),
        ("fit", "b2dstkpi", "plain", (2_000, 250_000), (20_000, 750_000)),
        ("fit", "lc2pkpi", "mixed", (2_000, 1_100_000), (20_000, 1_000_000)),
        ("fit", "b2dstkpi", "mixed", (2_000, 1_000_000), (20_000, 2_000_000)),
        ("fit", "d2kpipi_float", "mixed", (2_000, 1_000_000), (20_000, 1_000_000)),
        ("fit", "lc2pkpi_float", "mixed", (2_000, 1_100_000), (20_000, 1_000_000)),
        ("fit", "lc2pkpi_pol", "mixed", (2_000, 200_000), (20_000, 600_000)),
        ("hessian", "lc2pkpi", "mixed", (2_000, 1_100_000), (20_000, 200_000)),
        ("hessian", "b2dstkpi", "mixed", (2_000, 200_000), (20_000, 200_000)),
        ("setup", "lc2pkpi", "mixed", (2_000, 1_000_000), (20_000, 1_000_000)),
        ("setup", "b2dstkpi", "mixed", (2_000, 300_000), (20_000, 1_200_000)),
        ("kinematics", "d2kpipi", "plain", (2_000, 1_000_000), (0, 0)),
        ("kinematics", "b2dstkpi", "plain", (2_000, 1_000_000), (0, 0)),
        ("service", "d2kpipi", "mixed", (100_000, 16_000_000), (20_000, 500_000)),
    ])
    c = dict(kind=kind, model=model, precision=precision, n_data=_log(rng, *data), n_bg=0,
             n_mc=_log(rng, *mc) if mc[1] else 0)
    if model.startswith("lc2pkpi") and kind == "fit" and rng.random() < 0.5:
        c["n_bg"] = c["n_data"] // 11
        c["n_data"] -= c["n_bg"]
    if kind == "service":
        c["fits"] = _log(rng, 4, 256)
    return c


def work(case):
    m = case["model"].split("_")[0]
    nf, ncol, nout, nm, na, ops = SIZES[m]
    n, n_mc, kind = case["n_data"] + case["n_bg"], case["n_mc"], case["kind"]
    cached, fields = 8 * nf + 8, 8 * (nm + na + 1)
    gram = 4 * nout * ncol * (ncol + 1)      # the Hermitian half of a K x K product
    if kind == "kinematics":
        return {"bytes": (32 * len(MODELS[m]["order"]) + 8 * (nm + na)) * n, "flops": 1000 * n}
    if kind == "setup":
        return {"bytes": (fields + cached) * n + fields * n_mc, "flops": ops * (n + n_mc) + gram * n_mc}
    if kind == "hessian":
        return {"bytes": cached * n, "flops": (8 * nout * ncol * ncol + 8 * ncol * ncol) * n}
    if kind == "service" or case["precision"] == "mixed" and case["model"] in SIZES:
        return {"bytes": cached * n, "flops": 16 * nf * n}
    if case["model"].endswith("_float"):     # two points, each over data and MC
        return {"bytes": 2 * (cached + 8 * nm) * (n + n_mc), "flops": 2 * 32 * nf * (n + n_mc)}
    if case["model"].endswith("_pol"):       # FP32 angles
        return {"bytes": (8 * nm + 4 * na + 8) * (n + n_mc), "flops": 3 * ops * (n + n_mc)}
    return {"bytes": fields * (n + n_mc), "flops": 3 * ops * (n + n_mc)}  # values and adjoint


# ----------------------------------------------------------------- events
def _breakup(m0, m1, m2):
    s, d = m1 + m2, m1 - m2
    return ((m0 - s) * (m0 + s) * (m0 - d) * (m0 + d)).clamp(min=0).sqrt() / (2 * m0)


def _boost(p, frame):
    """p, given in frame's rest frame, in the frame that ``frame`` is given in."""
    m = (frame[:, :1] ** 2 - (frame[:, 1:] ** 2).sum(1, keepdim=True)).sqrt()
    dot = (p[:, 1:] * frame[:, 1:]).sum(1, keepdim=True)
    e = (frame[:, :1] * p[:, :1] + dot) / m
    return torch.cat([e, p[:, 1:] + frame[:, 1:] * (p[:, :1] + e) / (frame[:, :1] + m)], 1)


def _two_body(m0, m1, m2, gen):
    """Momenta of an isotropic two-body decay, in its rest frame."""
    n = m0.shape[0]
    z = torch.rand(n, generator=gen, dtype=torch.float64, device=DEV) * 2 - 1
    phi = torch.rand(n, generator=gen, dtype=torch.float64, device=DEV) * (2 * math.pi)
    q, s = _breakup(m0, m1, m2), (1 - z * z).sqrt()
    v = torch.stack([q * s * phi.cos(), q * s * phi.sin(), q * z], 1)
    e1, e2 = (q * q + m1 ** 2).sqrt(), (q * q + m2 ** 2).sqrt()
    return torch.cat([e1[:, None], v], 1), torch.cat([e2[:, None], -v], 1)


def _phase_space(model, n, gen):
    """(n, n_final, 4) momenta, flat in the phase space of the model's bodies."""
    pt = model["particles"]
    M, (m1, m2, m3) = pt[model["top"]][2], [pt[b][2] for b in model["bodies"]]
    got, have = [], 0
    while have < n:
        k = 2 * (n - have) + 1024
        m12 = m1 + m2 + (M - m3 - m1 - m2) * torch.rand(k, generator=gen, dtype=torch.float64,
                                                        device=DEV)
        top = torch.full_like(m12, M)
        w = _breakup(top, m12, torch.full_like(m12, m3)) * _breakup(m12, m1, m2)
        u = torch.rand(k, generator=gen, dtype=torch.float64, device=DEV)
        got.append(m12[u * w.max() < w])
        have += got[-1].shape[0]
    m12 = torch.cat(got)[:n]
    p12, p3 = _two_body(torch.full_like(m12, M), m12, m3, gen)
    p1, p2 = _two_body(m12, m1, m2, gen)
    p = dict(zip(model["bodies"], (_boost(p1, p12), _boost(p2, p12), p3)))
    if "Dst" in p:
        d, s = _two_body(torch.full_like(m12, pt["Dst"][2]), pt["D"][2], pt["pis"][2], gen)
        p["D"], p["pis"] = _boost(d, p["Dst"]), _boost(s, p["Dst"])
    return torch.stack([p[o] for o in model["order"]], 1)


def _fields(cl, model, n, gen):
    """Plan-ordered fields of n phase-space events (the package's torch code)."""
    return torch.cat([cl.data_from_p4(_phase_space(model, min(n - i, 1 << 20), gen)).fields
                      for i in range(0, n, 1 << 20)], 1)


def _data_fields(cl, model, vals, n, gen):
    """Events of the model: phase-space events resampled by sum |A|^2."""
    x = _fields(cl, model, 4 * n, gen)
    with torch.no_grad():
        f = torch.cat([_pdf(model, cl.plan.fields, x[:, i:i + CHUNK], vals)
                       for i in range(0, x.shape[1], CHUNK)])
    s = torch.cumsum(f, 0)
    u = (torch.arange(n, dtype=torch.float64, device=DEV)
         + torch.rand(n, generator=gen, dtype=torch.float64, device=DEV)) * (s[-1] / n)
    i = torch.searchsorted(s, u).clamp(max=x.shape[1] - 1)
    return x[:, i[torch.randperm(n, generator=gen, device=DEV)]].contiguous()


# ------------------------------------------------- amplitude, FP64 torch
def _spins(j):
    return [-j + k for k in range(int(2 * j) + 1)]


def _fact(x):
    return math.factorial(int(x))


@lru_cache(maxsize=None)
def _cg(j1, m1, j2, m2, j, m):
    """<j1 m1 j2 m2 | j m>, Racah's formula."""
    if m1 + m2 != m or not abs(j1 - j2) <= j <= j1 + j2 or abs(m) > j:
        return 0.0
    a = Fraction(int(2 * j + 1) * _fact(j1 + j2 - j) * _fact(j1 - j2 + j) * _fact(j2 - j1 + j),
                 _fact(j1 + j2 + j + 1))
    a *= _fact(j + m) * _fact(j - m) * _fact(j1 - m1) * _fact(j1 + m1) * _fact(j2 - m2) * _fact(j2 + m2)
    s = Fraction(0)
    for k in range(int(j1 + j2 + j) + 1):
        den = (k, j1 + j2 - j - k, j1 - m1 - k, j2 + m2 - k, j - j2 + m1 + k, j - j1 - m2 + k)
        if min(den) >= 0:
            s += Fraction((-1) ** k, math.prod(_fact(d) for d in den))
    return float(s) * math.sqrt(a)


def _ls(pt, a, b, c, weak):
    """(l, s) couplings of a -> b c, parity conserving unless weak."""
    (ja, pa), (jb, pb), (jc, pc) = (pt[q][:2] for q in (a, b, c))
    out = []
    for s in [abs(jb - jc) + k for k in range(int(jb + jc - abs(jb - jc)) + 1)]:
        for l in range(int(abs(ja - s)), int(ja + s) + 1):
            if weak or pa * pb * pc * (-1) ** l > 0:
                out.append((l, Fraction(s)))
    return sorted(out)


def _wigner_d(j, m1, m2, beta):
    """d^j_{m1 m2}(beta), Wigner's sum."""
    out = 0.0
    c, s = (beta / 2).cos(), (beta / 2).sin()
    root = math.sqrt(_fact(j + m1) * _fact(j - m1) * _fact(j + m2) * _fact(j - m2))
    for k in range(int(max(0, m2 - m1)), int(min(j + m2, j - m1)) + 1):
        den = _fact(j + m2 - k) * _fact(k) * _fact(m1 - m2 + k) * _fact(j - m1 - k)
        pw = int(m1 - m2) + 2 * k
        out = out + (-1) ** (int(m1 - m2) + k) * root / den * c ** int(2 * j - pw) * s ** pw
    return out


def _rot(j, m1, m2, alpha, beta, gamma=0.0):
    """conj(D^j_{m1 m2}(alpha, beta, gamma))."""
    phase = float(m1) * alpha + float(m2) * gamma
    return torch.polar(torch.ones_like(phase), phase) * _wigner_d(j, m1, m2, beta)


_BW = {0: [1], 1: [1, 1], 2: [1, 3, 9], 3: [1, 6, 45, 225], 4: [1, 10, 135, 1575, 11025]}


def _poly(l, z):
    r = 0.0 * z
    for c in _BW[l]:
        r = r * z + c
    return r


def _q2(m0, m1, m2):
    s, d = m1 + m2, m1 - m2
    return (m0 - s) * (m0 + s) * (m0 - d) * (m0 + d) / (2 * m0) ** 2


def _barrier(l, q2, q02, d=3.0):
    return q2 ** (l / 2) * (_poly(l, q02 * d * d) / _poly(l, q2 * d * d)).sqrt()


class _Chain:
    """Vertices (mother, first, second), field prefixes and LS lists of a chain."""

    def __init__(self, model, k):
        pt, (res, daughters, tops) = model["particles"], model["chains"][k]
        self.res, self.top = res, model["top"]
        inner = {res: set(daughters)}
        self.vertices = [(self.top,) + tops, (res,) + daughters]
        if "Dst" in model["bodies"]:
            inner["Dst"] = {"D", "pis"}
            self.vertices.insert(1 if "Dst" in tops else 2, ("Dst", "D", "pis"))
        finals = {q: set(s) for q, s in inner.items()}
        for q in finals:
            finals[q] = set().union(*[inner.get(f, {f}) for f in finals[q]])
        self.inner = list(inner)
        self.node = {q: "({})".format(", ".join(sorted(finals[q]))) if q in finals else q
                     for q in pt}
        self.tops, same = tops, {}
        for i, (r, ds, _) in enumerate(model["chains"]):
            same.setdefault(ds, i)
        self.topo = sorted(same.values()).index(same[daughters])
        self.ls = [_ls(pt, a, b, c, a in model["weak"]) for a, b, c in self.vertices]
        self.head = "".join(f"{a}->{b}.{c}" for a, b, c in self.vertices)


def _vertex_name(names, ch, v):
    """Field prefix <topology>/<decay> of vertex v."""
    a, b, c = (ch.node[q] for q in v)
    for second in (f"{b}+{c}", f"{c}+{b}"):
        if f"{ch.topo}/{a}->{second}/{b}/alpha" in names:
            return f"{ch.topo}/{a}->{second}"
    raise KeyError((ch.topo, v))


@lru_cache(maxsize=None)
def _chains_at(key):
    return [_Chain(MODELS[key], k) for k in range(len(MODELS[key]["chains"]))]


def _chains(model):
    return _chains_at(next(k for k, m in MODELS.items() if m is model))


def _columns(model, names, x, vals):
    """(N, K, parent helicities, final helicities): the amplitude at unit
    couplings, one column per chain and choice of LS couplings."""
    pt, at = model["particles"], {n: i for i, n in enumerate(names)}
    fin = [f for f in model["order"] if pt[f][0] != 0]
    one = torch.ones_like(x[0])
    cols = []
    for ch in _chains(model):
        mass = {q: x[at["m/" + ch.node[q]]] if q in ch.inner else pt[q][2] * one for q in pt}
        nominal = {q: one * vals.get(q + "_mass", pt[q][2]) for q in pt}
        vert = []
        for v, ls in zip(ch.vertices, ch.ls):
            a, b, c = v
            pre = _vertex_name(names, ch, v)
            al, be = (x[at[f"{pre}/{ch.node[b]}/{q}"]] for q in ("alpha", "beta"))
            q2, q02 = _q2(*(mass[q] for q in v)), _q2(*(nominal[q] for q in v))
            (ja, jb, jc), amp = (Fraction(pt[q][0]) for q in v), {}
            for l, s in ls:
                bf = _barrier(l, q2, q02)
                for la in _spins(ja):
                    for lb in _spins(jb):
                        for lc in _spins(jc):
                            g = math.sqrt((2 * l + 1) / float(2 * ja + 1)) * _cg(jb, lb, jc, -lc, s, lb - lc) \
                                * _cg(Fraction(l), Fraction(0), s, lb - lc, ja, lb - lc)
                            if g and abs(lb - lc) <= ja:
                                amp[(l, s), la, lb, lc] = g * bf * _rot(ja, la, lb - lc, al, be)
            vert.append((v, ls, amp))
        # the resonance's Breit-Wigner with its running width
        r, b, c = next(v for v in ch.vertices if v[0] == ch.res)
        L = min(l for l, _ in ch.ls[ch.vertices.index((r, b, c))])
        m, m0, g0 = mass[r], nominal[r], vals.get(r + "_width", pt[r][3])
        q, q0 = _q2(m, mass[b], mass[c]).clamp(min=0).sqrt(), _q2(m0, nominal[b], nominal[c]).clamp(min=0).sqrt()
        y = m0 * g0 * (q / q0) ** (2 * L + 1) * (m0 / m) * _poly(L, (3 * q0) ** 2) / _poly(L, (3 * q) ** 2)
        dx = m0 * m0 - m * m
        bw = torch.complex(dx, y) / (dx * dx + y * y)
        # turn of the spinning finals to their reference axes
        turn = {}
        for f in fin:
            pre = next((n[:-6] for n in names if n.startswith(f"{ch.topo}/")
                        and n.endswith(f"/{f}/aligned/alpha")), None)
            if pre:
                j = Fraction(pt[f][0])
                ang = [x[at[f"{pre}/{q}"]] for q in ("alpha", "beta", "gamma")]
                turn[f] = {(u, w): _rot(j, u, w, *ang) for u in _spins(j) for w in _spins(j)}
        combos = [()]
        for _, ls, _ in vert:
            combos = [k + (t,) for k in combos for t in ls]
        for combo in combos:
            out = {}
            terms = [({}, bw)]
            for (v, _, amp), t in zip(vert, combo):
                nxt = []
                for hel, val in terms:
                    for (tt, *ls3), z in amp.items():
                        if tt == t and all(hel.get(q, h) == h for q, h in zip(v, ls3)):
                            nxt.append(({**hel, **dict(zip(v, ls3))}, val * z))
                terms = nxt
            for hel, val in terms:
                key = (hel[ch.top],) + tuple(hel[f] for f in fin)
                out[key] = out.get(key, 0) + val
            rows = []
            for lt in _spins(Fraction(pt[ch.top][0])):
                fh = [()]
                for f in fin:
                    fh = [k + (h,) for k in fh for h in _spins(Fraction(pt[f][0]))]
                row = []
                for hs in fh:
                    if fin and fin[0] in turn:   # (at most one spinning final here)
                        z = sum(out[(lt, u)] * turn[fin[0]][u, hs[0]]
                                for u in _spins(Fraction(pt[fin[0]][0])) if (lt, u) in out)
                    else:
                        z = out.get((lt,) + hs, 0)
                    row.append(z + torch.zeros_like(bw))
                rows.append(torch.stack(row, -1))
            cols.append(torch.stack(rows, -2))
    return torch.stack(cols, 1)


def _couplings(model, vals):
    """Column couplings: chain total x one coupling per vertex, r e^{i phi}."""
    def z(name):
        r, p = (torch.as_tensor(vals[name + q], dtype=torch.float64, device=DEV) for q in "ri")
        return torch.complex(r * torch.cos(p), r * torch.sin(p))

    out = []
    for ch in _chains(model):
        cs = [z(ch.head + "_total_0")]
        for (a, b, c), ls in zip(ch.vertices, ch.ls):
            cs = [u * z(f"{a}->{b}.{c}_g_ls_{i}") for u in cs for i in range(len(ls))]
        out += cs
    return torch.stack(out)


def _intensity(model, F, c, vals):
    A = torch.einsum("nkab,k->nab", F, c)
    if "Lc_polarization_px" not in vals:
        return (A.real ** 2 + A.imag ** 2).sum((1, 2))
    px, py, pz = (torch.as_tensor(vals[f"Lc_polarization_p{q}"], dtype=torch.float64, device=DEV)
                  for q in "xyz")
    i = torch.complex(px, -py)
    rho = 0.5 * torch.stack([torch.stack([1 + pz + 0 * i, i]), torch.stack([i.conj(), 1 - pz + 0 * i])])
    return torch.einsum("nal,ab,nbl->n", A, rho, A.conj()).real


def _pdf(model, names, x, vals):
    return _intensity(model, _columns(model, names, x, vals), _couplings(model, vals), vals)


def _clip_log(f, eps=1e-6):
    d = (f - eps) / eps
    return torch.where(f > eps, f.clamp(min=eps).log(), math.log(eps) + d - d * d / 2)


# ------------------------------------------------------------ preparation
def _values(cl, seed):
    """A truth (couplings |g| in (0.5, 2), any phase; shapes near nominal)
    and the point of a fit on its way there."""
    rng = np.random.default_rng(seed)
    truth, point = {}, {}
    for k in cl.vm.trainable_vars:
        v = cl.vm.variables[k]
        if k.endswith("_mass"):
            truth[k], point[k] = v, v + 0.002 * rng.normal()
        elif k.endswith("_width"):
            truth[k], point[k] = v, v * (1 + 0.03 * rng.normal())
        elif "_polarization_" in k:
            truth[k] = rng.uniform(-0.5, 0.5)
            point[k] = truth[k] + 0.03 * rng.normal()
        else:
            truth[k] = rng.uniform(0.5, 2.0) if k.endswith("r") else rng.uniform(-math.pi, math.pi)
            point[k] = truth[k] + 0.05 * rng.normal()
    return truth, point


def _inputs(case, seed):
    """The loader with its parameters set, the points, and the events."""
    model = MODELS[case["model"]]
    cl = ConfigLoader(config_path(case["model"] + ".yml"), precision=case["precision"], seed=seed)
    truth, point = _values(cl, seed)
    cl.set_params(truth)
    gen = torch.Generator(device=DEV).manual_seed(seed)
    points = [np.array([point[k] for k in cl.vm.trainable_vars])]
    if case["model"].endswith("_float"):     # a minimiser moves the shapes at every call
        points.append(points[0] * (1 + 1e-3))
    vals = dict(cl.vm.variables)
    data = _data_fields(cl, model, vals, case["n_data"], gen)
    bg = _fields(cl, model, case["n_bg"], gen) if case["n_bg"] else None
    mc = _fields(cl, model, case["n_mc"], gen)
    return model, cl, points, data, bg, mc


def _service_inputs(case, seed):
    """Uneven fits (sizes over two decades), windows into one sample."""
    _, cl, points, data, _, mc = _inputs(dict(case, n_data=max(1000, case["n_data"] // 8)), seed)
    rng = np.random.default_rng(seed + 1)
    size = np.exp(rng.uniform(0, math.log(100), case["fits"]))
    size = np.maximum(1, size / size.sum() * case["n_data"]).astype(np.int64)
    size = np.minimum(size, data.shape[1])
    starts = [int(rng.integers(0, data.shape[1] - n + 1)) for n in size]
    xs = points[0] + 0.05 * rng.normal(size=(case["fits"], len(points[0])))
    return cl, [data[:, a:a + n] for a, n in zip(starts, size)], mc, xs


def _momenta(case, seed):
    return _phase_space(MODELS[case["model"]], case["n_data"],
                        torch.Generator(device=DEV).manual_seed(seed))


def prepare(case, seed):
    if case["kind"] == "kinematics":
        cl = ConfigLoader(config_path(case["model"] + ".yml"))
        cl.get_amplitude()._engine()
        return {"kind": case["kind"], "cl": cl, "p4": _momenta(case, seed),
                "w": np.ones(case["n_data"])}
    if case["kind"] == "service":
        cl, fits, mc, xs = _service_inputs(case, seed)
        tile_bytes = 128 * (8 * SIZES[case["model"]][0] + 8)
        tiles = sum(-(-f.shape[1] // 128) for f in fits)
        srv = FitServer(cl, EventData(mc), tiles * tile_bytes, max_active=len(fits), run=False)
        jobs = [srv.submit(FitJob(i, f, x)) for i, (f, x) in enumerate(zip(fits, xs))]
        srv._admit(start=False)
        V = np.repeat(srv.base_vars[None, :], len(fits), axis=0)
        V[:, srv.train_idx] = xs
        return {"kind": case["kind"], "srv": srv, "V": V, "first": [j.tiles[0] for j in jobs],
                "tiles": [j.tiles[1] for j in jobs], "sw": [float(j.n) for j in jobs]}
    model, cl, points, data, bg, mc = _inputs(case, seed)
    bg = None if bg is None else EventData(bg, -BG_WEIGHT * np.ones(bg.shape[1]))
    fcn = cl.get_fcn([EventData(data), EventData(mc), bg])
    fcn.nll_grad(points[0])                  # the initial NLL, as ``ConfigLoader.fit`` prints it
    return {"kind": case["kind"], "cl": cl, "fcn": fcn, "points": points}


def run(state):
    kind = state["kind"]
    if kind == "kinematics":
        return state["cl"].data_from_p4(state["p4"], state["w"], device=DEV).fields
    if kind == "service":
        return state["srv"].eng.pieces_multi(state["first"], state["tiles"], state["V"], state["sw"])
    fcn, points = state["fcn"], state["points"]
    if kind == "hessian":
        return fcn.nll_grad_hessian(points[0])
    if kind == "setup":
        vals = state["cl"].get_params()
        gram = fcn.eng.set_gram(vals)
        fcn.eng.cache_data(vals)
        return gram, fcn.nll_grad(points[0])
    return [fcn.nll_grad(x) for x in points]


# ------------------------------------------------------------------ exact
def _sums64(model, cl, x, fields, w, log):
    """Sum of w clip_log(f) (or w f) over the events, and its gradient."""
    train = list(cl.vm.trainable_vars)
    shapes = any(k.endswith(("_mass", "_width")) for k in train)
    th = torch.tensor(x, dtype=torch.float64, device=DEV, requires_grad=True)
    total = 0.0
    for i in range(0, fields.shape[1], CHUNK):
        vals = {**cl.vm.variables, **{k: th[j] for j, k in enumerate(train)}}
        with torch.set_grad_enabled(shapes):
            F = _columns(model, cl.plan.fields, fields[:, i:i + CHUNK], vals)
        f = _intensity(model, F, _couplings(model, vals), vals)
        s = (w[i:i + CHUNK] * (_clip_log(f) if log else f)).sum()
        s.backward()
        total += float(s.detach())
    return total, th.grad


def _nll_grad64(model, cl, x, data, w, mc):
    sd, gd = _sums64(model, cl, x, data, w, True)
    wm = torch.full((mc.shape[1],), 1.0 / mc.shape[1], dtype=torch.float64, device=DEV)
    sm, gm = _sums64(model, cl, x, mc, wm, False)
    sw = float(w.sum())
    return -sd + sw * math.log(sm), (-gd + sw * gm / sm).cpu().numpy()


def _gram64(model, names, mc, vals):
    M = 0
    with torch.no_grad():
        for i in range(0, mc.shape[1], CHUNK):
            F = _columns(model, names, mc[:, i:i + CHUNK], vals).flatten(2)
            F = F.transpose(1, 2).reshape(-1, F.shape[1])
            M = M + F.conj().T @ F / mc.shape[1]
    return M


def _hessian64(model, cl, x, data, w, mc):
    """NLL, gradient and Hessian in the couplings: sums in the column
    couplings u = (Re c, Im c), then the derivatives of u."""
    names, train = cl.plan.fields, list(cl.vm.trainable_vars)
    base = dict(cl.vm.variables)

    def u_of(th):
        c = _couplings(model, {**base, **{k: th[i] for i, k in enumerate(train)}})
        return torch.cat([c.real, c.imag])

    th = torch.tensor(x, dtype=torch.float64, device=DEV)
    u = u_of(th)
    K = u.shape[0] // 2
    c = torch.complex(u[:K], u[K:])

    def real2(Q):       # Hermitian form -> symmetric form in u, both doubled
        return 2 * torch.cat([torch.cat([Q.real, -Q.imag], 1), torch.cat([Q.imag, Q.real], 1)], 0)

    S, g, Hu = 0.0, 0.0, 0.0
    with torch.no_grad():
        for i in range(0, data.shape[1], CHUNK):
            F, ww = _columns(model, names, data[:, i:i + CHUNK], base).flatten(2), w[i:i + CHUNK]
            A = torch.einsum("nko,k->no", F, c)
            f = (A.abs() ** 2).sum(1)
            G = torch.einsum("no,nko->nk", A.conj(), F)
            gu = 2 * torch.cat([G.real, -G.imag], 1)
            lo = f <= 1e-6
            t1 = torch.where(lo, 1e6 - (f - 1e-6) * 1e12, 1 / f)
            t2 = torch.where(lo, torch.full_like(f, -1e12), -1 / f ** 2)
            S = S + (ww * _clip_log(f)).sum()
            g = g + (gu * (ww * t1)[:, None]).sum(0)
            Q = torch.einsum("nko,nlo,n->kl", F.conj(), F, (ww * t1).to(F.dtype))
            Hu = Hu + real2(Q) + gu.T @ (gu * (ww * t2)[:, None])
    M = _gram64(model, names, mc, base)
    Mu = real2(M)
    I, gI, sw = 0.5 * u @ Mu @ u, Mu @ u, w.sum()
    gu = -g + sw * gI / I
    Hu = -Hu + sw * (Mu / I - torch.outer(gI, gI) / I ** 2)
    J = torch.autograd.functional.jacobian(u_of, th)
    curl = torch.autograd.functional.hessian(lambda t: u_of(t) @ gu, th)
    nll = float(-S + sw * I.log())
    return nll, (J.T @ gu).cpu().numpy(), (J.T @ Hu @ J + curl).cpu().numpy()


def _service64(model, cl, fits, mc, xs):
    """Per fit: data sum, MC integral, weight, and the two sums' gradients."""
    train, rows = list(cl.vm.trainable_vars), []
    M = _gram64(model, cl.plan.fields, mc, dict(cl.vm.variables))
    for f, x in zip(fits, xs):
        n = f.shape[1]
        sd, gd = _sums64(model, cl, x, f, torch.ones(n, dtype=torch.float64, device=DEV), True)
        th = torch.tensor(x, dtype=torch.float64, device=DEV, requires_grad=True)
        c = _couplings(model, {**cl.vm.variables, **{k: th[i] for i, k in enumerate(train)}})
        integral = (c.conj() @ M @ c).real
        integral.backward()
        rows.append(np.concatenate([[sd, float(integral.detach()), n], gd.cpu().numpy(),
                                    th.grad.cpu().numpy()]))
    return np.stack(rows)


def _kinematics64(model, names, p4):
    """Masses and helicity angles: each daughter's direction in its mother's
    rest frame, the z axis along the mother, x in the plane of its decay."""
    mom = {o: p4[:, i] for i, o in enumerate(model["order"])}
    if "Dst" in model["bodies"]:
        mom["Dst"] = mom["D"] + mom["pis"]
    out = torch.empty((len(names), p4.shape[0]), dtype=torch.float64, device=p4.device)
    at = {n: i for i, n in enumerate(names)}

    def unit(v):
        return v / v.norm(dim=1, keepdim=True)

    def rest(p, frame):
        return _boost(p, torch.cat([frame[:, :1], -frame[:, 1:]], 1))

    axis = torch.eye(3, dtype=torch.float64, device=p4.device)
    for ch in _chains(model):
        _, b, c = next(v for v in ch.vertices if v[0] == ch.res)
        here = {**mom, ch.res: mom[b] + mom[c]}
        here[ch.top] = sum(mom[o] for o in model["order"])
        for q in ch.inner:
            m2 = here[q][:, 0] ** 2 - (here[q][:, 1:] ** 2).sum(1)
            out[at["m/" + ch.node[q]]] = m2.abs().sqrt()
        frame = {ch.top: ({q: rest(p, here[ch.top]) for q, p in here.items()},
                          axis[2].expand(p4.shape[0], 3), axis[0].expand(p4.shape[0], 3))}
        todo = list(ch.vertices)
        while todo:
            v = next(t for t in todo if t[0] in frame)
            todo.remove(v)
            a, b, c = v
            ps, z, x = frame[a]
            pre = _vertex_name(names, ch, v)
            first = b if pre.split("->")[1].startswith(ch.node[b] + "+") else c
            z = unit(z)
            y = unit(torch.linalg.cross(z, x))
            x = torch.linalg.cross(y, z)
            for d in (b, c):
                n = unit(ps[d][:, 1:])
                phi = torch.atan2((n * y).sum(1), (n * x).sum(1))
                cos = (n * z).sum(1)
                beta = torch.atan2((n - cos[:, None] * z).norm(dim=1), cos)
                lo = -math.pi if d == first else -2 * math.pi
                key = f"{pre}/{ch.node[d]}/alpha"
                if key in at:
                    out[at[key]] = torch.remainder(phi - lo, 2 * math.pi) + lo
                    out[at[f"{pre}/{ch.node[d]}/beta"]] = beta
                side = torch.linalg.cross(torch.linalg.cross(z, n), n)
                frame[d] = ({q: rest(p, ps[d]) for q, p in ps.items() if q != d}, n, side)
    return out


def exact(case, seed):
    if case["kind"] == "kinematics":
        names = ConfigLoader(config_path(case["model"] + ".yml")).plan.fields
        return _kinematics64(MODELS[case["model"]], names, _momenta(case, seed))
    if case["kind"] == "service":
        cl, fits, mc, xs = _service_inputs(case, seed)
        return _service64(MODELS[case["model"]], cl, fits, mc, xs)
    model, cl, points, data, bg, mc = _inputs(case, seed)
    w = torch.ones(data.shape[1], dtype=torch.float64, device=DEV)
    if bg is not None:
        data = torch.cat([data, bg], 1)
        w = torch.cat([w, torch.full((bg.shape[1],), -BG_WEIGHT, dtype=torch.float64, device=DEV)])
    w = w * (w.sum() / (w * w).sum())
    if case["kind"] == "hessian":
        return _hessian64(model, cl, points[0], data, w, mc)
    out = [_nll_grad64(model, cl, x, data, w, mc)[:2] for x in points]
    if case["kind"] == "setup":
        return _gram64(model, cl.plan.fields, mc, dict(cl.vm.variables)).cpu().numpy(), out[0]
    return out
