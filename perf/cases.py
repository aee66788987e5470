"""Performance cases of the force-evaluation path, each through an entry point that a program
of the framework's user calls.

A case is one configuration of seeded water boxes (the package's own generator, densities
around 1 g/cm^3) and one call:

  hot       Context.hot_path (host arrays, as the reference's Fortran caller has them) or
            Context.hot_path_device (resident arrays): the whole force evaluation of a step
  three     Context.threebody_term: FS2 + FS3 from host arrays
  induction Context.nb_induction: the dipole solve and its forces from host arrays
  kspace    kspace_ewald_fixed: reciprocal Ewald sum on resident arrays, no allocation
  train     three_body_induction_energy forward and backward, with the gradients of the
            positions and of the FS3 parameters (fitting the potential)
  batch     Batch.terms_device: independent frames in one call
  md        Context.md_set_state, md_nve, md_get_state: a few whole MD steps

``exact`` restates the terms' energies in plain torch FP64 and takes every force from them by
automatic differentiation; the induced dipoles come from a dense linear solve.
"""
from __future__ import annotations

import functools
import itertools
import math

import numpy as np
import torch

from ccpol23_plus_2025_mbmd_b200 import Batch, Context, Model, _lib, data_dir
from ccpol23_plus_2025_mbmd_b200.api import kspace_ewald_fixed
from ccpol23_plus_2025_mbmd_b200.autograd import fs3_param_tensors, three_body_induction_energy
from ccpol23_plus_2025_mbmd_b200.generator import water_box

THREE_IND = _lib.TERM_INDUCTION | _lib.TERM_FS2 | _lib.TERM_FS3
SITES_PER_MOL = 28
LD_REFERENCE = 50  # the reference's Fortran leading dimension


def _case(kind, nm, variant="fs2fs3", precision="fp64", host=False, ld=SITES_PER_MOL, frames=1,
          steps=0, density=1.0):
    # 29.93 A^3 per molecule: liquid water, the density of the benchmark boxes
    return {"kind": kind, "nm": nm, "box": round((29.93 * nm / density) ** (1.0 / 3.0), 4),
            "variant": variant, "precision": precision, "host": host, "ld": ld,
            "frames": frames, "steps": steps}


def listed():
    def named(name, *a, **k):
        return {"name": name, **_case(*a, **k)}
    return [
        # the smallest boxes a test or a debugging run uses: latency and launches
        named("hot_37_host", "hot", 37, host=True, ld=LD_REFERENCE),
        # a small FS3-only box called from the reference's host arrays
        named("hot_128_fs3_host", "hot", 128, variant="fs3", host=True, ld=LD_REFERENCE),
        # the benchmark box: one force evaluation of an MD step, state on the device
        named("hot_512", "hot", 512),
        # the same in the mixed-precision form
        named("hot_512_mixed", "hot", 512, precision="mixed"),
        # a ragged larger box in the mixed form
        named("hot_1003_mixed", "hot", 1003, precision="mixed"),
        # the large benchmark box
        named("hot_2048", "hot", 2048),
        # single reference entry points from host arrays, ragged sizes
        named("three_333_host", "three", 333, host=True, ld=LD_REFERENCE),
        named("induction_700_host", "induction", 700, host=True, ld=LD_REFERENCE),
        # the reciprocal sum alone, on resident arrays: the smallest call there is
        named("kspace_216", "kspace", 216),
        # one fitting step: energy, position and parameter gradients
        named("train_256", "train", 256, variant="fs3"),
        # independent frames in one call
        named("batch_16x256", "batch", 256, variant="fs3", frames=16),
        # whole MD steps (2-body term, force evaluation, integrator)
        named("md_512", "md", 512, steps=4),
    ]


def draw(rng):
    kind = rng.choice(["hot", "hot", "hot", "hot", "three", "induction", "kspace", "train",
                       "batch", "md"])
    top = {"hot": 1800, "three": 1400, "induction": 1400, "kspace": 1800, "train": 512,
           "batch": 300, "md": 640}[kind]
    nm = int(round(math.exp(rng.uniform(math.log(30.0), math.log(top)))))
    host = kind in ("three", "induction") or (kind == "hot" and rng.random() < 0.4)
    return _case(kind, nm, variant=rng.choice(["fs2fs3", "fs2fs3", "fs3"]),
                 precision="mixed" if kind in ("hot", "md") and rng.random() < 0.4 else "fp64",
                 host=host, ld=rng.choice([28, 31, LD_REFERENCE]) if kind in
                 ("hot", "three", "induction", "kspace") else SITES_PER_MOL,
                 frames=rng.randint(2, 16) if kind == "batch" else 1,
                 steps=rng.randint(1, 4) if kind == "md" else 0,
                 density=round(rng.uniform(0.95, 1.03), 3))


# ------------------------------------------------------------------------------- inputs
@functools.lru_cache(maxsize=None)
def _model(variant):
    return Model(data_dir(variant))


def _water(case, seed):
    model = _model(case["variant"])
    for k in range(20):  # a crowded random draw is redrawn
        try:
            return water_box(model, case["nm"], case["box"], 1000003 * seed + k, ld=case["ld"])
        except RuntimeError:
            continue
    raise RuntimeError("no box could be placed")


def _boxes(case, seed):
    return [_water(case, 64 * seed + f) for f in range(case["frames"])]


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a), device="cuda")


def prepare(case, seed):
    model = _model(case["variant"])
    boxes = _boxes(case, seed)
    b, kind, nm, L = boxes[0], case["kind"], case["nm"], case["box"]
    s = {"case": case, "model": model, "box": b}
    if kind == "batch":
        s["in"] = [_dev(np.stack([getattr(q, k) for q in boxes]))
                   for k in ("x", "y", "z", "xs", "ys", "zs")]
        x, xs = s["in"][0], s["in"][3]
        s["f"] = [torch.zeros_like(xs) for _ in range(3)]
        s["c"] = [torch.zeros_like(x) for _ in range(6)]
        s["mu"] = [torch.zeros_like(xs) for _ in range(3)]
        s["batch"] = Batch(model, nm, L, slots=8, precision=case["precision"])
        return s
    if kind != "kspace":
        s["ctx"] = Context(model, nm, L, precision=case["precision"])
    if kind == "train":
        s["com"] = _dev(np.stack([b.x, b.y, b.z], axis=-1)).requires_grad_()
        s["sites"] = _dev(np.stack([b.xs, b.ys, b.zs], axis=-1)).requires_grad_()
        s["par"] = fs3_param_tensors(s["ctx"], "cuda")
    elif not case["host"] and kind != "md":
        s["in"] = [_dev(a) for a in (b.x, b.y, b.z, b.xs, b.ys, b.zs)]
        x, xs = s["in"][0], s["in"][3]
        s["f"] = [torch.zeros_like(xs) for _ in range(3)]
        s["c"] = [torch.zeros_like(x) for _ in range(6)]
        s["mu"] = [torch.zeros_like(xs) for _ in range(3)]
        s["one"] = [torch.zeros(1, dtype=torch.float64, device="cuda") for _ in range(2)]
        s["alpha"], s["kmax"] = _ewald(L)
        if kind == "hot":  # queue on the program's stream, which also clears the forces
            s["ctx"].set_stream(torch.cuda.current_stream().cuda_stream or 1)
    return s


ENERGIES = ("scpe", "rcpe", "kcpe", "indpe", "fs2pe", "fs3pe", "vir")
COUNTS = ("ind_iters", "n_fs3_triples", "n_fs3_blend", "n_fs2_triples")


def _sorted(e):
    return {"energies": {k: e[k] for k in ENERGIES}, "counts": {k: e[k] for k in COUNTS}}


# ----------------------------------------------------------------------------- one pass
def run(s):
    case, b = s["case"], s["box"]
    kind, L, nm, ld = case["kind"], case["box"], case["nm"], case["ld"]
    pos = (b.x, b.y, b.z, b.xs, b.ys, b.zs)
    if kind == "hot" and case["host"]:
        r = s["ctx"].hot_path(*pos, L)
        return {**_sorted(r.energies), "f": [r.fxs, r.fys, r.fzs],
                "c2": [r.fxfs2, r.fyfs2, r.fzfs2], "c3": [r.fxfs3, r.fyfs3, r.fzfs3],
                "mu": [r.idmx, r.idmy, r.idmz]}
    if kind == "hot":
        for t in s["f"]:  # site forces accumulate
            t.zero_()
        e = s["ctx"].hot_path_device(*s["in"], L, *s["f"], *s["c"], *s["mu"])
        return {**_sorted(e), "f": s["f"], "c2": s["c"][:3], "c3": s["c"][3:], "mu": s["mu"]}
    if kind == "three":
        f = [np.zeros((nm, ld)) for _ in range(3)]
        c = [np.zeros(nm) for _ in range(6)]
        vir = np.zeros(1)
        e2, e3 = s["ctx"].threebody_term(*pos, L, *f, *c, vir)
        return {"fs2pe": e2, "fs3pe": e3, "vir": vir, "f": f, "c2": c[:3], "c3": c[3:]}
    if kind == "induction":
        mu = [np.zeros((nm, ld)) for _ in range(3)]
        f = [np.zeros((nm, ld)) for _ in range(3)]
        vir = np.zeros(1)
        e, it = s["ctx"].nb_induction(*pos, L, *mu, *f, vir)
        return {"indpe": e, "ind_iters": it, "vir": vir, "f": f, "mu": mu}
    if kind == "kspace":
        q, vir = s["one"]
        for t in s["f"]:
            t.zero_()
        vir.zero_()
        k = s["kmax"]
        kspace_ewald_fixed(s["model"], *s["in"], k, k, k, s["alpha"], L, q, *s["f"], vir,
                           torch.cuda.current_stream().cuda_stream or None)
        return {"kcpe": q, "vir": vir, "f": s["f"]}
    if kind == "train":
        leaves = [s["com"], s["sites"], *s["par"]]
        e = three_body_induction_energy(s["ctx"], L, *leaves)
        return {"energy": e.detach(), "grad": list(torch.autograd.grad(e, leaves))}
    if kind == "batch":
        for t in s["f"]:
            t.zero_()
        # the batch's slots run on their own streams: what was queued here comes first
        torch.cuda.current_stream().synchronize()
        es = s["batch"].terms_device(THREE_IND, L, *s["in"], *s["f"], *s["c"], *s["mu"])
        return {"energies": np.array([[e[k] for k in ("indpe", "fs2pe", "fs3pe")] for e in es]),
                "vir": np.array([e["vir"] for e in es]),
                "counts": np.array([[e[k] for k in COUNTS] for e in es]),
                "f": s["f"], "c2": s["c"][:3], "c3": s["c"][3:], "mu": s["mu"]}
    s["ctx"].md_set_state(L, b.x, b.y, b.z, b.v, b.q, b.jb)
    st = s["ctx"].md_nve(case["steps"], 0.0005)
    return {"state": s["ctx"].md_get_state(), "last": st[-1]}


# --------------------------------------------------------------------------------- work
def work(case):
    """Bytes of the inputs and results, and the arithmetic of the terms' sums: site pairs
    within the cut-offs, (k-vector, site) pairs and FS3's site-pair contractions."""
    nm, L = case["nm"], case["box"]
    rho = nm / L ** 3
    near = lambda r: min(nm - 1.0, rho * 4.0 / 3.0 * math.pi * r ** 3)  # noqa: E731
    _, kmax = _ewald(L)
    nk = 2.0 / 3.0 * math.pi * kmax ** 3
    kspace = nk * 5 * nm * 2 * 10
    pairs = 0.5 * nm * near(9.0)
    induction = pairs * 64 * 120 + 2 * kspace + 28 * (pairs * 18 * 15 + nk * 3 * nm * 16)
    # per FS3 triple: three contractions of 17 x 17 x 17 products in four power combinations
    fs3 = 1.25 * nm * near(6.3) ** 2 / 20.0 * 3 * 17 ** 3 * 4 * 2
    fs2 = 0.25 * nm * near(7.5) ** 2 * 45 * 60 if case["variant"] == "fs2fs3" else 0.0
    ewald = pairs * 25 * 40 + kspace
    vdw = pairs * 625 * 60
    flops = {"hot": ewald + induction + fs2 + fs3, "three": fs2 + fs3, "induction": induction,
             "kspace": kspace, "train": 1.3 * fs3 + fs2 + induction,
             "batch": induction + fs2 + fs3,
             "md": (case["steps"] + 1) * (ewald + induction + fs2 + fs3 + vdw)}[case["kind"]]
    doubles = {"kspace": 3 + 3 * 28 + 3 * 28, "md": 2 * 16}.get(
        case["kind"], 3 + 3 * 28 + 3 * 28 + 6 + 3 * 28)
    return {"bytes": 8 * doubles * nm * case["frames"], "flops": flops * case["frames"]}


# -------------------------------------------------------- the terms in plain torch, FP64
PI = math.pi
R4 = 138935.4835        # 1/(4 pi eps0), 10 J/mol A / e^2
BOHR = 0.529177249
H2KCAL = 627.510
KCAL = 418.4            # internal units (10 J/mol) per kcal/mol
RCUT = 9.0
FS3_TYPE = [0, 1, 1, 2, 2, 3, 3, 3, 3, 4, 4, 4, 4, 5, 5, 5, 5]


def _ewald(L):
    """alpha and k-max of the default precision 1e-6 at the 9 A cut-off."""
    e = 1.0e-6 * RCUT
    tol = math.sqrt(abs(math.log(e)))
    a = math.sqrt(abs(math.log(e * tol))) / RCUT
    tol1 = math.sqrt(-math.log(e * (2.0 * tol * a) ** 2))
    return a, int(math.floor(0.25 + L * a * tol1 / PI + 0.5))


@functools.lru_cache(maxsize=None)
def _fit(variant):
    """The model's numbers, read from its input files."""
    d = data_dir(variant)
    with open(d / "FIELD") as f:
        rows = [ln.split() for ln in f]
    with open(d / "CONTROL") as f:
        ctl = [ln.split() for ln in f]
    ns, npol = int(rows[2][0]), int(rows[3][0])
    site = rows[5:5 + ns]
    p = {"ns": ns, "npol": npol, "q": np.array([float(t[5]) for t in site]),
         "pol": np.array([float(t[6]) for t in site]),
         "fs2": ctl[13][2].startswith("T"), "rc3": float(ctl[14][0]),
         "alpha3": float(ctl[14][1]), "delta33": float(ctl[14][3])}
    for tag, name in (("sr", "data3b_full"), ("lr", "data3b_full_LR_4p5")):
        with open(d / name) as f:
            t = [ln.split() for ln in f]
        p["bgr_" + tag] = np.array([[float(v) for v in r[:3]] for r in t[1:290]]).T.copy()
        n = int(t[291][0])
        p["cs_" + tag] = np.array([float(r[1]) for r in t[292:292 + n]])
    # coefficient classes: (type, power) triples up to a common permutation, numbered in the
    # order in which the site loops meet them
    cls, index = {}, np.zeros((17, 17, 17, 2, 2, 2), dtype=np.int64)
    for i, j, k in itertools.product(range(17), repeat=3):
        for a, b, c in itertools.product(range(2), repeat=3):
            key = tuple(sorted([(FS3_TYPE[i], a), (FS3_TYPE[j], b), (FS3_TYPE[k], c)]))
            index[i, j, k, a, b, c] = cls.setdefault(key, len(cls))
    p["index"] = index
    return p


def _image(d, L):
    """The whole boxes that the minimum image of the differences d takes off."""
    return torch.sign(d) * torch.floor(torch.abs(d / L) + 0.5)


class _Box:
    """One box as leaves (site positions P, centres C) and the neighbour pairs of C."""

    def __init__(self, b, L, ns, dev):
        t = lambda *a: torch.tensor(np.stack(a, axis=-1), dtype=torch.float64, device=dev)  # noqa: E731
        self.L, self.dev, self.nm = L, dev, len(b.x)
        self.C = t(b.x, b.y, b.z).requires_grad_()
        off = t(b.xs[:, :ns], b.ys[:, :ns], b.zs[:, :ns])
        self.P = (self.C.detach()[:, None, :] + off).requires_grad_()
        self.scale = torch.ones((), dtype=torch.float64, device=dev).requires_grad_()

    def c(self):
        return self.C * self.scale

    def p(self):
        return self.P * self.scale

    def pairs(self, rc):
        """(i, j, whole boxes) of the pairs i < j closer than rc."""
        found, C = [], self.C.detach()
        for i0 in range(0, self.nm, 512):
            d = C[i0:i0 + 512, None, :] - C[None, :, :]
            n = _image(d, self.L)
            r2 = ((d - self.L * n) ** 2).sum(-1)
            i, j = torch.nonzero(r2 < rc * rc, as_tuple=True)
            keep = i + i0 < j
            i, j = i[keep], j[keep]
            found.append((i + i0, j, n[i, j]))
        return [torch.cat(v) for v in zip(*found)]

    def backward(self, e, ones=()):
        leaves = [self.P, self.C, self.scale, *ones]
        g = torch.autograd.grad(e, leaves, allow_unused=True)
        return [torch.zeros_like(x) if v is None else v for x, v in zip(leaves, g)]


def _self_energy(B, q, alpha):
    n = q.numel()
    i, j = torch.triu_indices(n, n, 1, device=B.dev)
    keep = q[i] * q[j] != 0
    i, j = i[keep], j[keep]
    P = B.p()
    r = torch.linalg.norm(P[:, i] - P[:, j], dim=-1)
    e = -alpha * B.nm * (q * q).sum() / math.sqrt(PI)
    return R4 * (e - (torch.erf(alpha * r) * q[i] * q[j] / r).sum())


def _real_energy(B, q, alpha, near):
    s = torch.nonzero(q)[:, 0]
    i, j, n = near
    P = B.p()[:, s]
    d = P[i][:, :, None] - P[j][:, None, :] - (B.L * B.scale) * n[:, None, None, :]
    r = torch.linalg.norm(d, dim=-1)
    return R4 * (q[s][:, None] * q[s][None, :] * torch.erfc(alpha * r) / r).sum()


def _kvectors(L, kmax, dev):
    r = torch.arange(-kmax, kmax + 1, dtype=torch.float64, device=dev)
    k = torch.cartesian_prod(r, r, r)
    k = k[((k * k).sum(-1) <= kmax * kmax) & ((k * k).sum(-1) > 0)]
    half = (k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0))))
    return k[half]


def _phases(B, site, k):
    """k . r of the sites (n, 3), scale-free because k scales inversely."""
    return (2.0 * PI / B.L) * (site @ k.T)


def _kspace_energy(B, q, alpha, kmax, mu=None, only_dipoles=False):
    """Reciprocal energy of the charges, or of charges and dipoles with the charge-charge
    part left out."""
    s = torch.nonzero(q)[:, 0]
    Lv = B.L * B.scale
    parts = []
    k_all = _kvectors(B.L, kmax, B.dev)
    for k0 in range(0, k_all.shape[0], 1024):
        k = k_all[k0:k0 + 1024]
        kk = 2.0 * PI / Lv * k
        k2 = (kk * kk).sum(-1)
        ak = 2.0 * PI / Lv ** 3 * torch.exp(-0.25 * k2 / alpha ** 2) / k2
        ph = _phases(B, B.P[:, s].reshape(-1, 3), k)
        qs = q[s].repeat(B.nm)
        qc, qn = qs @ torch.cos(ph), qs @ torch.sin(ph)
        if mu is None:
            parts.append((ak * (qc ** 2 + qn ** 2)).sum())
            continue
        pm = _phases(B, B.P[:, -mu.shape[1]:].reshape(-1, 3), k)
        dk = mu.reshape(-1, 3) @ kk.T
        # exp(i k.(r + mu)) to first order: dipoles add i (k.mu) exp(i k.r)
        dc, dn = (dk * torch.cos(pm)).sum(0), (dk * torch.sin(pm)).sum(0)
        parts.append((ak * (2.0 * (qn * dc - qc * dn) + dc ** 2 + dn ** 2)).sum())
    return 2.0 * R4 * torch.stack(parts).sum()


def _tt(n, x):
    t, s = torch.ones_like(x), torch.ones_like(x)
    for k in range(1, n + 1):
        t = t * x / k
        s = s + t
    return 1.0 - torch.exp(-x) * s


def _damped(r, alpha, erf_part):
    """The Ewald radial factors of 1/r^3 and 1/r^5: of erfc, or with erf_part of erf."""
    g = 2.0 / math.sqrt(PI) * alpha * torch.exp(-(alpha * r) ** 2) / r ** 2
    h = g / r ** 2 + 2.0 / 3.0 * alpha ** 2 * g
    if erf_part:
        ef = torch.erf(alpha * r)
        return ef / r ** 3 - g, ef / r ** 5 - h
    ec = torch.erfc(alpha * r)
    return ec / r ** 3 + g, ec / r ** 5 + h


def _dipole_parts(B, q, alpha, near, npol):
    """Blocks of the real-space and intramolecular dipole energy: lists of (site rows, site
    columns, field coefficient vectors or tensors).  Charges first, dipoles second."""
    P = B.p()
    s = torch.nonzero(q)[:, 0]
    i, j, n = near
    shift = (B.L * B.scale) * n[:, None, None, :]
    Q, D = P[:, s], P[:, -npol:]

    def field(d, sign, erf_part, damp):
        r = torch.linalg.norm(d, dim=-1)
        b3, _ = _damped(r, alpha, erf_part)
        if damp:
            b3 = b3 + (_tt(2, 1.65 / BOHR * r) - 1.0) / r ** 3
        return sign * b3[..., None] * d

    def tensor(d, sign, erf_part, damp):
        r = torch.linalg.norm(d, dim=-1)
        b3, b5 = _damped(r, alpha, erf_part)
        if damp:
            f3 = _tt(3, 1.55 / BOHR * r) - 1.0
            b3, b5 = b3 + f3 / r ** 3, b5 + f3 / r ** 5
        eye = torch.eye(3, dtype=torch.float64, device=B.dev)
        return sign * (3.0 * b5[..., None, None] * d[..., :, None] * d[..., None, :]
                       - b3[..., None, None] * eye)

    # field at the dipoles of i from the charges of j and the other way round
    e_ij = field(D[i][:, :, None] - Q[j][:, None, :] - shift, 1.0, False, True)
    e_ji = field(D[j][:, :, None] - Q[i][:, None, :] + shift, 1.0, False, True)
    t_ij = tensor(D[i][:, :, None] - D[j][:, None, :] - shift, 1.0, False, True)
    # intramolecular: what the reciprocal sum has too much; coincident sites are left out
    a, c = torch.meshgrid(torch.arange(npol, device=B.dev), torch.arange(len(s), device=B.dev),
                          indexing="ij")
    apart = torch.linalg.norm(B.P.detach()[0, -npol:][:, None] - B.P.detach()[0, s][None], dim=-1) > 1e-9
    a, c = a[apart], c[apart]
    e_in = field(D[:, a] - Q[:, c], -1.0, True, False)
    u, v = torch.triu_indices(npol, npol, 1, device=B.dev)
    t_in = tensor(D[:, u] - D[:, v], -1.0, True, False)
    return (s, i, j, e_ij, e_ji, t_ij), (a, c, e_in, u, v, t_in)


def _induction_energy(B, q, pol, alpha, kmax, near, npol, mu):
    """Energy of fixed dipoles mu (nm, npol, 3): polarisation, charge-dipole, dipole-dipole."""
    (s, i, j, e_ij, e_ji, t_ij), (a, c, e_in, u, v, t_in) = _dipole_parts(B, q, alpha, near, npol)
    qs = q[s]
    e = (mu ** 2 / (2.0 * pol[:, None])).sum()
    e = e - torch.einsum("pad,pacd,c->", mu[i], e_ij, qs) - torch.einsum("pad,pacd,c->", mu[j], e_ji, qs)
    e = e - torch.einsum("pax,pabxy,pby->", mu[i], t_ij, mu[j])
    e = e - (mu[:, a] * e_in * qs[c][None, :, None]).sum()
    e = e - torch.einsum("mnx,mnxy,mny->", mu[:, u], t_in, mu[:, v])
    e = e - 0.5 * 4.0 * alpha ** 3 / (3.0 * math.sqrt(PI)) * (mu ** 2).sum()
    return R4 * e + _kspace_energy(B, q, alpha, kmax, mu)


def _dipoles(B, q, pol, alpha, kmax, near, npol):
    """The converged dipoles: A mu = E0 solved densely, A and E0 read off the energy."""
    nm, n3 = B.nm, B.nm * npol * 3
    with torch.no_grad():
        (s, i, j, e_ij, e_ji, t_ij), (a, c, e_in, u, v, t_in) = _dipole_parts(B, q, alpha, near, npol)
        qs = q[s]
        E0 = torch.zeros((nm, npol, 3), dtype=torch.float64, device=B.dev)
        E0.index_add_(0, i, torch.einsum("pacd,c->pad", e_ij, qs))
        E0.index_add_(0, j, torch.einsum("pacd,c->pad", e_ji, qs))
        E0.index_add_(1, a, e_in * qs[c][None, :, None])
        A = torch.zeros((nm, npol, 3, nm, npol, 3), dtype=torch.float64, device=B.dev)
        for x in range(npol):
            for y in range(npol):
                A[i, x, :, j, y, :] = -t_ij[:, x, y]
                A[j, y, :, i, x, :] = -t_ij[:, x, y].transpose(1, 2)
        m = torch.arange(nm, device=B.dev)
        for k, (x, y) in enumerate(zip(u.tolist(), v.tolist())):
            A[m, x, :, m, y, :] = -t_in[:, k]
            A[m, y, :, m, x, :] = -t_in[:, k].transpose(1, 2)
        A = A.view(n3, n3)
        ident = 1.0 / pol - 4.0 * alpha ** 3 / (3.0 * math.sqrt(PI))
        A.diagonal().add_(ident.repeat(nm).repeat_interleave(3))
        k_all = _kvectors(B.L, kmax, B.dev)
        for k0 in range(0, k_all.shape[0], 1024):
            k = k_all[k0:k0 + 1024]
            kk = 2.0 * PI / B.L * k
            k2 = (kk * kk).sum(-1)
            ak = 4.0 * 2.0 * PI / B.L ** 3 * torch.exp(-0.25 * k2 / alpha ** 2) / k2
            ph = _phases(B, B.P[:, s].reshape(-1, 3), k)
            rep = qs.repeat(nm)
            qc, qn = rep @ torch.cos(ph), rep @ torch.sin(ph)
            pm = _phases(B, B.P[:, -npol:].reshape(-1, 3), k)
            co, si = torch.cos(pm), torch.sin(pm)
            E0 += ((ak * (si * qc - co * qn)) @ kk).view(nm, npol, 3)
            for f in (co, si):
                w = (f[:, None, :] * kk.T[None] * torch.sqrt(ak)).reshape(n3, -1)
                A.addmm_(w, w.T)
        mu = torch.linalg.solve(A, E0.reshape(n3, 1)).view(nm, npol, 3)
        return mu, R4 * -0.5 * (mu * E0).sum()


FS2_CHARGE = [0.258504607653328389, 0.564050362569283648, 0.564050362569283648,
              -0.693302666395947953, -0.693302666395947953]


def _triples(B, rc, first):
    """Molecular triples with all three centres within rc, by chunks: FS2's (k; i < j) with
    the pair (i, j) first, or FS3's i < j < k."""
    i, j, _ = B.pairs(rc)
    C, L = B.C.detach(), B.L
    for p0 in range(0, i.numel(), max(1, 4_000_000 // B.nm)):
        a, b = i[p0:p0 + 4_000_000 // B.nm], j[p0:p0 + 4_000_000 // B.nm]
        dij = C[a] - C[b]
        nij = _image(dij, L)
        xij = dij - L * nij
        if first == "pair":   # third molecule k seen from i
            dki = C[None] - C[a][:, None]
            nki = _image(dki, L)
            xki = dki - L * nki
            xkj = xki + xij[:, None]
            ok = ((xki ** 2).sum(-1) < rc * rc) & ((xkj ** 2).sum(-1) < rc * rc)
            m = torch.arange(B.nm, device=B.dev)[None]
            ok &= (m != a[:, None]) & (m != b[:, None])
        else:
            dik = C[a][:, None] - C[None]
            nki = _image(dik, L)
            xik = dik - L * nki
            xjk = C[b][:, None] - C[None] + L * nij[:, None] - L * nki
            ok = ((xik ** 2).sum(-1) < rc * rc) & ((xjk ** 2).sum(-1) < rc * rc)
            ok &= torch.arange(B.nm, device=B.dev)[None] > b[:, None]
        p, k = torch.nonzero(ok, as_tuple=True)
        yield a[p], b[p], k, nij[p], nki[p, k]


def _fs2(B, fit):
    """FS2 energy (kcal/mol), its gradients and the number of spectator triples."""
    g = [torch.zeros_like(x) for x in (B.P, B.C, B.scale)]
    total, count = 0.0, 0
    qk = torch.tensor(FS2_CHARGE, dtype=torch.float64, device=B.dev)
    for tri in _triples(B, fit["rc3"], "pair"):
        count += tri[0].numel()
        for part in zip(*(t.split(40000) for t in tri)):
            i, j, k, nij, nki = part
            c, P, L = B.c() / BOHR, B.p() / BOHR, B.L * B.scale / BOHR
            xij = c[i] - c[j] - L * nij
            xki = c[k] - c[i] - L * nki
            xkj = xki + xij
            rij = torch.linalg.norm(xij, dim=-1)
            flr = 1.0
            for x in (xki, xkj):
                w = 1.0 + torch.exp(fit["alpha3"] * BOHR * (torch.linalg.norm(x, dim=-1) - 7.40446 / BOHR))
                flr = flr * w ** -fit["delta33"]
            d = P[i][:, :3, None] - P[j][:, None, :3] - (L * nij)[:, None, None, :]
            exch = 0.48056977605478400 * torch.exp(-0.85836606579445000 * torch.linalg.norm(d, dim=-1))
            spect = P[k][:, :5] - c[i][:, None] - (L * nki)[:, None]
            u = (0.4 * xij / rij[:, None])[:, None]
            n = lambda t: 1.0 / torch.linalg.norm(t, dim=-1)  # noqa: E731
            term = n(spect) + n(spect + xij[:, None]) - n(spect - u) - n(spect + xij[:, None] + u)
            e = H2KCAL * (exch.sum((1, 2)) * flr * (term * qk).sum(-1)).sum()
            for t, v in zip(g, B.backward(e)):
                t += v
            total = total + e.detach()
    return total, g, count


def _fs3(B, fit, par):
    """FS3 energy (kcal/mol), gradients (P, C, scale and the fit), triple and blend counts."""
    index = torch.as_tensor(fit["index"], device=B.dev)
    g = [torch.zeros_like(x) for x in (B.P, B.C, B.scale, *par)]
    total, count, blend = 0.0, 0, 0
    for tri in _triples(B, 6.3, "triple"):
        count += tri[0].numel()
        for part in zip(*(t.split(1024) for t in tri)):
            i, j, k, nij, nik = part
            c, P, L = B.c() / BOHR, B.p()[:, :17] / BOHR, B.L * B.scale / BOHR
            njk = nik - nij
            sep = lambda a, b, n: (a[:, :, None] - b[:, None, :]) - (L * n)[:, None, None, :]  # noqa: E731
            norm = lambda t: torch.linalg.norm(t, dim=-1)  # noqa: E731
            ravg = (norm(c[i] - c[j] - L * nij) + norm(c[i] - c[k] - L * nik) +
                    norm(c[j] - c[k] - L * njk)) / 3.0
            damp = (1.0 + torch.exp(fit["alpha3"] * BOHR * (ravg - 6.20446 / BOHR))) ** -fit["delta33"]
            lo, hi = 4.5 / BOHR, 5.5 / BOHR
            f = (ravg - lo) / (hi - lo)
            mid = 1.0 + 2.0 * f ** 3 - 3.0 * f ** 2
            one, zero = torch.ones_like(f), torch.zeros_like(f)
            w_sr = torch.where(ravg <= lo, one, torch.where(ravg >= hi, zero, mid))
            blend += int(((ravg > lo) & (ravg < hi)).sum())
            r = [norm(sep(P[i], P[j], nij)), norm(sep(P[i], P[k], nik)), norm(sep(P[j], P[k], njk))]
            e = 0.0
            for cs, bgr, w in ((par[0], par[2], w_sr), (par[1], par[3], 1.0 - w_sr)):
                b, gg, r0 = (bgr[n].view(17, 17) for n in range(3))
                ex = [torch.exp(-b * x) / (1.0 + torch.exp(-gg * (x - r0))) for x in r]
                U, V, W = ([y, y * x] for y, x in zip(ex, r))
                coef = cs[index]
                S = 0.0
                # power of a site belongs to the distance between the two others
                for pi, pj in itertools.product(range(2), repeat=2):
                    M = V[pj][:, :, None, :] * W[pi][:, None, :, :]
                    for pk in range(2):
                        S = S + (U[pk] * torch.einsum("nabc,abc->nab", M, coef[..., pi, pj, pk])).sum((1, 2))
                e = e + (w * damp * S).sum()
            e = H2KCAL * e
            for t, v in zip(g, B.backward(e, par)):
                t += v
            total = total + e.detach()
    return total, g, count, blend


def _evaluate(case, b, terms, dev):
    """Energies, the virial, -gradients by positions and centres, dipoles, FS3 parameter
    gradients and counts of the named terms."""
    fit = _fit(case["variant"])
    B = _Box(b, case["box"], fit["ns"], dev)
    t = lambda a: torch.tensor(a, dtype=torch.float64, device=dev)  # noqa: E731
    q, npol = t(fit["q"]), fit["npol"]
    pol = t(fit["pol"])[-npol:] * BOHR ** 3
    alpha, kmax = _ewald(case["box"])
    out = {"e": {k: 0.0 for k in ENERGIES}, "vir": 0.0, "f": torch.zeros_like(B.P),
           "c2": torch.zeros_like(B.C), "c3": torch.zeros_like(B.C), "mu": None, "par": None,
           "n": {}}

    def add(name, e, grads, unit=1.0):  # e in internal units / unit
        out["e"][name] = torch.as_tensor(e).item() * unit / KCAL
        out["f"] -= grads[0] * unit
        out["vir"] = out["vir"] + float(grads[2]) * unit

    near = B.pairs(RCUT) if terms & {"real", "induction"} else None
    for name, term, energy in (("scpe", "self", lambda: _self_energy(B, q, alpha)),
                               ("rcpe", "real", lambda: _real_energy(B, q, alpha, near)),
                               ("kcpe", "kspace", lambda: _kspace_energy(B, q, alpha, kmax))):
        if term in terms:
            e = energy()
            add(name, e, B.backward(e))
    if "induction" in terms:
        mu, e_ind = _dipoles(B, q, pol, alpha, kmax, near, npol)
        add("indpe", e_ind, B.backward(_induction_energy(B, q, pol, alpha, kmax, near, npol, mu)))
        out["mu"] = mu
    if "fs2" in terms and fit["fs2"]:
        e, g, out["n"]["n_fs2_triples"] = _fs2(B, fit)
        add("fs2pe", e, g, KCAL)
        out["c2"] -= g[1] * KCAL
    if "fs3" in terms:
        par = [t(fit[k]).requires_grad_() for k in ("cs_sr", "cs_lr", "bgr_sr", "bgr_lr")]
        e, g, out["n"]["n_fs3_triples"], out["n"]["n_fs3_blend"] = _fs3(B, fit, par)
        add("fs3pe", e, g, KCAL)
        out["c3"] -= g[1] * KCAL
        out["par"] = g[3:]
    return out


def _site_array(v, ld, first=0):
    """(nm, n, 3) site values as three (nm, ld) arrays, starting at site `first`."""
    a = v.cpu().numpy()
    full = np.zeros((a.shape[0], ld, 3))
    full[:, first:first + a.shape[1]] = a
    return [np.ascontiguousarray(full[:, :, k]) for k in range(3)]


def _centre_array(v):
    return [np.ascontiguousarray(v.cpu().numpy()[:, k]) for k in range(3)]


def exact(case, seed):
    """What run() returns, from the plain restatement; None where it gives no value: integer
    counts, the state after MD steps, and boxes whose dense dipole matrix is too large."""
    kind, nm, ld, ns = case["kind"], case["nm"], case["ld"], SITES_PER_MOL
    if kind == "md" or nm > 2200 or (kind == "batch" and case["frames"] * nm > 4500):
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    terms = {"hot": {"self", "real", "kspace", "induction", "fs2", "fs3"}, "three": {"fs2", "fs3"},
             "induction": {"induction"}, "kspace": {"kspace"}}.get(kind, {"induction", "fs2", "fs3"})
    all_ = [_evaluate(case, b, terms, dev) for b in _boxes(case, seed)]
    o, e = all_[0], all_[0]["e"]
    fit = _fit(case["variant"])
    p0 = ns - fit["npol"]
    if kind == "hot":
        return {"energies": {**{k: e[k] for k in ENERGIES if k != "vir"}, "vir": o["vir"]},
                "counts": None, "f": _site_array(o["f"], ld),
                "c2": _centre_array(o["c2"]) if fit["fs2"] else None,
                "c3": _centre_array(o["c3"]), "mu": _site_array(o["mu"], ld, p0)}
    if kind == "three":
        return {"fs2pe": e["fs2pe"], "fs3pe": e["fs3pe"], "vir": np.array([o["vir"]]),
                "f": _site_array(o["f"], ld), "c2": _centre_array(o["c2"]) if fit["fs2"] else None,
                "c3": _centre_array(o["c3"])}
    if kind == "induction":
        return {"indpe": e["indpe"], "ind_iters": None, "vir": np.array([o["vir"]]),
                "f": _site_array(o["f"], ld), "mu": _site_array(o["mu"], ld, p0)}
    if kind == "kspace":
        return {"kcpe": np.array([e["kcpe"]]), "vir": np.array([o["vir"]]),
                "f": _site_array(o["f"], ld)}
    if kind == "train":
        energy = e["indpe"] + e["fs2pe"] + e["fs3pe"]
        g_sites = -o["f"] / KCAL
        g_com = g_sites.sum(1) - (o["c2"] + o["c3"]) / KCAL
        return {"energy": np.float64(energy),
                "grad": [g_com.cpu().numpy(), g_sites.cpu().numpy()] +
                        [v.cpu().numpy() for v in o["par"]]}
    stack = lambda rows: [np.stack(v) for v in zip(*rows)]  # noqa: E731
    # the batch's virial also counts the real-space Ewald terms, whose energies it leaves out
    return {"energies": np.array([[a["e"]["indpe"], a["e"]["fs2pe"], a["e"]["fs3pe"]]
                                  for a in all_]),
            "vir": None, "counts": None, "f": stack([_site_array(a["f"], ld) for a in all_]),
            "c2": stack([_centre_array(a["c2"]) for a in all_]) if fit["fs2"] else None,
            "c3": stack([_centre_array(a["c3"]) for a in all_]),
            "mu": stack([_site_array(a["mu"], ld, p0) for a in all_])}
