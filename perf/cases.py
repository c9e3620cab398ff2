"""The work that users of the engine have it do, as timed and compared cases.

Every case is one call (or one host-driven step) of the public Python API on a synthetic SPC/E +
NaCl system of `yamc_b200.systems` (jittered lattice, seeded orientations), with the random
numbers of the gfortran stream.  The kinds:

  step      one movemc driven by the host (`move_old` / `move_eval` / `move_commit`): the drop-in
            of a Fortran program that keeps its own loop; a call of a few ten microseconds
  npt       one host-driven volume step and one exchange step (`volume_*`, `xchange_*`)
  chain     one Markov chain on the device (`Engine.run_chain`), then its energies and positions:
            the whole run_mc loop of one simulation, FP64 or mixed, unbiased or force-biased
  batch     many independent chains advanced together (`Batch.run`), then every chain's energies
            and positions: production sampling, equal or ragged replicas
  energy    a new configuration's total energy (`set_positions`): start-up, rescoring of frames
  gradient  energy and its gradient through autograd (`total_energy(...).backward()`)
  rdf       radial distribution functions of a frame (`RDF.add_frame`, `result`)

FP64 chains return their move log as well; a mixed chain's per-move numbers are FP32 sums by
design, so it returns what such a run is kept for, its energies and configuration.  `exact` gives
the 64-bit value in plain torch wherever the outputs are one evaluation of a formula; the later
moves of a chain follow from all earlier accept decisions, so chains and batches have none.
"""
from __future__ import annotations

import math
import tempfile

import numpy as np
import torch

from yamc_b200 import _lib, api, rng as grng, systems
from yamc_b200.autograd import total_energy

PI = math.pi
PASSES = 4  # passes of fresh random numbers before a stream is used from its start again


# ------------------------------------------------------------------------------------------
# the cases
# ------------------------------------------------------------------------------------------
def _named(name):
    """System fields of one of the repository's named workloads."""
    s = systems.WORKLOADS[name]
    return {"n_water": s.n_water, "n_na": s.n_na, "n_cl": s.n_cl, "box": s.box, "alpha": s.alpha, "rc": s.rc,
            "kmax": s.kmax, "xlambda": s.xlambda}


def listed():
    small, medium, biased, large = (_named(n) for n in ("spce256", "nacl1m", "nacl4k", "nacl16k"))
    return [
        # a Fortran host calling the engine move by move (2048 waters + NaCl): latency
        {"name": "step_nacl1m", "kind": "step", **medium},
        # a host that runs its own NPT and exchange loop: one volume step, one exchange step
        {"name": "npt_nacl1m", "kind": "npt", **medium},
        # the smallest simulation, one cycle of one chain
        {"name": "chain_spce256", "kind": "chain", "precision": "fp64", "moves": 256, **small},
        # one production chain of the plain FP64 form, unbiased moves
        {"name": "chain_nacl1m", "kind": "chain", "precision": "fp64", "moves": 512, **medium},
        # one chain of the plain FP64 form, force-biased moves
        {"name": "chain_nacl4k_biased", "kind": "chain", "precision": "fp64", "moves": 200, **biased},
        # the largest system, one chain, force-biased, mixed precision
        {"name": "chain_nacl16k_biased_mixed", "kind": "chain", "precision": "mixed", "moves": 100, **large},
        # as many small chains as the GPU has SMs, plain FP64
        {"name": "batch_spce256", "kind": "batch", "precision": "fp64", "moves": 1024, "replicas": 148, **small},
        # the batched force-biased mixed form on 4096 waters + NaCl: as many chains as fit at once
        {"name": "batch_nacl4k_biased_mixed", "kind": "batch", "precision": "mixed", "moves": 64, "replicas": 45, **biased},
        # ragged replicas in one batch (216..4096 waters, 0..2 M NaCl, 280..360 K)
        {"name": "batch_ragged_biased_mixed", "kind": "batch", "precision": "mixed", "moves": 64, "replicas": 32, "ragged": 7},
        # the largest system's total energy
        {"name": "energy_nacl16k", "kind": "energy", **large},
        # energy and gradient, forward and backward
        {"name": "gradient_nacl4k", "kind": "gradient", **biased},
        # radial distribution functions of the largest system's frame
        {"name": "rdf_nacl16k", "kind": "rdf", "dr": 0.1, "rmax": 12.0, **large},
    ]


def _drawn_system(rng, n_lo, n_hi, biased):
    """A box of water and ions at the density, cutoff and Ewald accuracy range of the named ones."""
    nw = int(round(math.exp(rng.uniform(math.log(n_lo), math.log(n_hi)))))
    nion = int(round(nw * rng.uniform(0.0, 2.0) / 55.5))
    nmol = nw + 2 * nion
    box = (nmol / (0.0334 * (1.0 + rng.uniform(-0.02, 0.02)))) ** (1.0 / 3.0)
    rc = min(12.0, rng.uniform(0.44, 0.49) * box)
    sr = rng.uniform(2.7, 3.5)
    alpha = sr / rc
    kmax = max(3, int(round(alpha * box * rng.uniform(0.95, 1.15))))
    return {"n_water": nw, "n_na": nion, "n_cl": nion, "box": box, "alpha": alpha, "rc": rc, "kmax": kmax,
            "xlambda": 0.1 if biased else 0.0}


def draw(rng):
    kind = rng.choice(["step", "npt", "chain", "chain", "batch", "batch", "energy", "gradient", "rdf"])
    biased = rng.random() < 0.5
    if kind == "chain":
        return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "moves": rng.randint(64, 200),
                **_drawn_system(rng, 100, 8000, biased)}
    if kind == "batch":
        n = rng.randint(8, 40)
        if rng.random() < 0.3:
            return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "moves": rng.randint(32, 64), "replicas": n,
                    "ragged": rng.randint(8, 10000)}
        return {"kind": kind, "precision": rng.choice(["fp64", "mixed"]), "moves": rng.randint(32, 64), "replicas": n,
                **_drawn_system(rng, 100, 3000, biased)}
    case = {"kind": kind, **_drawn_system(rng, 100, 8000 if kind in ("energy", "rdf") else 4000, biased)}
    if kind == "rdf":
        case.update(dr=rng.choice([0.05, 0.1, 0.2]), rmax=min(12.0, 0.9 * rng.uniform(0.5, 1.0) * case["box"]))
    return case


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _spec(case, name="case"):
    return systems.SystemSpec(name, case["n_water"], case["n_na"], case["n_cl"], case["box"], case["alpha"], case["rc"],
                              case["kmax"], xlambda=case["xlambda"])


def _inputs(spec, seed):
    with tempfile.TemporaryDirectory() as d:
        f = systems.write_system(spec, d, seed=seed)
        return api.load_inputs(f["parameters"], f["composition"], f["moltab"])


def _batch_specs(case):
    if "ragged" in case:
        return systems.batch_specs(case["replicas"], seed=case["ragged"])
    return [_spec(case)] * case["replicas"]


def _draws(case):
    """Random numbers set aside for a pass of one chain (a move takes ~15 unbiased, ~22 force-biased)."""
    return case["moves"] * (48 if "ragged" in case or case["xlambda"] > 0 else 24)


def _precision(case):
    return _lib.YAMC_MIXED if case["precision"] == "mixed" else _lib.YAMC_FP64


def _proposal(case, seed, inp):
    """A rigid translation and rotation of one water: (molecule, new x, y, z of its atoms)."""
    r = np.random.default_rng(seed)
    imol = int(r.integers(1, case["n_water"] + 1))
    a, b = inp.first_atom[imol - 1] - 1, inp.last_atom[imol - 1]
    p = np.stack([inp.x[a:b], inp.y[a:b], inp.z[a:b]], 1)
    t = r.uniform(-0.05, 0.05)
    rot = np.array([[math.cos(t), -math.sin(t), 0.0], [math.sin(t), math.cos(t), 0.0], [0.0, 0.0, 1.0]])
    n = p[0] + (p - p[0]) @ rot.T + r.uniform(-0.05, 0.05, 3) / case["box"]
    return imol, n[:, 0].copy(), n[:, 1].copy(), n[:, 2].copy()


def _pair_of(case, seed):
    """Two different molecules that swap places: a water and an ion where there are ions."""
    r = np.random.default_rng(seed + 17)
    nmol = case["n_water"] + case["n_na"] + case["n_cl"]
    a = int(r.integers(1, case["n_water"] + 1))
    b = int(r.integers(case["n_water"] + 1, nmol + 1)) if nmol > case["n_water"] else a % nmol + 1
    return a, b


def _new_box(case, seed):
    return case["box"] * (1.0 + 0.001 * float(np.random.default_rng(seed + 23).uniform(0.2, 1.0)))


def _frame(case, seed):
    x, y, z, *_ = systems.generate(_spec(case), seed)
    return x, y, z


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "rdf":
        counts = np.array([n for n in (case["n_water"], case["n_na"], case["n_cl"]) if n], dtype=np.int32)
        s["rdf"] = api.RDF(np.repeat(np.arange(1, counts.size + 1, dtype=np.int32), counts), counts, case["dr"], case["rmax"])
        s["frame"] = _frame(case, seed)
    elif kind == "batch":
        specs = _batch_specs(case)
        s["batch"] = api.Batch([_inputs(sp, 1000 * seed + 3 + i) for i, sp in enumerate(specs)], precision=_precision(case))
        n = PASSES * _draws(case)
        stream = grng.gfortran_stream(12345 + seed, n * len(specs))
        s["streams"] = [stream[i * n:(i + 1) * n] for i in range(len(specs))]
        s["cursors"] = np.zeros(len(specs), dtype=np.int64)
    else:
        inp = _inputs(_spec(case), seed)
        s["engine"] = api.Engine(inp, precision=_precision(case) if kind == "chain" else _lib.YAMC_FP64)
        if kind == "step":
            s["move"] = _proposal(case, seed, inp)
        elif kind == "npt":
            s["pair"] = _pair_of(case, seed)
            s["new_box"] = _new_box(case, seed)
        elif kind == "chain":
            s["stream"] = grng.gfortran_stream(12345 + seed, PASSES * _draws(case))
            s["cursor"] = 0
        elif kind == "energy":
            s["xyz"] = (inp.x, inp.y, inp.z)
        elif kind == "gradient":
            s["positions"] = torch.from_numpy(np.stack([inp.x, inp.y, inp.z], 1)).cuda().requires_grad_()
    return s


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(s):
    return globals()["_run_" + s["kind"]](s)


def _run_step(s):
    imol, xn, yn, zn = s["move"]
    eng = s["engine"]
    f0, t0 = eng.move_old(imol)
    du, overlap, f1, t1 = eng.move_eval(imol, xn, yn, zn)
    eng.move_commit(False)
    return {"force_old": f0, "torque_old": t0, "du": du, "overlap": int(overlap), "force_new": f1, "torque_new": t1}


def _run_npt(s):
    eng = s["engine"]
    dv, ov = eng.volume_eval(s["new_box"])
    eng.volume_commit(False)
    dx, ox = eng.xchange_eval(*s["pair"])
    eng.xchange_commit(False)
    return {"du_volume": dv, "overlap_volume": int(ov), "du_xchange": dx, "overlap_xchange": int(ox)}


def _run_chain(s):
    case, eng = s["case"], s["engine"]
    need = _draws(case)
    if s["cursor"] + need > s["stream"].size:
        s["cursor"] = 0
    window = s["stream"][: s["cursor"] + need]
    log, _, s["cursor"], done, status = eng.run_chain(window, case["moves"], cursor=s["cursor"], log=case["precision"] == "fp64")
    out = {"cursor": int(s["cursor"]), "done": int(done), "status": int(status), "energies": eng.energies(),
           "positions": list(eng.positions())}
    if case["precision"] == "fp64":
        out["log"] = {k: log[k] for k in log.dtype.names}
    return out


def _run_batch(s):
    case, b = s["case"], s["batch"]
    need = _draws(case)
    if int(s["cursors"].max()) + need > s["streams"][0].size:
        s["cursors"][:] = 0
    _, s["cursors"], done, status, _ = b.run(s["streams"], case["moves"], cursors=s["cursors"], limits=s["cursors"] + need)
    views = [b.replica(i) for i in range(b.n)]
    return {"cursors": s["cursors"].copy(), "done": done, "status": status,
            "energies": np.stack([v.energies() for v in views]),
            "positions": np.concatenate([np.stack(v.positions()) for v in views], axis=1)}


def _run_energy(s):
    return s["engine"].set_positions(*s["xyz"])


def _run_gradient(s):
    p = s["positions"]
    p.grad = None
    u = total_energy(s["engine"], p)
    u.backward()
    return {"energy": u.detach(), "gradient": p.grad}


def _run_rdf(s):
    s["rdf"].add_frame(*s["frame"], s["case"]["box"])
    _, g, _, _ = s["rdf"].result()
    return g


# ------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------
def _k_count(kmax):
    """Signed k vectors of the half space kx >= 0 inside the sphere of radius kmax, without 0."""
    k = np.arange(-kmax, kmax + 1)
    k2 = (np.arange(0, kmax + 1) ** 2)[:, None, None] + (k ** 2)[None, :, None] + (k ** 2)[None, None, :]
    return int((k2 <= kmax * kmax).sum()) - 1


def _sizes(spec):
    nt = 1 + (spec.n_na > 0) + (spec.n_cl > 0)
    near = spec.natom / spec.box ** 3 * 4.0 / 3.0 * PI * spec.rc ** 3
    return nt, _k_count(spec.kmax), near


def _move_work(spec, forces):
    """One trial move: the neighbours of the molecule, the structure factors read (and written when
    accepted, taken as half of the moves), beta tables, two evaluations of its phases and pairs."""
    nt, S, near = _sizes(spec)
    na = spec.natom / spec.nmol
    nbytes = 40 * 1.3 * near + (1 + nt) * S * 16 * 1.5 + (1 + nt) * S * 8
    flops = 2 * na * near * 60 + S * (2 * na * 14 + 6 * (1 + nt))
    if forces:
        flops += S * 2 * na * (6 + 6 * nt)
    return nbytes, flops


def _sum_work(spec, per_pair):
    """A whole configuration: each pair inside the cutoff once, each atom's phase at each k vector
    (4 flop once the products along an axis are shared), the structure factors once."""
    nt, S, near = _sizes(spec)
    return 40 * spec.natom + (1 + nt) * S * 24, 0.5 * spec.natom * near * per_pair + 4.0 * spec.natom * S


def work(case):
    kind = case["kind"]
    if kind == "batch":
        specs = _batch_specs(case)
        parts = [_move_work(sp, sp.xlambda > 0) for sp in specs]
        return {"bytes": case["moves"] * sum(p[0] for p in parts), "flops": case["moves"] * sum(p[1] for p in parts)}
    spec = _spec(case)
    if kind == "step":
        b, f = _move_work(spec, True)
    elif kind == "chain":
        b, f = (case["moves"] * w for w in _move_work(spec, spec.xlambda > 0))
    elif kind == "npt":
        b, f = (x + y for x, y in zip(_sum_work(spec, 60), _move_work(spec, False)))
    elif kind == "energy":
        b, f = _sum_work(spec, 60)
    elif kind == "gradient":
        b, f = _sum_work(spec, 150)
        b, f = b + 48 * spec.natom, f + 12.0 * spec.natom * _k_count(spec.kmax)
    else:
        m, rho = spec.nmol, spec.nmol / spec.box ** 3
        nt, _, _ = _sizes(spec)
        b = 24 * m + 8 * nt * nt * case["rmax"] / case["dr"]
        f = m * rho * 4.0 / 3.0 * PI * case["rmax"] ** 3 * 14
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------------------------------
# the same numbers in plain torch, 64 bits
# ------------------------------------------------------------------------------------------
P_AS = (0.3275911, 0.254829592, -0.284496736, 1.421413741, -1.453152027, 1.061405429)
PI05 = 1.7724538509055


def _erfc_luc(x):
    """The energy's erfc: a series below 0.455, Abramowitz & Stegun 7.1.26 to 3, asymptotic above."""
    x2 = x * x
    e2 = torch.exp(-x2)
    series = 1.0 - 2.0 / PI05 * x * (1.0 - x2 * (1.0 / 3.0 - x2 * (0.1 - x2 * (1.0 / 42.0 - x2 / 216.0))))
    far = (1.0 - 0.5 * (1.0 - 1.5 / x2) / x2) / (PI05 * x) * e2
    p, a1, a2, a3, a4, a5 = P_AS
    t = 1.0 / (1.0 + p * x)
    mid = t * (a1 + t * (a2 + t * (a3 + t * (a4 + t * a5)))) * e2
    return torch.where(x < 0.455, series, torch.where(x > 3.0, far, mid))


def _beta_lj(b):
    """beta_6 and beta_12 of the dispersion sum at b = pi k / (alpha L), for an array of b."""
    p15 = PI ** 1.5
    nodes, weights = np.polynomial.legendre.leggauss(40)
    b6, b12 = np.empty_like(b), np.empty_like(b)
    for i, x in enumerate(b):
        if x <= 0.5:
            e2, x2 = math.exp(-x * x), x * x
            ek = float(_erfc_luc(torch.tensor(x, dtype=torch.float64)))
            b6[i] = p15 / 3.0 * x ** 3 * (math.sqrt(PI) * ek + (0.5 / x2 - 1.0) / x * e2)
            poly = (((1.0 / x2 - 2.0 / 7.0) / x2 + 4.0 / 35.0) / x2 - 8.0 / 105.0) / x2 + 16.0 / 105.0
            b12[i] = p15 / 1080.0 * x ** 9 * (-16.0 * math.sqrt(PI) / 105.0 * ek + poly / x * e2)
        else:
            edges = x * (1.0 + 14.0 / x) ** (np.arange(25) / 24.0)  # panels to where exp(-y^2) has vanished
            h = 0.5 * np.diff(edges)
            y = (edges[:-1] + h)[:, None] + h[:, None] * nodes[None, :]
            w = h[:, None] * weights[None, :] * np.exp(-y * y)
            b6[i] = p15 * x ** 3 / 2.0 * float((w / y ** 4).sum())
            b12[i] = p15 * x ** 9 / 120.0 * float((w / y ** 10).sum())
    return b6, b12


class _Exact:
    """The system of a case at box length `box`: tables and energies in 64 bits on the GPU."""

    def __init__(self, case, inp, box, temp=298.15, eps_ext=70.0):
        t = lambda v: torch.as_tensor(np.asarray(v, dtype=np.float64)).cuda()
        self.case, self.box = case, box
        self.aL = case["alpha"] * case["box"]
        self.rmax2 = (case["alpha"] * case["rc"] / self.aL) ** 2
        elec, epsi0, boltz = 1.602176e-19, 8.854187e-12, 1.38065e-23
        self.xclb = elec * elec / (4.0 * PI * epsi0 * boltz * temp) / 1.0e-10 / box
        self.kext = 2.0 * self.xclb * (PI / (2.0 * eps_ext + 1.0))
        self.q = t(inp.charge)
        self.mass = t(inp.mass)
        mol = np.repeat(np.arange(inp.first_atom.size), inp.last_atom - inp.first_atom + 1)
        self.mol = torch.as_tensor(mol).cuda()
        # LJ types in order of first appearance (none for atoms without sigma)
        key = [(a, b) if a >= 1e-8 else None for a, b in zip(inp.sigma.tolist(), inp.epsilon.tolist())]
        types = list(dict.fromkeys(k for k in key if k))
        self.nt = len(types)
        self.type = torch.as_tensor([types.index(k) if k else -1 for k in key]).cuda()
        sig = np.array([k[0] for k in types]) * (case["box"] / box)
        eps = np.array([k[1] for k in types])
        s6 = ((sig[:, None] + sig[None, :]) / 2.0) ** 6
        fe = 4.0 * np.sqrt(eps[:, None] * eps[None, :])
        self.s6, self.fe = t(s6), t(fe)
        self.lj6, self.lj12 = fe * s6, fe * s6 * s6
        # the signed k vectors of the half space and their weights
        km = case["kmax"]
        k = np.stack(np.meshgrid(np.arange(0, km + 1), np.arange(-km, km + 1), np.arange(-km, km + 1), indexing="ij"), -1)
        k = k.reshape(-1, 3)
        k2 = (k * k).sum(1)
        k, k2 = k[(k2 > 0) & (k2 <= km * km)], k2[(k2 > 0) & (k2 <= km * km)]
        two = np.where(k[:, 0] > 0, 2.0, 1.0)
        uniq, inv = np.unique(k2, return_inverse=True)
        b = PI / self.aL * np.sqrt(uniq.astype(np.float64))
        beta = self.xclb * np.exp(-b * b) / uniq / (2.0 * PI)
        b6, b12 = _beta_lj(b)
        b6, b12 = b6 * self.aL ** 3, b12 * self.aL ** 9
        self.k, self.beta = t(k), t(beta[inv] * two)
        lj = self.lj12[..., None] * b12[None, None, :] - self.lj6[..., None] * b6[None, None, :]
        self.beta_lj = t(lj[..., inv] * two)  # [nt, nt, S]
        n = np.asarray(inp.mol_numbers[: self.nt], dtype=np.float64)
        a = self.aL
        self.tail_c = -self.xclb * a / math.sqrt(PI) * float((self.q * self.q).sum())
        self.tail6 = PI ** 1.5 * a ** 3 / 6.0 * float(n @ self.lj6 @ n) - a ** 6 / 12.0 * float(np.diag(self.lj6) @ n)
        self.tail12 = PI ** 1.5 * a ** 9 / 1080.0 * float(n @ self.lj12 @ n) - a ** 12 / 1440.0 * float(np.diag(self.lj12) @ n)

    def pairs(self, x, i, j, same):
        """(ew, lj6, lj12, radial force factor, separation) of the atom pairs (i, j) inside the cutoff."""
        d = x[i] - x[j]
        d = torch.where(d > 0.5, d - 1.0, d)
        d = torch.where(d < -0.5, d + 1.0, d)
        r2 = (d * d).sum(-1)
        near = r2 < self.rmax2
        i, j, d, r2 = i[near], j[near], d[near], r2[near]
        r, a = r2.sqrt(), self.aL * r2.sqrt()
        a2 = a * a
        e2 = torch.exp(-a2)
        f = _erfc_luc(a) - (same[near].double() if same is not None else 0.0)
        qq = self.xclb * self.q[i] * self.q[j]
        ti, tj = self.type[i], self.type[j]
        lj = ((ti >= 0) & (tj >= 0)).double()
        s6 = self.s6[ti.clamp(min=0), tj.clamp(min=0)] / r2 ** 3
        fe = self.fe[ti.clamp(min=0), tj.clamp(min=0)] * lj
        c6 = 1.0 + a2 * (1.0 + a2 * 0.5)
        a6 = a2 ** 3
        c12 = c6 + a6 * (1.0 + a2 * (1.0 + a2 / 5.0) * 0.25) / 6.0
        fr = qq * (f / r + 2.0 * self.aL / math.sqrt(PI) * e2) / r2
        fr = fr + fe * 6.0 * s6 * e2 * (2.0 * s6 * (c12 + a6 * a6 / 720.0) - (c6 + a6 / 6.0)) / r2
        return qq * f / r, fe * s6 * e2 * c6, fe * s6 * s6 * e2 * c12, fr, d, near

    def real(self, x):
        """(ew, lj6, lj12) over all pairs, each once."""
        n = x.shape[0]
        tot = x.new_zeros(3)
        step = max(1, 6_000_000 // n)
        for i0 in range(0, n, step):
            with torch.no_grad():
                ii = torch.arange(i0, min(n, i0 + step), device=x.device)
                d = x.detach()[ii, None, :] - x.detach()[None, i0:, :]
                d = d - torch.round(d)
                hit = ((d * d).sum(-1) < self.rmax2 * (1.0 + 1e-9)).nonzero()
                a, b = hit[:, 0] + i0, hit[:, 1] + i0
                a, b = a[b > a], b[b > a]
                same = self.mol[a] == self.mol[b]
            ew, l6, l12, *_ = self.pairs(x, a, b, same)
            tot = tot + torch.stack([ew.sum(), l6.sum(), l12.sum()])
        return tot

    def rho(self, x, atoms=None):
        """Structure factors [1 + nt, S] (complex) of the atoms (all by default)."""
        atoms = torch.arange(x.shape[0], device=x.device) if atoms is None else atoms
        w = torch.stack([self.q] + [(self.type == t).double() for t in range(self.nt)])
        out = 0
        for c in atoms.split(max(1, 20_000_000 // self.k.shape[0])):
            ph = 2.0 * PI * (x[c] @ self.k.T)
            out = out + torch.complex(w[:, c] @ torch.cos(ph), w[:, c] @ torch.sin(ph))
        return out

    def k_energy(self, rho):
        c = (self.beta * (rho[0].real ** 2 + rho[0].imag ** 2)).sum()
        r = rho[1:]
        lj = (self.beta_lj * (r[:, None].real * r[None].real + r[:, None].imag * r[None].imag)).sum()
        return c, lj

    def external(self, mu):
        return self.kext * (mu * mu).sum()

    def energies(self, x):
        """The eight numbers of `Engine.energies`."""
        ew, l6, l12 = self.real(x)
        kc, kl = self.k_energy(self.rho(x))
        u_ew = ew + kc + self.tail_c + self.external((self.q[:, None] * x).sum(0))
        u_lj = l12 - l6 + kl + self.tail12 - self.tail6
        return torch.stack([u_ew + u_lj, u_ew, u_lj, ew, l6, l12, kc, kl])

    def molecule(self, x, m, xm):
        """Real-space energy and forces of molecule m placed at xm, in the configuration x."""
        own = (self.mol == m).nonzero()[:, 0]
        y = x.clone()
        y[own] = xm
        rest = (self.mol != m).nonzero()[:, 0]
        i, j = own.repeat_interleave(rest.numel()), rest.repeat(own.numel())
        ew, l6, l12, fr, d, near = self.pairs(y, i, j, None)
        f = torch.zeros_like(xm).index_add_(0, (i[near] - own[0]), d * fr[:, None])
        return ew.sum() + l12.sum() - l6.sum(), f, y

    def step(self, x, m, xm):
        """What the step case returns: forces and torques at the old and new positions, dU."""
        own = (self.mol == m).nonzero()[:, 0]
        rho0 = self.rho(x)
        out = {}
        e, mu = [], []
        rho = rho0
        for word, pos in (("old", x[own]), ("new", xm)):
            u, f, y = self.molecule(x, m, pos)
            if word == "new":
                rho = rho0 + self.rho(y, own) - self.rho(x, own)
            ph = 2.0 * PI * (pos @ self.k.T)
            c, s = torch.cos(ph), torch.sin(ph)
            w = self.q[own][:, None] * self.beta * (rho[0].real * s - rho[0].imag * c)
            for t in range(self.nt):
                field = self.beta_lj[t] * rho[1:]
                v = field.real.sum(0) * s - field.imag.sum(0) * c
                w = w + (self.type[own] == t).double()[:, None] * v
            mu.append((self.q[:, None] * y).sum(0))
            f = f + 4.0 * PI * (w @ self.k) - 2.0 * self.kext * self.q[own][:, None] * mu[-1]
            mass = self.mass[own]
            centre = (mass[:, None] * pos).sum(0) / mass.sum()
            out["force_" + word] = f.sum(0).cpu()
            out["torque_" + word] = torch.linalg.cross(pos - centre, f).sum(0).cpu()
            e.append(u)
        k0, k1 = self.k_energy(rho0), self.k_energy(rho)
        out["du"] = torch.stack([e[1] - e[0], k1[0] - k0[0], k1[1] - k0[1], self.external(mu[1]) - self.external(mu[0])]).cpu()
        return out

    def exchange(self, x, m1, m2):
        """dU of the exchange step: centres of mass swapped; the pair term of the two molecules
        counts with each of them, as in the acceptance test of the method."""
        own = [(self.mol == m).nonzero()[:, 0] for m in (m1, m2)]
        cm = [(self.mass[o][:, None] * x[o]).sum(0) / self.mass[o].sum() for o in own]
        y = x.clone()
        y[own[0]] = x[own[0]] - cm[0] + cm[1]
        y[own[1]] = x[own[1]] - cm[1] + cm[0]
        real = sum(self.molecule(y, m, y[o])[0] - self.molecule(x, m, x[o])[0] for m, o in zip((m1, m2), own))
        both = torch.cat(own)
        rho0 = self.rho(x)
        k0, k1 = self.k_energy(rho0), self.k_energy(rho0 + self.rho(y, both) - self.rho(x, both))
        mu0, mu1 = ((self.q[:, None] * v).sum(0) for v in (x, y))
        return torch.stack([real, k1[0] - k0[0], k1[1] - k0[1], self.external(mu1) - self.external(mu0)]).cpu()

    def scaled(self, x, ratio):
        """The atoms of every molecule drawn to its centre of mass by `ratio` (a larger box)."""
        n = int(self.mol.max()) + 1
        m = torch.zeros(n, dtype=torch.float64, device=x.device).index_add_(0, self.mol, self.mass)
        c = torch.zeros(n, 3, dtype=torch.float64, device=x.device).index_add_(0, self.mol, self.mass[:, None] * x) / m[:, None]
        c = c[self.mol]
        return (x - c) * ratio + c


def _exact_rdf(case, seed):
    pos = [torch.as_tensor(v).cuda() for v in _frame(case, seed)]
    counts = [n for n in (case["n_water"], case["n_na"], case["n_cl"]) if n]
    nt, L, dr, rmax = len(counts), case["box"], case["dr"], case["rmax"]
    if rmax >= L / 2:
        return None  # periodic images are counted too: the general loop
    typ = torch.repeat_interleave(torch.arange(nt), torch.tensor(counts)).cuda()
    nbin = int((rmax - 1e-10) / dr) + 2
    hist = torch.zeros(nt * nt * nbin, dtype=torch.float64, device="cuda")
    m = typ.numel()
    for i0 in range(0, m, 500):
        r2 = 0.0
        for v in pos:
            a, b = v[i0:i0 + 500, None], v[None, :]
            d = a - b
            b = torch.where(d > 0.5, b + 1.0, torch.where(d < -0.5, b - 1.0, b))
            r2 = r2 + ((a - b) * L) ** 2
        r2[torch.arange(r2.shape[0], device="cuda"), torch.arange(i0, i0 + r2.shape[0], device="cuda")] = 1e30
        i, j = (r2 <= rmax * rmax - 1e-10).nonzero(as_tuple=True)
        b = (torch.sqrt(r2[i, j]) / dr).long()
        ti, tj = typ[i + i0], typ[j]
        off = torch.minimum(ti, tj) * nt + torch.maximum(ti, tj)
        hist += torch.bincount((off * nbin + b)[b < nbin], minlength=hist.numel()).double()
    h = hist.reshape(nt, nt, nbin).cpu().numpy()
    r = np.arange(nbin) * dr
    dv = 4.0 * PI * dr * (r * r + r * dr) + 4.0 / 3.0 * PI * dr ** 3
    n = np.array(counts, dtype=np.float64)
    return h * L ** 3 / (n[:, None, None] * n[None, :, None]) / dv / np.where(np.eye(nt) > 0, 1.0, 2.0)[:, :, None]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("chain", "batch"):
        return None
    if kind == "rdf":
        return _exact_rdf(case, seed)
    inp = _inputs(_spec(case), seed)
    x = torch.from_numpy(np.stack([inp.x, inp.y, inp.z], 1)).cuda()
    sys_ = _Exact(case, inp, case["box"])
    if kind == "energy":
        return sys_.energies(x).cpu().numpy()
    if kind == "gradient":
        x.requires_grad_()
        u = sys_.energies(x)[0]
        u.backward()
        return {"energy": u.detach(), "gradient": x.grad}
    if kind == "step":
        imol, *xn = _proposal(case, seed, inp)
        return {"overlap": None, **sys_.step(x, imol - 1, torch.from_numpy(np.stack(xn, 1)).cuda())}
    new = _new_box(case, seed)
    big = _Exact(case, inp, new)
    du = big.energies(big.scaled(x, case["box"] / new))[0] - sys_.energies(x)[0]
    a, b = _pair_of(case, seed)
    return {"du_volume": float(du), "overlap_volume": None, "du_xchange": sys_.exchange(x, a - 1, b - 1), "overlap_xchange": None}
