"""Performance cases: the work a variational Monte Carlo optimisation has this library do.

Each case is one call sequence of a user's program through the public binding
(mvmc-rs_b200/mvmc_b200.py, or the device-buffer entry points of include/mvmc_b200.h):

  step     sample -> measure -> SR solve, one whole optimisation step of a small chain
  sample   one block of Metropolis sweeps and its measurement, FP64 or mixed precision
  measure  local energies and O rows of configurations already sampled
  green    the PhysCal measurement: energy and the one- and two-body Green functions
  cg       SR-CG on device buffers the caller owns
  sr       the SR step of measured samples through the Gram matrix (TF32 / BF16 tensor
           cores and CG, or the direct solve by Cholesky)
  pfinv    batched Pfaffian + inverse on device buffers, uniform or mixed sides

Models, sizes and settings are those of mvmc-rs_b200/lattice.py and bench.py; synthetic
parameters uniform in [-0.05, 0.05], planes N(0, 1) + 0.5 J, as there.
"""
import ctypes
import importlib.util
import math
import os
import tempfile

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PACKAGE = os.path.join(ROOT, "mvmc-rs_b200")  # its name is no Python identifier
_MODULES = {}


def _module(name):
    if name not in _MODULES:
        spec = importlib.util.spec_from_file_location(name, os.path.join(PACKAGE, name + ".py"))
        _MODULES[name] = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(_MODULES[name])
    return _MODULES[name]


# ---- the cases -----------------------------------------------------------------------------
def _model(lx, ly, n_up, sub=1, nmp=1, nsp=1, tp=0.0, U=4.0):
    """Lattice, electrons per spin, sub-lattice period along x (and y for 4), momentum and
    spin projection points (NQP = nmp * nsp planes per walker)."""
    return {"lx": lx, "ly": ly, "n_up": n_up, "sub": sub, "nmp": nmp, "nsp": nsp, "tp": tp, "U": U}


SQUARE8 = _model(8, 8, 32, sub=2, nmp=4, nsp=2)           # n = 64, eight planes, 162 parameters
SQUARE16 = _model(16, 16, 112, tp=-0.2, U=6.0)            # n = 224, one plane, 386 parameters
SQUARE16_SR = _model(16, 16, 112, sub=4, tp=-0.2, U=6.0)  # n = 224, 4226 parameters


def listed():
    return [
        # the smallest model of an optimisation: short launches, host work between them
        {"name": "step_chain16", "kind": "step", "walkers": 256, "interval": 16, **_model(16, 1, 8)},
        # the production sampler with quantum-number projection: eight planes of side 64 per walker
        {"name": "sample_square8", "kind": "sample", "walkers": 1024, "interval": 8, "precision": 64, **SQUARE8},
        # the large lattice: one plane of side 224 per walker
        {"name": "sample_square16", "kind": "sample", "walkers": 1024, "interval": 1, "precision": 64, **SQUARE16},
        # the same in the mixed path: FP32 updates, FP64 refresh
        {"name": "sample_square16_mixed", "kind": "sample", "walkers": 1024, "interval": 1, "precision": 32,
         **SQUARE16},
        # measurement alone: every sample's planes from its configuration, O rows, averages
        {"name": "measure_square8", "kind": "measure", "walkers": 4096, **SQUARE8},
        {"name": "measure_square16", "kind": "measure", "walkers": 2048, **SQUARE16_SR},
        # fixed-parameter observables: 8192 + 16384 Green functions
        {"name": "green_square8", "kind": "green", "walkers": 1024, **SQUARE8},
        # SR-CG at the parameter count of the large lattice
        {"name": "cg_8192x4226", "kind": "cg", "samples": 8192, "params": 4226},
        # SR on the tensor cores (the mixed path's operator) and the direct solve
        {"name": "sr_tf32_square16", "kind": "sr", "solver": "tf32", "walkers": 4096, **SQUARE16_SR},
        {"name": "sr_direct_square16", "kind": "sr", "solver": "direct", "walkers": 4096, **SQUARE16_SR},
        # batched Pfaffian + inverse: a uniform batch and five sides in one launch
        {"name": "pfinv_64", "kind": "pfinv", "sides": "64", "planes": 8192},
        {"name": "pfinv_mix", "kind": "pfinv", "sides": "32 48 64 96 128", "planes": 8190},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(max(lo, hi))))))


def _draw_model(rng, max_sites=256, max_planes=8):
    """Chains and rectangles of 8 to max_sites sites, from a third to half filling."""
    while True:
        if rng.random() < 0.2:
            lx, ly = _log_uniform(rng, 8, min(64, max_sites)), 1
        else:
            lx, ly = rng.randint(3, 16), rng.randint(3, 16)
        if 8 <= lx * ly <= max_sites:
            break
    ns = lx * ly
    n_up = rng.randint(max(2, ns // 3), ns // 2)
    sub = 2 if lx % 2 == 0 and rng.random() < 0.5 else 1
    nmp, nsp = rng.choice([1, 1, 2, 4]), rng.choice([1, 1, 2])
    if ns > 100 or nmp * nsp > max_planes:
        nmp = nsp = 1
    return _model(lx, ly, n_up, sub, nmp, nsp, tp=rng.choice([0.0, -0.2]) if ly > 1 else 0.0,
                  U=float(rng.choice([2.0, 4.0, 6.0])))


def draw(rng):
    kind = rng.choice(["step", "sample", "sample", "measure", "green", "cg", "sr", "pfinv", "pfinv"])
    if kind == "pfinv":
        sides = sorted({2 * rng.randint(4, 64) for _ in range(rng.choice([1, 1, 3, 5]))})
        if len(sides) == 1 and rng.random() < 0.25:
            sides = [2 * rng.randint(65, 112)]
        cost = sum(s ** 3 for s in sides) / len(sides)
        return {"kind": kind, "sides": " ".join(map(str, sides)),
                "planes": max(1, _log_uniform(rng, 32, min(8192, 5e9 / cost)))}
    if kind == "cg":
        samples = _log_uniform(rng, 200, 8192)
        return {"kind": kind, "samples": samples, "params": _log_uniform(rng, 60, min(samples, 4226))}
    case = {"kind": kind, **_draw_model(rng, *{"green": (64,), "step": (64, 4)}.get(kind, ()))}
    n, sites, planes = 2 * case["n_up"], case["lx"] * case["ly"], case["nmp"] * case["nsp"]
    if kind in ("step", "sample"):
        case["interval"] = rng.randint(1, 16)
        moves = case["interval"] * sites * planes * max(n, 16) ** 2
        case["walkers"] = _log_uniform(rng, 16, min(1024, max(16, 1.5e10 / moves)))
        if kind == "sample":
            case["precision"] = rng.choice([64, 64, 64, 32]) if planes == 1 else 64
    elif kind == "measure":
        case["walkers"] = _log_uniform(rng, 64, min(4096, max(64, 1e10 / (planes * n ** 3))))
    elif kind == "green":
        case["walkers"] = _log_uniform(rng, 32, 1024)
    else:
        case["solver"] = rng.choice(["tf32", "bf16", "direct"])
        case["walkers"] = _log_uniform(rng, 256, 4096)
    return case


# ---- inputs --------------------------------------------------------------------------------
def _engine(case, seed):
    """The engine of a case's model, made from Expert-mode files as a user's program does."""
    lattice, mb = _module("lattice"), _module("mvmc_b200")
    sub, kind = case["sub"], case["kind"]
    args = dict(t=1.0, tp=case["tp"], U=case["U"], n_up=case["n_up"], sub=(4, 4) if sub == 4 else (sub, 1),
                nmp=case["nmp"], shifts=[(0, 0), (1, 0), (0, 1), (1, 1)] if case["ly"] > 1 else
                [(0, 0), (1, 0), (2, 0), (3, 0)],
                nsp_gauss_leg=case["nsp"], interval=case.get("interval", 1), samples=1,
                warmup=4 if kind in ("step", "sample") else 1, param_seed=seed,
                nsrcg=0 if case.get("solver") == "direct" else 1, calc_mode=1 if kind == "green" else 0,
                green="corr" if kind == "green" else None)
    opt = dict(walkers=case["walkers"], precision=case.get("precision", 64), seed=seed % (1 << 31))
    if opt["precision"] == 32:
        opt.update(refresh_sweeps=32, refresh_guard=0.03)
    if case.get("solver") in ("tf32", "bf16"):
        opt.update(sr_precision=32 if case["solver"] == "tf32" else 16, sr_gram=1)
    with tempfile.TemporaryDirectory(prefix="mvmc_case_") as path:
        namelist, initial, _ = lattice.write_inputs(path, case["lx"], case["ly"], **args)
        if kind == "green":
            return mb.Engine(namelist, physcal_zqp=initial, **opt)
        return mb.Engine(namelist, initial_def=initial, **opt)


def _planes(case, seed):
    sides = [int(s) for s in case["sides"].split()]
    order = [sides[p % len(sides)] for p in range(case["planes"])]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    offsets = np.concatenate([[0], np.cumsum(np.asarray(order, dtype=np.int64) ** 2)])
    x = torch.empty(int(offsets[-1]), dtype=torch.float64, device="cuda")
    off = torch.from_numpy(offsets[:-1].copy()).cuda()
    for k, n in enumerate(sides):
        start = off[k::len(sides)]
        a = torch.triu(torch.randn((len(start), n, n), dtype=torch.float64, device="cuda", generator=gen), 1)
        even = torch.arange(0, n, 2, device="cuda")
        a[:, even, even + 1] += 0.5
        a = a.transpose(1, 2) - a  # column-major planes: the transpose of the skew matrix
        x[(start[:, None] + torch.arange(n * n, device="cuda")[None, :]).reshape(-1)] = a.reshape(-1)
    return sides, order, x, off


def _cg_operands(case, seed):
    """Sample matrix with column means and scales as O rows have them, a few collective
    directions, and the energy gradient of a local energy that follows some of them."""
    ns, na = case["samples"], case["params"]
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, dtype=torch.float64, device="cuda", generator=gen)

    scale = 0.2 + 1.6 * torch.rand(na, dtype=torch.float64, device="cuda", generator=gen)
    modes = normal(ns, 8)
    o = normal(ns, na)
    o += modes @ normal(8, na) * 0.2
    o *= scale
    o += normal(na)
    mean = o.mean(0)
    diag = (o * o).mean(0) - mean * mean
    e = modes[:, :4].sum(1) + 2.0 * normal(ns) + 0.5 * (o[:, ::7] - mean[::7]).sum(1) / math.sqrt(na)
    g = -2.0 * 0.02 * ((o * (e - e.mean())[:, None]).mean(0))
    return o, mean, diag, g


CG_SHIFT, CG_TOL, CG_MAX = 0.02, 1e-9, 200


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "pfinv":
        sides, order, x, off = _planes(case, seed)
        uniform = len(sides) == 1
        state.update(x=x, planes=len(order), n_max=max(sides), n_uniform=sides[0] if uniform else 0,
                     sizes=None if uniform else torch.tensor(order, dtype=torch.int32, device="cuda"),
                     offsets=None if uniform else off, inv=torch.zeros_like(x),
                     pf=torch.zeros(len(order), dtype=torch.float64, device="cuda"),
                     status=torch.zeros(len(order), dtype=torch.int32, device="cuda"))
    elif kind == "cg":
        o, mean, diag, g = _cg_operands(case, seed)
        state.update(o=o, mean=mean, diag=diag, g=g, x=torch.zeros_like(g),
                     result=torch.zeros(3, dtype=torch.float64, device="cuda"))
    else:
        state["engine"] = engine = _engine(case, seed)
        if kind in ("measure", "green", "sr"):
            engine.sample()
        if kind == "sr":
            engine.measure()
    return state


# ---- one pass ------------------------------------------------------------------------------
def _address(t):
    return None if t is None else ctypes.c_void_p(t.data_ptr())


def _split(case, energy, ho, oo):
    """Averages of the projection factors' columns and of the orbitals' apart: their sizes
    differ by orders of magnitude."""
    k, size = 1 + _n_projection(case), len(ho)
    return {"energy": energy, "ho_projection": ho[:k], "ho_orbitals": ho[k:], "o_projection": oo[:k],
            "o_orbitals": oo[k:size], "oo_projection": oo[size:size + k], "oo_orbitals": oo[size + k:]}


def run(state):
    case, mb = state["case"], _module("mvmc_b200")
    kind = case["kind"]
    if kind == "pfinv":
        s = state
        rc = mb.lib().mvmc_b200_pfinv_batch_device(
            _address(s["x"]), _address(s["sizes"]), _address(s["offsets"]), s["n_uniform"], s["planes"], s["n_max"],
            _address(s["pf"]), _address(s["inv"]), _address(s["status"]), 64,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError("pfinv_batch_device: %d" % rc)
        return {"pf": s["pf"], "inv": s["inv"], "status": s["status"]}
    if kind == "cg":
        o, p = state["o"], torch.Tensor.data_ptr
        mb.cg_solve_noalloc(p(o), o.shape[0], o.shape[1], p(state["mean"]), p(state["diag"]), p(state["g"]),
                            1.0 / o.shape[0], CG_SHIFT, CG_TOL, CG_MAX, False, p(state["x"]), p(state["result"]),
                            torch.cuda.current_stream().cuda_stream)
        return {"x": state["x"]}
    engine = state["engine"]
    if kind == "green":
        energy, one, ex, two = engine.measure_green()
        return {"energy": energy, "one": one, "two": two}
    if kind == "sr":
        engine.sr_cg()
        return {"parameters": engine.parameters()}
    if kind in ("step", "sample"):
        engine.sample()
    energy, ho, oo = engine.measure()
    out = _split(case, energy, ho, oo)
    if kind == "step":
        engine.sr_cg()
        out["parameters"] = engine.parameters()
    return out


# ---- what a pass cannot do without ----------------------------------------------------------
def _n_projection(case):
    """One Gutzwiller factor and the Jastrow classes."""
    pairs = {min((dx, dy), ((-dx) % case["lx"], (-dy) % case["ly"]))
             for dx in range(case["lx"]) for dy in range(case["ly"])}
    return 1 + (len(pairs) - 1)


def _n_params(case):
    return _n_projection(case) + (16 if case["sub"] == 4 else case["sub"]) * case["lx"] * case["ly"]


def work(case):
    kind = case["kind"]
    if kind == "pfinv":
        sides = [int(s) for s in case["sides"].split()]
        order = [sides[p % len(sides)] for p in range(case["planes"])]
        # a skew plane in and out; its factorisation and inverse on one triangle
        return {"bytes": sum(16.0 * n * n for n in order), "flops": sum(float(n) ** 3 for n in order)}
    if kind == "cg":
        ns, na = case["samples"], case["params"]
        # the matrix once, and the 70 to 140 products with it and its transpose
        return {"bytes": 8.0 * ns * na + 40.0 * na, "flops": 140 * 4.0 * ns * na}
    w, ns, n = case["walkers"], case["lx"] * case["ly"], 2 * case["n_up"]
    planes, np_ = case["nmp"] * case["nsp"], _n_params(case)
    rows = 8.0 * w * (1 + np_)
    measure = {"bytes": rows + 4.0 * w * (n + 4 * ns), "flops": w * planes * (float(n) ** 3 + 2.0 * n * n)}
    if kind == "measure":
        return measure
    if kind == "green":
        # the factorisation, every allowed one-body hop of a plane, the lists' averages
        hops = 2.0 * case["n_up"] * (ns - case["n_up"])
        return {"bytes": 4.0 * w * (n + 4 * ns) + 8.0 * 6 * ns * ns,
                "flops": w * planes * (float(n) ** 3 + 2.0 * n * hops)}
    if kind == "sr":
        gram = float(w) * np_ * np_
        # S of the samples' one triangle, then its factorisation, or about 200 products with it
        return {"bytes": rows + 8.0 * np_,
                "flops": gram + (np_ ** 3 / 3.0 if case["solver"] == "direct" else 200 * 2.0 * np_ * np_)}
    # two blocks of `interval` sweeps; half of the proposals are hops (a row product), half
    # exchanges (a plane product), about a quarter is accepted (rank-2 or rank-4 update)
    moves = 2.0 * case["interval"] * ns * w * planes
    flops = moves * (n + n * n + 0.25 * (3.0 * n * n + 6.0 * n * n)) + measure["flops"]
    out = {"bytes": measure["bytes"] + 2.0 * 4 * w * (624 + n + 4 * ns), "flops": flops}
    if kind == "step":
        out["flops"] += 60 * 4.0 * w * np_
    return out


def tolerance(case):
    kind = case["kind"]
    if kind == "pfinv":
        # 64-bit sweeps with partial pivoting; the worst of thousands of random planes has a
        # condition number of 1e4 and more
        return {"rel": 1e-9, "max": 1e-6}
    if kind == "cg":
        # the solve stops at its tolerance, perhaps an iteration earlier or later
        return {"rel": 1e-5}
    if kind == "sr":
        # direct: 64-bit Gram and Cholesky; the others round the samples to TF32 / BF16 and
        # stop the CG before it has converged
        return {"rel": 1e-7} if case["solver"] == "direct" else {"rel": 3e-3, "max": 0.3}
    if kind == "green" or kind == "measure":
        return {"rel": 1e-7, "max": 1e-5}
    if case.get("precision") == 32:
        # an FP32 ratio near its threshold may decide otherwise: a few chains in a hundred
        # take another path, and their samples move the averages
        return {"rel": 0.03, "max": 0.9}
    if kind == "sample" and case["nmp"] * case["nsp"] > 1:
        # projected amplitudes: an ill-conditioned plane may turn one decision of one chain
        return {"rel": min(0.03, 1e-6 + 4.0 / case["walkers"]), "max": 0.9}
    # a step's CG stops at its tolerance, and the next pass samples the updated parameters
    return {"rel": 1e-4, "max": 1e-2} if kind == "step" else {"rel": 1e-6, "max": 1e-4}


# ---- 64-bit references ----------------------------------------------------------------------
def _pfaffian(a):
    """Pfaffians of a batch of skew matrices: Parlett-Reid elimination with partial pivoting."""
    a = a.clone()
    batch, n = a.shape[0], a.shape[1]
    pf = torch.ones(batch, dtype=a.dtype, device=a.device)
    rows = torch.arange(batch, device=a.device)
    for k in range(0, n - 1, 2):
        piv = k + 1 + a[:, k, k + 1:].abs().argmax(1)
        pf = torch.where(piv != k + 1, -pf, pf)
        t = a[rows, piv].clone()
        a[rows, piv] = a[:, k + 1]
        a[:, k + 1] = t
        t = a[rows, :, piv].clone()
        a[rows, :, piv] = a[:, :, k + 1]
        a[:, :, k + 1] = t
        d = a[:, k, k + 1].clone()
        pf = pf * d
        if k + 2 < n:
            u = a[:, k, k + 2:] / d[:, None]
            v = a[:, k + 1, k + 2:]
            a[:, k + 2:, k + 2:] += v[:, :, None] * u[:, None, :] - u[:, :, None] * v[:, None, :]
    return pf


class _Tables:
    """Index tables of a case's model (sites x + lx y; pair orbitals by sublattice and
    displacement; Jastrow classes by displacement under inversion)."""

    def __init__(self, case, parameters):
        lx, ly = case["lx"], case["ly"]
        self.ns = ns = lx * ly
        sx, sy = (4, 4) if case["sub"] == 4 else (case["sub"], 1)
        site = np.arange(ns)
        x, y = site % lx, site // lx
        dx, dy = (x[None, :] - x[:, None]) % lx, (y[None, :] - y[:, None]) % ly
        self.orb = ((x % sx) + sx * (y % sy))[:, None] * ns + dx + lx * dy
        self.n_orb = sx * sy * ns
        cls, jast = {}, np.full((ns, ns), -1)
        for i in range(ns):
            for j in range(ns):
                if i != j:
                    a, b = int(dx[i, j]), int(dy[i, j])
                    jast[i, j] = cls.setdefault(min((a, b), ((-a) % lx, (-b) % ly)), len(cls))
        self.jast, self.n_jast = jast, len(cls)
        p = np.asarray(parameters)
        self.gutz, self.f = p[0], p[1 + self.n_jast:]
        self.v = np.where(jast >= 0, p[1:1 + self.n_jast][np.maximum(jast, 0)], 0.0)
        shifts = [(0, 0), (1, 0), (0, 1), (1, 1)] if ly > 1 else [(0, 0), (1, 0), (2, 0), (3, 0)]
        trans = [((x + a) % lx) + lx * ((y + b) % ly) for a, b in shifts[:case["nmp"]]]
        if case["nsp"] == 1:
            spin = [(0.0, 1.0, 0.0, 1.0)]
        else:
            z, w = np.polynomial.legendre.leggauss(case["nsp"])
            beta, w = 0.5 * math.pi * (z + 1.0), 0.5 * math.pi * w
            spin = [(math.cos(b / 2) * math.sin(b / 2), math.cos(b / 2) ** 2, math.sin(b / 2) ** 2,
                     0.5 * math.sin(b) * c) for b, c in zip(beta, w)]
        self.planes = [(t, s) for t in trans for s in spin]
        hop = np.zeros((ns, ns))  # amplitude of every listed transfer i <- j
        for i in range(ns):
            near = [(1, 0, 1.0), (-1, 0, 1.0)]
            if ly > 1:
                near += [(0, 1, 1.0), (0, -1, 1.0)]
                if case["tp"] != 0.0:
                    near += [(a, b, case["tp"]) for a in (1, -1) for b in (1, -1)]
            for a, b, amp in near:
                hop[i, (x[i] + a) % lx + lx * ((y[i] + b) % ly)] += amp
        self.hop, self.U = hop, case["U"]

    def slater(self, plane, dev):
        t, (cs, cc, ss, _) = plane
        f = torch.from_numpy(self.f[self.orb[np.ix_(t, t)]]).to(dev)
        g = f.T
        return torch.cat([torch.cat([-(f - g) * cs, f * cc + g * ss], 1),
                          torch.cat([-f * ss - g * cc, (f - g) * cs], 1)], 0)


def _observables(case, tables, idx, num, green):
    """Local energies and O rows (or one-body Green functions) of configurations idx [W, n]
    (site of each electron, up electrons first), num [W, 2 ns], in 64 bits."""
    dev, ns, ne = "cuda", tables.ns, case["n_up"]
    w, n = idx.shape
    spin = torch.cat([torch.zeros(ne), torch.ones(ne)]).long().to(dev)
    rs = idx + ns * spin[None, :]
    ip = torch.zeros(w, dtype=torch.float64, device=dev)
    hop = torch.zeros((w, n, ns), dtype=torch.float64, device=dev)  # electron -> site of its spin
    deriv = None if green else torch.zeros((w, tables.n_orb), dtype=torch.float64, device=dev)
    for plane in tables.planes:
        t, (cs, cc, ss, weight) = plane
        table = tables.slater(plane, dev)
        x = table[rs[:, :, None], rs[:, None, :]]
        inv = torch.linalg.inv(x)
        inv = 0.5 * (inv - inv.transpose(1, 2))
        pf = weight * _pfaffian(x)
        ip += pf
        for s in (0, 1):
            m = slice(s * ne, (s + 1) * ne)
            rows = table[s * ns:(s + 1) * ns][:, rs].permute(1, 0, 2)  # [W, ns, n]
            hop[:, m] -= pf[:, None, None] * (inv[:, m] @ rows.transpose(1, 2))
        if deriv is not None:
            tr = torch.from_numpy(t).to(dev)[idx]
            orb = torch.from_numpy(tables.orb).to(dev)[tr[:, :, None], tr[:, None, :]]
            fac = torch.empty((n, n), dtype=torch.float64, device=dev)
            fac[:ne, :ne], fac[:ne, ne:], fac[ne:, :ne], fac[ne:, ne:] = cs, -cc, ss, -cs
            deriv.scatter_add_(1, orb.reshape(w, -1), (pf[:, None, None] * fac * inv).reshape(w, -1))
    up, dn = num[:, :ns].double(), num[:, ns:].double()
    charge = up + dn - 1.0
    v = torch.from_numpy(tables.v).to(dev)
    field = charge @ v
    # ratio of moving electron m to site i: exp(change of the projection) * Pf'/IP
    at = torch.gather(field, 1, idx)
    other = torch.cat([dn[:, None, :].expand(w, ne, ns), up[:, None, :].expand(w, ne, ns)], 1)  # other spin at i
    own = torch.gather(other, 2, idx[:, :, None])
    log = field[:, None, :] - at[:, :, None] - v[idx] + tables.gutz * (other - own)
    same = torch.cat([up[:, None, :].expand(w, ne, ns), dn[:, None, :].expand(w, ne, ns)], 1)
    ratio = torch.where(same == 0, torch.exp(log) * hop / ip[:, None, None], torch.zeros_like(hop))
    amp = torch.from_numpy(tables.hop).to(dev).T[idx]  # [W, n, i]: transfer i <- site of m
    energy = tables.U * (up * dn).sum(1) - (amp * ratio).sum((1, 2))
    if green:
        one = torch.zeros((w, 2, ns, ns), dtype=torch.float64, device=dev)  # [s, i, j]
        for s in (0, 1):
            m = slice(s * ne, (s + 1) * ne)
            one[:, s].scatter_(2, idx[:, None, m].expand(w, ns, ne), ratio[:, m].transpose(1, 2))
            one[:, s].diagonal(dim1=1, dim2=2).copy_((up, dn)[s])
        return energy, one
    double = (up * dn).sum(1, keepdim=True)
    pairs = torch.zeros((w, tables.n_jast), dtype=torch.float64, device=dev)
    i, j = np.triu_indices(ns, 1)
    pairs.index_add_(1, torch.from_numpy(tables.jast[i, j]).to(dev),
                     charge[:, torch.from_numpy(i).to(dev)] * charge[:, torch.from_numpy(j).to(dev)])
    return energy, torch.cat([torch.ones_like(double), double, pairs, deriv / ip[:, None]], 1)


def _averages(case, engine):
    got = engine.samples()
    w, ns, n = case["walkers"], case["lx"] * case["ly"], 2 * case["n_up"]
    idx = torch.from_numpy(got["ele_idx"].reshape(w, n)).cuda()
    num = torch.from_numpy(got["ele_num"].reshape(w, 2 * ns)).cuda()
    tables, green = _Tables(case, engine.parameters()), case["kind"] == "green"
    step = max(1, int(2e8 / (8.0 * max(n * n, n * ns))))
    e, rows = zip(*[_observables(case, tables, idx[k:k + step], num[k:k + step], green) for k in range(0, w, step)])
    e, sz = torch.cat(e), (num[:, :ns] - num[:, ns:]).double().sum(1)
    energy = torch.stack([torch.tensor(float(w), dtype=torch.float64, device="cuda"), e.mean(), (e * e).mean(),
                          sz.mean(), (sz * sz).mean()])
    if green:
        one = sum(r.sum(0) for r in rows) / w
        occ = num.double().reshape(w, 2, ns)
        two = torch.einsum("wsi,wtj->ijst", occ, occ) / w
        return {"energy": energy, "one": one, "two": two}
    o = torch.cat(rows)
    return _split(case, energy, (e[:, None] * o).mean(0), torch.cat([o.mean(0), (o * o).mean(0)]))


def _cg(o, mean, diag, g, max_iter):
    """Conjugate gradients on S = O^T O / W - mean mean^T + shift diag, residual refreshed
    every 20th iteration, stopped at |r|^2 < (tol n)^2."""
    def product(v):
        return (o @ v) @ o / o.shape[0] - mean * (mean @ v) + CG_SHIFT * diag * v

    x, r, d = torch.zeros_like(g), g.clone(), g.clone()
    delta = float(r @ r)
    for k in range(max_iter):
        if delta < (CG_TOL * len(g)) ** 2:
            break
        q = product(d)
        alpha = delta / float(d @ q)
        x = x + alpha * d
        r = g - product(x) if (k + 1) % 20 == 0 else r - alpha * q
        new = float(r @ r)
        d = r + (new / delta) * d
        delta = new
    return x


def _updated(case, engine, solver):
    """Parameters after the SR update of the engine's measured samples."""
    o = torch.from_numpy(engine.o_store()).cuda()
    e = torch.from_numpy(engine.local_energies()).cuda()
    mean = o.mean(0)
    var = (o * o).mean(0) - mean * mean
    g = -2.0 * 0.02 * ((e[:, None] * o).mean(0) - e.mean() * mean)
    active = torch.nonzero(var[1:] >= 1e-8 * var[1:].max()).reshape(-1) + 1
    a, m, d, g = o[:, active], mean[active], var[active], g[active]
    if solver == "direct":
        s = a.T @ a / len(e) - m[:, None] * m[None, :]
        x = torch.linalg.solve(s + torch.diag(CG_SHIFT * torch.diagonal(s)), g)
    else:
        x = _cg(a, m, d, g, CG_MAX)
    p = torch.from_numpy(engine.parameters()).cuda()
    p[active - 1] += x
    nproj = _n_projection(case)
    p[:nproj] -= p[:nproj].mean()
    p[nproj:] *= 4.0 / p[nproj:].abs().max()
    return {"parameters": p}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pfinv":
        sides, order, x, off = _planes(case, seed)
        pf = torch.zeros(len(order), dtype=torch.float64, device="cuda")
        inv = torch.zeros_like(x)
        for k, n in enumerate(sides):
            at = off[k::len(sides), None] + torch.arange(n * n, device="cuda")[None, :]
            a = x[at.reshape(-1)].reshape(-1, n, n).transpose(1, 2)
            pf[k::len(sides)] = _pfaffian(a)
            inv[at.reshape(-1)] = torch.linalg.inv(a).transpose(1, 2).reshape(-1)
        return {"pf": pf, "inv": inv, "status": None}
    if kind == "cg":
        return {"x": _cg(*_cg_operands(case, seed), CG_MAX)}
    if kind in ("measure", "green", "sr"):
        # the sampled configurations (or the measured rows) are these calls' inputs
        engine = prepare(case, seed)["engine"]
        if kind == "sr":
            return _updated(case, engine, case["solver"])
        return _averages(case, engine)
    return None  # a Markov chain: its decisions have no value in other arithmetic
