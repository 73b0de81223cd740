"""Performance cases of the nonbonded library: what its callers have it do, over the range of
sizes they have, through the public entry points (moil_fnrfd_gb300.nb, include/moil_nb.h).

The families (field "kind"):
  eval      one nonbonded evaluation (gradient and energies) of a handle: a lone system or a batch
            of uneven replicas, on device buffers or through page-locked host buffers (MOIL's
            drop-in call), mixed or plain FP64
  md        a short device-resident trajectory from a saved state (a milestoning swarm, or one
            large box): leapfrog with rigid waters, lists rebuilt every 10 steps
  adjoint   parameter derivatives of perturbed copies of a solute system (force-field fitting)
  pressure  the molecular-virial analysis of a batch, host coordinates in, tensor out
  pme       the reciprocal sum alone through the allocation-free entry point

Handles are made once, as a program keeps them, with lists rebuilt every 10 evaluations.  The
C interface hands every result over in doubles; a result is returned here in the type whose
accuracy it has: float32 from the mixed path (its pair, spline and FFT arithmetic, and the
type of trajectory frames, is FP32), float64 from the plain FP64 path.
"""
import ctypes
import functools
import itertools
import math

import numpy as np
import torch

from moil_fnrfd_gb300 import nb as NB
from moil_fnrfd_gb300 import systems as S

LIST_PERIOD = 10
DT = 0.002                    # ps
ACCEL = 418.4                 # (kcal/mol/Å) / amu in Å/ps^2
KT300 = 0.0019872041 * 300.0  # kcal/mol
HEAVY_BOX = 62.2              # Å: the solute system the smaller ones are scaled from


def listed():
    def water(name, replicas, lo, hi, **kw):
        return {"name": name, "kind": "eval", "replicas": replicas, "waters_min": lo, "waters_max": hi,
                "precision": "mixed", "buffers": "device", **kw}

    return [
        # the smallest periodic system the 9 Å cutoff allows: a minimiser or sampler that calls
        # once per step, where latency counts
        water("box_216", 1, 216, 216),
        # the FP64 path as accuracy reference and for finite differences: smallest and middle size
        water("box_216_fp64", 1, 216, 216, precision="fp64"),
        water("box_1334_fp64", 1, 1334, 1334, precision="fp64"),
        # protein-like solute in water, one call per MOIL energy evaluation, host arrays
        {"name": "solute_host", "kind": "eval", "solute_box": HEAVY_BOX, "copies": 1, "precision": "mixed",
         "buffers": "host"},
        # a sweep over the interior images of a chain (images of one size), host arrays
        water("images_24_host", 24, 803, 803, buffers="host"),
        # 512 uneven replicas at once: path images or a milestoning swarm
        water("batch_512", 512, 500, 4000),
        # one 96,000-atom box through one list period of steps
        {"name": "md_96000", "kind": "md", "replicas": 1, "waters_min": 32000, "waters_max": 32000, "steps": 10},
        # a small swarm of short trajectories
        {"name": "swarm_16", "kind": "md", "replicas": 16, "waters_min": 500, "waters_max": 4000, "steps": 10},
        # parameter derivatives: one small solute per call, and a batch of perturbed copies
        {"name": "fit_small", "kind": "adjoint", "solute_box": 27.0, "copies": 1},
        {"name": "fit_8", "kind": "adjoint", "solute_box": HEAVY_BOX, "copies": 8},
        # pressure analysis of trajectory frames, several replicas per call
        {"name": "pressure_48", "kind": "pressure", "replicas": 48, "waters_min": 500, "waters_max": 4000},
        # the reciprocal sum beside another runtime's memory pool
        {"name": "pme_noalloc", "kind": "pme", "atoms": 23556, "box": HEAVY_BOX},
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["single", "single", "fp64", "solute", "batch", "batch_host", "md", "swarm", "adjoint",
                       "pressure", "pme"])
    if what in ("single", "fp64"):
        n = log_int(216, 24000 if what == "single" else 2600)
        return {"kind": "eval", "replicas": 1, "waters_min": n, "waters_max": n,
                "precision": "fp64" if what == "fp64" else "mixed",
                "buffers": rng.choice(["device", "host"]) if what == "single" else "device"}
    if what == "solute":
        return {"kind": "eval", "solute_box": round(rng.uniform(26.0, HEAVY_BOX), 1), "copies": rng.choice([1, 1, 2]),
                "precision": "mixed", "buffers": rng.choice(["device", "host"])}
    if what in ("batch", "batch_host"):
        host = what == "batch_host"
        n, lo = log_int(2, 64 if host else 256), log_int(216, 2000)
        return {"kind": "eval", "replicas": n, "waters_min": lo, "waters_max": min(4000, lo * rng.choice([1, 2, 8])),
                "precision": "mixed", "buffers": "host" if host else "device"}
    if what == "md":
        n = log_int(216, 24000)
        return {"kind": "md", "replicas": 1, "waters_min": n, "waters_max": n, "steps": rng.choice([1, 10, 17, 25])}
    if what == "swarm":
        lo = log_int(216, 2000)
        return {"kind": "md", "replicas": log_int(2, 48), "waters_min": lo, "waters_max": 2 * lo,
                "steps": rng.choice([5, 10, 20])}
    if what == "adjoint":
        return {"kind": "adjoint", "solute_box": round(rng.uniform(26.0, 50.0), 1), "copies": log_int(1, 12)}
    if what == "pressure":
        lo = log_int(216, 2000)
        return {"kind": "pressure", "replicas": log_int(1, 48), "waters_min": lo, "waters_max": 2 * lo}
    return {"kind": "pme", "atoms": log_int(500, 65000), "box": round(rng.uniform(20.0, 63.9), 1)}


# ---- inputs ---------------------------------------------------------------------------


def _rng(*words):
    return np.random.Generator(np.random.PCG64([int(w) & 0x7FFFFFFF for w in words]))


def _water_counts(case):
    """Waters per replica, log-uniform between the case's limits (the same for every seed)."""
    lo, hi, n = case["waters_min"], case["waters_max"], case["replicas"]
    u = _rng(n, lo, hi).random(n)
    return [int(round(lo * (hi / lo) ** x)) for x in u]


def _water_geometry(rng, n):
    """n rigid TIP3P molecules about their oxygens, uniformly random orientations, (n, 3, 3)."""
    half = math.radians(S.TIP3_HOH_DEG) / 2.0
    h = S.TIP3_ROH * np.array([math.sin(half), math.cos(half)])
    q = rng.normal(size=(n, 2, 3))
    a = q[:, 0] / np.linalg.norm(q[:, 0], axis=1)[:, None]
    b = q[:, 1] - (q[:, 1] * a).sum(1)[:, None] * a
    b /= np.linalg.norm(b, axis=1)[:, None]
    return np.stack([np.zeros((n, 3)), h[0] * a + h[1] * b, -h[0] * a + h[1] * b], axis=1)


def _water_system(n, seed):
    """A box of n TIP3P waters at liquid density: jittered lattice, random orientations (the
    layout of systems.water_box, assembled in whole arrays); 9 Å cutoff below 24,000 waters,
    above it the 10 Å cutoff of the large box."""
    rng = _rng(seed, n)
    box, rc, alpha = (n / S.WATER_DENSITY) ** (1.0 / 3.0), 9.0, 0.35
    if n == 216:
        box = 18.62
    if n > 24000:
        box, rc, alpha = box * 98.6 / (32000 / S.WATER_DENSITY) ** (1.0 / 3.0), 10.0, 0.32
    m = int(math.ceil(round(n ** (1.0 / 3.0), 9)))
    g = (np.arange(m) + 0.5) * (box / m) - box / 2.0
    sites = np.stack([v.ravel() for v in np.meshgrid(g, g, g, indexing="ij")], axis=1)
    sites = sites[np.sort(rng.choice(m ** 3, size=n, replace=False))]
    oxy = sites + rng.uniform(-0.3, 0.3, size=sites.shape)
    coor = (_water_geometry(rng, n) + oxy[:, None, :]).reshape(-1, 3)
    sig = S.rmin2_to_sigma(S.TIP3_RMIN2_O)
    e6, e12 = S.lj_encode(np.tile([S.TIP3_EPS_O, 0.0, 0.0], n), np.tile([sig, 0.0, 0.0], n), False)
    first = 3 * np.arange(n, dtype=np.int32)[:, None]
    exc1 = np.concatenate([[0], (first + np.array([2, 3, 3])).ravel()])
    grid = S.smooth_grid(box)
    return S.MoilSystem(
        name="water", coor=coor, ptchg=np.tile([S.TIP3_QO, S.TIP3_QH, S.TIP3_QH], n), epsgm6=e6, epsgm12=e12,
        exc1=exc1.astype(np.int32), exc2=(first + np.array([2, 3, 3])).ravel().astype(np.int32),
        spec1=np.zeros(0, np.int32), spec2=np.zeros(0, np.int32), p14=np.zeros((0, 3)),
        poipt=(first.ravel() + 3).astype(np.int32), montype=np.full(n, S.MON_WATER, np.int32), box=(box,) * 3,
        rvmx=rc, relx=rc, alpha=alpha, nfft=(grid,) * 3, seed=seed)


@functools.lru_cache(maxsize=2)
def _solute_base(box):
    f = (box / HEAVY_BOX) ** 3
    if box == HEAVY_BOX:
        return S.config1()
    s = S.config1(seed=41, n_solute=max(60, int(2489 * f)), n_ions=7, n_waters=int(5600 * f), box=box)
    s.nfft = (S.smooth_grid(box),) * 3
    return s


def _solute_systems(box, copies, seed):
    """Copies of the solute system with +-1% perturbed parameters (the first with its own), the
    coordinates moved from the seed: waters and ions as wholes, solute atoms a little."""
    base = _solute_base(box)
    out = [base] + (S.perturbed_copies(base, copies - 1, seed=4000) if copies > 1 else [])
    moved = []
    for k, s in enumerate(out):
        rng = _rng(seed, 17, k)
        d = rng.uniform(-0.02, 0.02, size=(s.npt, 3))
        w = s.npt - 3 * s.nwaters
        d[w:] = np.repeat(rng.uniform(-0.15, 0.15, size=(s.nwaters, 3)), 3, axis=0)
        t = s.copy()
        t.coor = s.coor + d
        moved.append(t)
    return moved


def _systems(case, seed):
    if "solute_box" in case:
        return _solute_systems(case["solute_box"], case["copies"], seed)
    return [_water_system(n, 1000 * seed + k) for k, n in enumerate(_water_counts(case))]


def _masses(n_waters):
    return np.tile([S.MASS_O, S.MASS_H, S.MASS_H], n_waters)


def _velocities(s, seed):
    """Rigid-body velocities of every water at 300 K (Å/ps)."""
    rng = _rng(seed, 23, s.npt)
    x = s.coor.reshape(-1, 3, 3)
    m = np.array([S.MASS_O, S.MASS_H, S.MASS_H])
    r = x - ((m[:, None] * x).sum(1) / m.sum())[:, None, :]
    n = x.shape[0]
    vc = rng.normal(size=(n, 3)) * math.sqrt(KT300 * ACCEL / m.sum())
    om = rng.normal(size=(n, 3)) * math.sqrt(KT300 * ACCEL / 1.2)      # moments of inertia near 1.2 amu Å^2
    return (vc[:, None, :] + np.cross(om[:, None, :], r)).reshape(-1, 3)


def _pme_inputs(case, seed):
    """Waters' worth of charges at random places of a cubic box (neutral in threes)."""
    n = case["atoms"]
    rng = _rng(seed, 31, n)
    q = np.tile([S.TIP3_QO, S.TIP3_QH, S.TIP3_QH], n // 3 + 1)[:n].copy()
    q -= q.sum() / n
    return rng.uniform(-0.5, 0.5, size=(n, 3)) * case["box"], q


def _pme_grid(case):
    return min(S.smooth_grid(case["box"]), 64)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "pme":
        x, q = _pme_inputs(case, seed)
        L = NB.load()
        fn = L.moil_nb_pme_noalloc
        fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                       ctypes.POINTER(ctypes.c_int), ctypes.c_double, ctypes.c_double, ctypes.c_void_p,
                       ctypes.POINTER(ctypes.c_double), ctypes.c_void_p]
        dx = torch.from_numpy(x).cuda()
        st = {"kind": kind, "fn": fn, "x": dx, "q": torch.from_numpy(q).cuda(), "g": torch.empty_like(dx),
              "box": (ctypes.c_double * 3)(*([case["box"]] * 3)), "grid": (ctypes.c_int * 3)(*([_pme_grid(case)] * 3))}
        torch.cuda.synchronize()
        return st
    systems = _systems(case, seed)
    one = len(systems) == 1
    fp64 = case.get("precision") == "fp64"
    nb = NB.Nonbonded(systems[0] if one else systems, precision=NB.MOIL_NB_FP64 if fp64 else NB.MOIL_NB_MIXED,
                      skin=1.5 if kind == "md" else 1.0, list_period=LIST_PERIOD)
    coor = torch.from_numpy(np.concatenate([s.coor for s in systems]))
    st = {"kind": kind, "nb": nb, "dtype": torch.float64 if fp64 else torch.float32,
          "stream": torch.cuda.ExternalStream(nb.stream())}
    if kind == "eval" and case["buffers"] == "device":
        st.update(kind="device", x=coor.cuda(), g=torch.empty_like(coor, device="cuda"))
    elif kind == "md":
        vel = torch.from_numpy(np.concatenate([_velocities(s, seed) for s in systems]))
        st.update(x0=coor.cuda(), v0=vel.cuda(), m=torch.from_numpy(_masses(nb.natom // 3)).cuda(),
                  steps=case["steps"])
        st.update(x=torch.empty_like(st["x0"]), v=torch.empty_like(st["v0"]))
    else:
        st["x"] = coor.pin_memory()
        if kind == "adjoint":
            st["out"] = [torch.empty(nb.natom, dtype=torch.float64).pin_memory() for _ in range(3)]
        elif kind == "pressure":
            nb.set_molecules(np.concatenate([np.arange(s.npt, dtype=np.int32) // 3 for s in systems]),
                             _masses(nb.natom // 3))
        else:
            st["g"] = torch.empty_like(coor).pin_memory()
    torch.cuda.synchronize()
    return st


# ---- one pass -------------------------------------------------------------------------


def _energies(es, dtype):
    """(replicas, 11) in the order of the interface's structure."""
    kind = np.float64 if dtype == torch.float64 else np.float32
    return np.fromiter(itertools.chain.from_iterable(e.values() for e in es), kind,
                       len(es) * len(NB.ENERGY_KEYS)).reshape(len(es), -1)


def run(state):
    kind = state["kind"]
    if kind == "pme":
        e = ctypes.c_double()
        stream = torch.cuda.current_stream()
        rc = state["fn"](state["x"].data_ptr(), state["q"].data_ptr(), state["x"].shape[0], state["box"],
                         state["grid"], 0.35, 1.0, state["g"].data_ptr(), ctypes.byref(e), stream.cuda_stream)
        if rc != 0:
            raise RuntimeError(f"moil_nb_pme_noalloc: status {rc}")
        return {"dpot": state["g"].float(), "energy": e.value}
    nb, dtype = state["nb"], state["dtype"]
    if kind == "device":
        es = nb.eforce_device(state["x"].data_ptr(), state["g"].data_ptr())
        with torch.cuda.stream(state["stream"]):      # before the handle's next evaluation writes it
            return {"dpot": state["g"].to(dtype), "energies": _energies(es, dtype)}
    if kind == "md":
        with torch.cuda.stream(state["stream"]):
            state["x"].copy_(state["x0"])
            state["v"].copy_(state["v0"])
            es, ek = nb.md_step(state["x"].data_ptr(), state["v"].data_ptr(), state["m"].data_ptr(), DT,
                                state["steps"])
            return {"x": state["x"].to(dtype), "v": state["v"].to(dtype), "energies": _energies(es, dtype),
                    "kinetic": ek}
    if kind == "adjoint":
        es = nb.adjoint_into(state["x"].numpy(), *(o.numpy() for o in state["out"]))
        return {"dq": state["out"][0].to(dtype), "deps": state["out"][1].to(dtype), "dsig": state["out"][2].to(dtype),
                "energies": _energies(es, dtype)}
    if kind == "pressure":
        _, es, press = nb.pressure(state["x"].numpy(), with_gradient=False)
        es, press = (es, press) if nb.batch else ([es], [press])
        return {"press": torch.from_numpy(np.stack(press)).to(dtype), "energies": _energies(es, dtype)}
    es = nb.eforce_into(state["x"].numpy(), state["g"].numpy())
    return {"dpot": state["g"].to(dtype), "energies": _energies(es, dtype)}


# ---- what a pass cannot do without ----------------------------------------------------


def _sizes(case):
    """(waters, other atoms, cutoff, grid points per side) of every replica."""
    if "solute_box" in case:
        f = (case["solute_box"] / HEAVY_BOX) ** 3
        big = case["solute_box"] == HEAVY_BOX
        w, o = (7020, 2496) if big else (int(5600 * f), max(60, int(2489 * f)) + 7)
        n = 64 if big else S.smooth_grid(case["solute_box"])
        return [(w, o, 9.0, n)] * case["copies"]
    out = []
    for n in _water_counts(case):
        box = 98.6 * (n / 32000) ** (1 / 3) if n > 24000 else (18.62 if n == 216 else (n / S.WATER_DENSITY) ** (1 / 3))
        out.append((n, 0, 10.0 if n > 24000 else 9.0, S.smooth_grid(box)))
    return out


def _pme_flops(atoms, n):
    # 64 grid points per atom, spread (weights and adds) and gathered (three derivatives); two
    # real transforms of the grid
    return atoms * 64 * 12 + 2 * 2.5 * n ** 3 * math.log2(n ** 3)


def work(case):
    """Coordinates (and velocities) read once, results written once; 50 operations per site pair
    inside the cutoff, the spline sums and the transforms."""
    if case["kind"] == "pme":
        return {"bytes": 56 * case["atoms"], "flops": _pme_flops(case["atoms"], _pme_grid(case))}
    atoms, flops = 0, 0.0
    for w, o, rc, n in _sizes(case):
        shell = S.WATER_DENSITY * 4.0 / 3.0 * math.pi * rc ** 3
        pairs = 9 * w * min(shell, w) / 2 + 3 * o * min(shell, w + o / 3)
        atoms += 3 * w + o
        flops += 50 * pairs + _pme_flops(3 * w + o, n)
    if case["kind"] == "md":
        return {"bytes": 104 * atoms, "flops": flops * case["steps"]}
    return {"bytes": 24 * atoms + {"eval": 24, "adjoint": 24, "pressure": 0}[case["kind"]] * atoms, "flops": flops}


# ---- the same in 64 bits, in plain torch ------------------------------------------------


def _erfc_pair(q, alpha, r2):
    """(energy, minus dE/dr / r) of q erfc(alpha r) / r."""
    r = r2.sqrt()
    e = q * torch.erfc(alpha * r) / r
    return e, (e + q * (2.0 * alpha / math.sqrt(math.pi)) * torch.exp(-alpha * alpha * r2)) / r2


class _Exact:
    """One system in 64 bits: the sums over its pairs, its exclusions and its grid."""

    def __init__(self, s):
        self.s = s
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, k=torch.float64: torch.as_tensor(a, device=self.dev).to(k)
        self.t, self.L = t, t(np.array(s.box))
        self.k = S.KOFDIE / s.eps
        self.q, self.e6, self.e12 = t(s.ptchg), t(s.epsgm6), t(s.epsgm12)
        mon0 = np.concatenate([[0], s.poipt[:-1]])
        self.o = t(mon0[s.montype == S.MON_WATER], torch.int64)
        water = np.zeros(s.npt, bool)
        for d in range(3):
            water[mon0[s.montype == S.MON_WATER] + d] = True
        self.rest = t(np.nonzero(~water)[0], torch.int64)
        self.is_water = t(water, torch.bool)
        self.rc2 = max(s.rvmx, s.relx) ** 2
        low = np.repeat(np.arange(s.npt), np.diff(s.exc1))
        self.ex_i, self.ex_j = t(low, torch.int64), t(s.exc2 - 1, torch.int64)

    def _image(self, d):
        n = torch.round(d / self.L)
        return d - n * self.L, (n != 0).any(-1)

    def forces(self, x, xrel=None, adjoint=False):
        """Gradient, the eleven energies, and with xrel (positions relative to the molecules'
        centres of mass) the pressure terms or with adjoint the parameter derivatives."""
        s, q, k, al = self.s, self.q, self.k, self.s.alpha
        self.x = x = self.t(x)
        self.g = torch.zeros_like(x)
        self.E = {name: 0.0 for name in NB.ENERGY_KEYS}
        self.vir = torch.zeros((4, 3), dtype=torch.float64, device=self.dev)      # LJ, direct, reciprocal, relative
        self.xrel = None if xrel is None else self.t(xrel)
        self.adj = torch.zeros((3, s.npt), dtype=torch.float64, device=self.dev) if adjoint else None
        if adjoint:
            eps, sig = S.lj_decode(s)
            self.eps, self.sig = self.t(eps), self.t(sig)
        self._water_pairs()
        self._other_pairs()
        i, j = self.ex_i, self.ex_j
        d = x[i] - x[j]
        r2 = (d * d).sum(1)
        r = r2.sqrt()
        qq, er = k * q[i] * q[j], torch.erf(al * r)
        self._add(i, j, d, (qq * (2 * al / math.sqrt(math.pi)) * torch.exp(-al * al * r2) - qq * er / r) / r2)
        self.E["e_corr"] = float(-(qq * er / r).sum())
        if adjoint:
            self._phi(i, j, -k * er / r)
        self._one_four()
        self._reciprocal()
        self.E["e_self"] = float(-al / math.sqrt(math.pi) * k * (q * q).sum())
        if adjoint:
            self.adj[0] -= 2.0 * al / math.sqrt(math.pi) * k * q
        E = self.E
        E["e_dir"] = E["e_el"] + E["e_lsym"]
        E["e_total"] = sum(v for n, v in E.items() if n not in ("e_total", "e_dir"))
        return self.g, torch.tensor([E[n] for n in NB.ENERGY_KEYS], dtype=torch.float64)

    def _add(self, i, j, d, mdf):
        """Pairs with separation d = x_i - x_j and minus dE/dr / r."""
        f = mdf[:, None] * d
        self.g.index_add_(0, i, -f)
        self.g.index_add_(0, j, f)

    def _phi(self, i, j, w):
        self.adj[0].index_add_(0, i, w * self.q[j])
        self.adj[0].index_add_(0, j, w * self.q[i])

    def _lj_adj(self, i, j, A, B):
        gsum = 6.0 * A - 3.0 * B
        for a, b in ((i, j), (j, i)):
            ea, sa = self.eps[a], self.sig[a]
            den = 0.5 * (sa + self.sig[b]) if self.s.arith else sa
            self.adj[1].index_add_(0, a, torch.where(ea > 0, (A - B) / (2.0 * ea.clamp_min(1e-300)), 0.0))
            self.adj[2].index_add_(0, a, torch.where(den > 0, gsum / den.clamp_min(1e-300), 0.0))

    def _split(self, near, far, e, img):
        self.E[near] += float(e[~img].sum())
        self.E[far] += float(e[img].sum())

    def _lj(self, i, j, r2):
        e12, e6 = self.e12[i] * self.e12[j], self.e6[i] * self.e6[j]
        if self.s.arith:
            s6 = (0.5 * (self.e6[i] + self.e6[j])) ** 6
            e12, e6 = e12 * s6 * s6, e12 * s6
        return e12 / r2 ** 6, e6 / r2 ** 3

    def _water_pairs(self):
        """Molecule pairs by the O-O distance, then all nine site pairs."""
        s, x, o = self.s, self.x, self.o
        n = o.numel()
        step = max(1, min(n, 20_000_000 // max(n, 1)))
        for i0 in range(0, n, step):
            oi = o[i0:i0 + step]
            d, _ = self._image(x[oi][:, None, :] - x[o][None, :, :])
            near = (d * d).sum(-1) <= self.rc2
            near &= torch.arange(n, device=self.dev)[None, :] > torch.arange(i0, i0 + oi.numel(), device=self.dev)[:, None]
            a, b = near.nonzero(as_tuple=True)
            del d, near
            i, j = oi[a], o[b]
            oo, img = self._image(x[i] - x[j])
            shift = oo - (x[i] - x[j])
            r2 = (oo * oo).sum(1)
            lj = r2 <= s.rvmx ** 2
            A, B = self._lj(i, j, r2)
            A, B = torch.where(lj, A, 0.0), torch.where(lj, B, 0.0)
            self._split("e_vdw", "e_vsym", A - B, img)
            m_lj = 6.0 * (2.0 * A - B) / r2
            self._add(i, j, oo, m_lj)
            if self.adj is not None:
                self._lj_adj(i, j, A, B)
            if self.xrel is not None:
                rm = oo - self.xrel[i] + self.xrel[j]
                self.vir[0] += (m_lj[:, None] * oo * rm).sum(0)
            for p in range(3):
                for w in range(3):
                    d = x[i + p] - x[j + w] + shift
                    e, mdf = _erfc_pair(self.k * self.q[i + p] * self.q[j + w], s.alpha, (d * d).sum(1))
                    self._split("e_el", "e_lsym", e, img)
                    self._add(i + p, j + w, d, mdf)
                    if self.adj is not None:
                        self._phi(i + p, j + w, e / (self.q[i + p] * self.q[j + w]))
                    if self.xrel is not None:
                        self.vir[1] += (mdf[:, None] * d * rm).sum(0)

    def _other_pairs(self):
        """Atoms outside waters with every other site, exclusions left out."""
        s, x = self.s, self.x
        rest, n = self.rest, s.npt
        if rest.numel() == 0:
            return
        gone = torch.sort(torch.minimum(self.ex_i, self.ex_j) * n + torch.maximum(self.ex_i, self.ex_j))[0]
        step = max(1, 20_000_000 // n)
        every = torch.arange(n, device=self.dev)
        for i0 in range(0, rest.numel(), step):
            ri = rest[i0:i0 + step]
            d, _ = self._image(x[ri][:, None, :] - x[None, :, :])
            near = (d * d).sum(-1) < self.rc2
            near &= self.is_water[None, :] | (every[None, :] > ri[:, None])
            a, j = near.nonzero(as_tuple=True)
            del d, near
            i = ri[a]
            key = torch.minimum(i, j) * n + torch.maximum(i, j)
            at = torch.searchsorted(gone, key).clamp_max(gone.numel() - 1)
            keep = gone[at] != key
            i, j = i[keep], j[keep]
            d, img = self._image(x[i] - x[j])
            r2 = (d * d).sum(1)
            lj = r2 < s.rvmx ** 2
            if s.hvdw0 and not s.arith:
                lj &= ~(((self.e12[i] < 1e-3) | (self.e12[j] < 1e-3)) & (r2 < s.relx ** 2))
            A, B = self._lj(i, j, r2)
            A, B = torch.where(lj, A, 0.0), torch.where(lj, B, 0.0)
            e, mdf = _erfc_pair(self.k * self.q[i] * self.q[j], s.alpha, r2)
            self._split("e_vdw", "e_vsym", A - B, img)
            self._split("e_el", "e_lsym", e, img)
            self._add(i, j, d, mdf + 6.0 * (2.0 * A - B) / r2)
            if self.adj is not None:
                self._lj_adj(i, j, A, B)
                self._phi(i, j, self.k * torch.erfc(s.alpha * r2.sqrt()) / r2.sqrt())

    def _one_four(self):
        s = self.s
        if len(s.spec1) == 0:
            return
        i, j = self.t(s.spec1 - 1, torch.int64), self.t(s.spec2 - 1, torch.int64)
        p = self.t(s.p14)
        d = self.x[i] - self.x[j]
        r2 = (d * d).sum(1)
        on = p[:, 0] > 1e-12
        A, B = torch.where(on, p[:, 0] / r2 ** 6, 0.0), torch.where(on, p[:, 1] / r2 ** 3, 0.0)
        e = p[:, 2] / r2.sqrt()
        self._add(i, j, d, (6.0 * (2.0 * A - B) + e) / r2)
        self.E["e_vdw14"], self.E["e_el14"] = float((A - B).sum()), float(e.sum())
        if self.adj is not None:
            self._lj_adj(i, j, A, B)
            self.adj[0].index_add_(0, i, e / self.q[i])
            self.adj[0].index_add_(0, j, e / self.q[j])

    def _reciprocal(self):
        s, al = self.s, self.s.alpha
        e, g, phi, rec = _pme64(self.x, self.q, s.box, s.nfft, al, self.k, self.t)
        self.E["e_ew_receip"] = e
        self.g += g
        self.vir[2] = rec
        if self.xrel is not None:
            self.vir[3] = -(g * self.xrel).sum(0)
        if self.adj is not None:
            self.adj[0] += phi


def _pme64(x, q, box, nfft, alpha, k, t):
    """Order-4 smooth PME: energy, gradient, potential per unit charge, diagonal virial."""
    n, fc = nfft, math.sqrt(k)
    idx, th, dth = [], [], []
    for d in range(3):
        w = x[:, d] / box[d]
        fr = n[d] * (w - torch.round(w) + 0.5)
        i = fr.floor()
        w = (fr - i)[:, None]
        m = 1.0 - w
        idx.append((i.to(torch.int64)[:, None] - 3 + torch.arange(4, device=x.device)) % n[d])
        th.append(torch.cat([m ** 3, 4 - 6 * w ** 2 + 3 * w ** 3, 1 + 3 * (w + w ** 2 - w ** 3), w ** 3], 1) / 6.0)
        dth.append(torch.cat([-m * m, w * (3 * w - 4), 1 + 2 * w - 3 * w * w, w * w], 1) / 2.0)
    at = ((idx[0][:, :, None, None] * n[1] + idx[1][:, None, :, None]) * n[2] + idx[2][:, None, None, :]).reshape(x.shape[0], 64)

    def weights(a, b, c):
        return (a[:, :, None, None] * b[:, None, :, None] * c[:, None, None, :]).reshape(x.shape[0], 64)

    grid = torch.zeros(n[0] * n[1] * n[2], dtype=torch.float64, device=x.device)
    grid.index_add_(0, at.reshape(-1), (fc * q[:, None] * weights(*th)).reshape(-1))
    F = torch.fft.fftn(grid.reshape(*n))
    msq, bmod, m2 = 0.0, 1.0, []
    for d in range(3):
        kk = torch.arange(n[d], device=x.device, dtype=torch.float64)
        m = torch.where(kk < (n[d] + 1) // 2, kk, kk - n[d]) / box[d]
        shape = [1, 1, 1]
        shape[d] = n[d]
        b = (2.0 / 3.0 + torch.cos(2.0 * math.pi * kk / n[d]) / 3.0) ** 2
        m2.append((m * m).reshape(shape))
        msq, bmod = msq + m2[d], bmod * b.reshape(shape)
    vol = box[0] * box[1] * box[2]
    safe = msq.clamp_min(1e-300)
    et = torch.exp(-(math.pi / alpha) ** 2 * msq) / (math.pi * vol * bmod * safe)
    et[0, 0, 0] = 0.0
    em = et * (F.real ** 2 + F.imag ** 2)
    rec = torch.stack([0.5 * (em * (1.0 - 2.0 * (1.0 + (math.pi / alpha) ** 2 * msq) * m2[d] / safe)).sum() for d in range(3)])
    pot = (torch.fft.ifftn(et * F).real * (n[0] * n[1] * n[2])).reshape(-1)[at]
    g = torch.stack([(n[0] / box[0]) * (pot * weights(dth[0], th[1], th[2])).sum(1),
                     (n[1] / box[1]) * (pot * weights(th[0], dth[1], th[2])).sum(1),
                     (n[2] / box[2]) * (pot * weights(th[0], th[1], dth[2])).sum(1)], 1)
    return float(0.5 * em.sum()), fc * q[:, None] * g, fc * (pot * weights(*th)).sum(1), rec


def _rigid(p0, p1, doh, dhh, m):
    """p1 (waters, 3, 3) moved along the constraint directions of p0 until the three distances
    hold (the solution SHAKE converges to), by Newton steps on the three multipliers."""
    pairs, dist = ((0, 1), (0, 2), (1, 2)), (doh, doh, dhh)
    d0 = torch.stack([p0[:, a] - p0[:, b] for a, b in pairs], 1)
    lam = torch.zeros(p0.shape[0], 3, dtype=torch.float64, device=p0.device)
    sgn = torch.zeros(3, 3, dtype=torch.float64, device=p0.device)     # atom a's share of constraint k
    for k, (a, b) in enumerate(pairs):
        sgn[a, k], sgn[b, k] = 1.0 / m[a], -1.0 / m[b]
    for _ in range(12):
        p = p1 + torch.einsum("ak,wk,wkd->wad", sgn, lam, d0)
        J = torch.empty(p.shape[0], 3, 3, dtype=torch.float64, device=p.device)
        r = torch.empty_like(lam)
        for k, (a, b) in enumerate(pairs):
            d = p[:, a] - p[:, b]
            r[:, k] = (d * d).sum(1) - dist[k] ** 2
            for c in range(3):
                J[:, k, c] = 2.0 * (sgn[a, c] - sgn[b, c]) * (d * d0[:, c]).sum(1)
        lam = lam - torch.linalg.solve(J, r)
    return p1 + torch.einsum("ak,wk,wkd->wad", sgn, lam, d0)


def _exact_md(case, systems, seed):
    m3 = np.array([S.MASS_O, S.MASS_H, S.MASS_H])
    dhh = 2.0 * S.TIP3_ROH * math.sin(math.radians(S.TIP3_HOH_DEG) / 2.0)
    xs, vs, es, kin = [], [], [], 0.0
    for s in systems:
        X = _Exact(s)
        x, v, m = X.t(s.coor), X.t(_velocities(s, seed)), X.t(_masses(s.nwaters))[:, None]
        for _ in range(case["steps"]):
            g, e = X.forces(x)
            free = x + DT * (v - DT * ACCEL * g / m)
            new = _rigid(x.reshape(-1, 3, 3), free.reshape(-1, 3, 3), S.TIP3_ROH, dhh, m3).reshape(-1, 3)
            v, x = (new - x) / DT, new
        xs.append(x.cpu())
        vs.append(v.cpu())
        es.append(e)
        kin += float(0.5 * (m * v * v).sum()) / ACCEL
    return {"x": torch.cat(xs), "v": torch.cat(vs), "energies": torch.stack(es), "kinetic": kin}


def exact(case, seed):
    kind = case["kind"]
    if kind == "pme":
        x, q = _pme_inputs(case, seed)
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a: torch.as_tensor(a, dtype=torch.float64, device=dev)
        e, g, _, _ = _pme64(t(x), t(q), (case["box"],) * 3, (_pme_grid(case),) * 3, 0.35, S.KOFDIE, t)
        return {"dpot": g.cpu(), "energy": e}
    systems = _systems(case, seed)
    if kind == "md":
        if case["steps"] * sum(s.npt for s in systems) > 2_500_000:
            return None
        return _exact_md(case, systems, seed)
    if kind == "eval":
        got = [_Exact(s).forces(s.coor) for s in systems]
        return {"dpot": torch.cat([g.cpu() for g, _ in got]), "energies": torch.stack([e for _, e in got])}
    out, es = [], []
    for s in systems:
        X = _Exact(s)
        if kind == "adjoint":
            _, e = X.forces(s.coor, adjoint=True)
            out.append(X.adj.cpu())
        else:
            xyz, m = s.coor.reshape(-1, 3, 3), np.array([S.MASS_O, S.MASS_H, S.MASS_H])[:, None]
            _, e = X.forces(s.coor, xrel=(xyz - ((m * xyz).sum(1) / m.sum())[:, None, :]).reshape(-1, 3))
            out.append(X.vir.reshape(-1).cpu())
        es.append(e)
    if kind == "adjoint":
        a = torch.cat(out, dim=1)
        return {"dq": a[0], "deps": a[1], "dsig": a[2], "energies": torch.stack(es)}
    return {"press": torch.stack(out), "energies": torch.stack(es)}
