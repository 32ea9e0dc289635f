"""Timed cases: the calls a program makes on this library, over the sizes it is used at.

Families (key "family" of a case):

  eval     Engine.evaluate in mixed precision: positions in, list rebuilt,
           forces and energies out.  Host arrays (a host MD code calling the
           library every step) or device arrays (a program that keeps its
           atoms on the GPU: set positions, build, compute, read forces).
  batch    the same on many independent boxes in one engine (replica
           ensembles, screening).
  md_water rigid-water dynamics with the Berendsen thermostat, 1 fs steps,
           constraints, displacement-triggered rebuilds; a pass is one md_run
           and the trajectory frame a program writes after it.
  md_chain flexible six-atom chains: every bonded kind and SPME in the step.
  fp64     the plain FP64 form on host arrays (reference-quality forces; the
           all-pairs list builder in small boxes, link cells in large ones).
  dropin   MDBas's own calls on MDBas's arrays, in the library's default
           (FP64) mode: makelist at a step where the list is due, then energy.
  spme     the smooth particle-mesh reciprocal sum on host arrays.
  ewald    the explicit reciprocal Ewald sum on host arrays.
  grad     energy and forces as a differentiable function (parameter fitting
           by force matching): forward and backward.

Sizes are the ones of this repository's configurations and tests: 3,000,
18,558, 96,000 and 999,999 atoms of rigid water at 0.0334 molecules/A^3, 64
replicas of 1,500 to 30,000 atoms, a 12,000-atom charged LJ fluid in a 50 A
box, a 128^3 grid at order 8 for the 98.6 A box.  All potentials are cut-off
12 A, switch 10 A, skin 2 A, alpha 0.34 / A.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from mdbas_b200 import grad, nb, systems

RC, RON, ALPHA = systems.POTENTIAL["cutOff"], systems.POTENTIAL["cutOn"], systems.POTENTIAL["alpha"]
CC = systems.CHARGE_CONST
PREC = 1e-6           # relative precision of the reciprocal sums (MDBas's rule for the m-range)
LJ_DENSITY = 12000 / 50.0 ** 3


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # one small solvated molecule's worth of water, called every step from
        # a host code: latency and launches count
        {"name": "eval_3k_host", "family": "eval", "n": 3000, "arrays": "host"},
        # the headline box, called from a host code
        {"name": "eval_96k_host", "family": "eval", "n": 96000, "arrays": "host"},
        # the largest box, atoms resident on the GPU
        {"name": "eval_1m_device", "family": "eval", "n": 999999, "arrays": "device"},
        # a replica ensemble of ragged sizes in one engine
        {"name": "batch_64", "family": "batch", "count": 64},
        # production dynamics of the headline box
        {"name": "md_water_96k", "family": "md_water", "n": 96000, "steps": 40},
        # flexible molecules with full electrostatics
        {"name": "md_chain_10k", "family": "md_chain", "side": 12, "steps": 40},
        # reference-quality forces: a small box (all-pairs list) and the
        # headline box (link cells)
        {"name": "fp64_3k", "family": "fp64", "n": 3000},
        {"name": "fp64_96k", "family": "fp64", "n": 96000},
        # MDBas itself with this library linked in, a step where the list is due
        {"name": "dropin_18k", "family": "dropin", "n": 18558},
        # reciprocal space of the headline box, and explicit for a small one
        {"name": "spme_96k", "family": "spme", "n": 96000, "order": 8},
        {"name": "ewald_3k", "family": "ewald", "n": 3000},
        # one force-matching gradient step
        {"name": "grad_12k", "family": "grad", "n": 12000},
    ]


def _log_int(rng, lo, hi, step=1):
    return step * int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step))


def draw(rng):
    family = rng.choice(["eval", "eval", "eval", "batch", "md_water", "md_chain", "fp64", "fp64",
                         "dropin", "spme", "ewald", "grad"])
    case = {"family": family}
    if family == "eval":
        case["n"] = _log_int(rng, 2000, 400000, 3)
        case["arrays"] = rng.choice(["host", "device"])
    elif family == "batch":
        case["count"] = rng.randint(3, 64)
    elif family == "md_water":
        case["n"] = _log_int(rng, 3000, 96000, 3)
        case["steps"] = rng.choice([20, 40])
    elif family == "md_chain":
        case["side"] = rng.randint(5, 13)
        case["steps"] = rng.choice([20, 40])
    elif family == "fp64":
        case["n"] = _log_int(rng, 2000, 96000, 3)
    elif family == "dropin":
        case["n"] = _log_int(rng, 3000, 30000, 3)
    elif family == "spme":
        case["n"] = _log_int(rng, 2000, 96000, 3)
        case["order"] = rng.choice([4, 6, 8])
    elif family == "ewald":
        case["n"] = _log_int(rng, 1500, 9000, 3)
    else:
        case["n"] = rng.randint(6000, 16000)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _edge(n):
    """Edge of the water box of n atoms; the named sizes keep their named boxes."""
    return {3000: 31.0, 96000: 98.6, 999999: 215.0}.get(
        n, (n / 3 / systems.WATER_DENSITY) ** (1.0 / 3.0))


def _water(n, seed, temperature=None):
    return systems.water_box(n // 3, _edge(n), seed=seed, temperature=temperature)


def _replicas(count, seed):
    """The ensemble's boxes: the sizes of the 64-replica configuration."""
    sizes = systems.replica_sizes(count, seed=1)
    return systems.concat([systems.water_box_for_atoms(k, seed=1000 * seed + i)
                           for i, k in enumerate(sizes)])


def _water_excl(n):
    """Exclusion rows of rigid water, both directions (start[n+1], flat)."""
    base = 3 * (np.arange(n, dtype=np.int32) // 3)
    own = np.arange(n, dtype=np.int32) - base
    flat = np.stack([base + (own == 0), base + 2 - (own == 2)], 1).astype(np.int32)
    return 2 * np.arange(n + 1, dtype=np.int32), flat.reshape(-1)


def _lj(n, seed):
    """Charged LJ fluid at the density of the 12,000-atom box: a jittered
    lattice, atoms dealt to its sites at random."""
    rng = np.random.default_rng(seed)
    box = (n / LJ_DENSITY) ** (1.0 / 3.0)
    m = math.ceil(round(n ** (1.0 / 3.0), 9))
    sp = box / m
    site = rng.permutation(m ** 3)[:n]
    idx = np.stack([site % m, (site // m) % m, site // (m * m)], 1)
    pos = (idx + 0.5) * sp - 0.5 * box + rng.uniform(-0.08, 0.08, size=(n, 3))
    types = rng.integers(0, 4, size=n).astype(np.int32)
    t_eps, t_sig = rng.uniform(0.05, 0.3, size=4), rng.uniform(2.8, 3.8, size=4)
    q = rng.uniform(-0.8, 0.8, size=n)
    q -= q.mean()
    e2, e3 = np.zeros((0, 2), np.int32), np.zeros((0, 3), np.int32)
    return systems.System("lj", box, pos[:, 0].copy(), pos[:, 1].copy(), pos[:, 2].copy(), q,
                          np.sqrt(t_eps[types] * systems.KCAL_TO_IU), 0.5 * t_sig[types],
                          np.full(n, 39.948), e2, e3, types=types, type_eps_kcal=t_eps,
                          type_sigma=t_sig)


def _m_max(box):
    """m-range of MDBas's precision rule for a box width."""
    tol = math.sqrt(abs(math.log(PREC * RC)))
    tol1 = math.sqrt(-math.log(PREC * RC * (2.0 * tol * ALPHA) ** 2))
    return int(0.25 + box * ALPHA * tol1 / math.pi + 0.5)


def _grid(box):
    p = 1
    while _m_max(box) > p and p < 256:
        p *= 2
    return 2 * p


def _dev():
    return torch.device("cuda", torch.cuda.current_device())


def _dev_arrays(*arrays):
    return [torch.from_numpy(np.ascontiguousarray(a)).to(_dev()) for a in arrays]


def prepare(case, seed):
    f = case["family"]
    st = {"family": f}
    if f in ("eval", "fp64"):
        s = _water(case["n"], seed)
        st["engine"] = nb.Engine(s, precision=1 if f == "eval" else 0,
                                 exclusions=_water_excl(s.n), **systems.POTENTIAL)
        if case.get("arrays") == "device":
            st["pos"] = _dev_arrays(s.x, s.y, s.z)
            st["force"] = [torch.zeros(s.n, dtype=torch.float64, device=_dev()) for _ in range(3)]
            st["family"] = "device"
        else:
            st["pos"] = [s.x, s.y, s.z]
            st["force"] = [np.zeros(s.n) for _ in range(3)]
    elif f == "batch":
        s = _replicas(case["count"], seed)
        st["engine"] = nb.Engine(s, precision=1, exclusions=_water_excl(s.n), **systems.POTENTIAL)
        st["pos"] = _dev_arrays(s.x, s.y, s.z)
        st["force"] = [torch.zeros(s.n, dtype=torch.float64, device=_dev()) for _ in range(3)]
        st["family"] = "device"
    elif f == "md_water":
        s = _water(case["n"], seed, temperature=300.0)
        e = nb.Engine(s, precision=1, exclusions=_water_excl(s.n), **systems.POTENTIAL)
        cons = s.water_constraints()
        # the lattice start settles before the production step is used
        e.md_init(s.mass, (s.vx, s.vy, s.vz), time_step=0.0005, constraints=cons)
        e.md_run(200, target_temp=300.0, tau_t=0.05)
        vel = e.velocities()
        e.md_init(s.mass, vel, time_step=0.001, constraints=cons)
        st.update(engine=e, steps=case["steps"], bath=(300.0, 0.1))
    elif f == "md_chain":
        side = case["side"]
        s = systems.flexible_chains(side, 6.5 * side, seed=seed, temperature=300.0)
        e = nb.Engine(s, precision=1, **systems.POTENTIAL)
        e.set_bonded(s.meta["bonded"])
        m = _grid(s.box)
        e.set_kspace(2, (m, m, m), 6)
        e.md_init(s.mass, (s.vx, s.vy, s.vz), time_step=0.0005)
        st.update(engine=e, steps=case["steps"], bath=(0.0, 0.0))
    elif f == "dropin":
        st["md"] = _Mdbas(_water(case["n"], seed))
    elif f == "spme":
        s = _water(case["n"], seed)
        m = _grid(s.box)
        st.update(system=s, grid=(m, m, m), order=case["order"])
    elif f == "ewald":
        s = _water(case["n"], seed)
        m = _m_max(s.box)
        st.update(system=s, mmax=(m, m, m))
    else:
        s = _lj(case["n"], seed)
        rng = np.random.default_rng(seed + 1)
        pos = np.stack([s.x, s.y, s.z], 1)
        st["model"] = grad.RealSpaceModel(s, s.types)
        st["args"] = [torch.from_numpy(a).requires_grad_() for a in
                      (pos, s.q.copy(), s.type_eps_kcal.copy(), s.type_sigma.copy())]
        # upstream gradients of a force-matching loss
        st["up"] = (torch.tensor(0.01, dtype=torch.float64),
                    torch.from_numpy(rng.normal(size=(s.n, 3))))
    return st


class _Mdbas:
    """The structs and arrays MDBas holds when it calls the library: built as
    its main program does, lists allocated by the first makelist."""

    def __init__(self, s):
        self.lib = nb.bind_dropin()
        n = self.n = s.n
        self.ctrl, self.neigh, self.ewald, self.ener = nb.CTRL(), nb.NEIGH(), nb.EWALD(), nb.ENERGY()
        self.ctrl.newjob, self.ctrl.keyEwald = 1, 3  # 3: real space alone
        self.ctrl.elecType, self.ctrl.vdwType = nb.FULL, nb.VSWITCH
        self.neigh.update, self.neigh.linkRatio = 1, 1
        self.ewald.alpha = ALPHA
        self.param = nb.make_param(n, RC, RON, systems.POTENTIAL["delr"])
        self.param.nBond, self.param.nAngle = len(s.bonds), len(s.angles)
        self.box = nb.make_pbc(s.cell())
        self.bond, self.angle = (nb.BOND * len(s.bonds))(), (nb.ANGLE * len(s.angles))()
        for t, (a, b) in zip(self.bond, s.bonds.tolist()):
            t.a, t.b = a, b
        for t, (a, b, c) in zip(self.angle, s.angles.tolist()):
            t.a, t.b, t.c = a, b, c
        self.none = (nb.DIHE * 1)()
        self.const = (nb.CONSTRAINT * 1)()
        self.pos = [np.ascontiguousarray(a, dtype=np.float64).copy() for a in (s.x, s.y, s.z)]
        self.vel = [np.zeros(n) for _ in range(3)]
        self.force = [np.zeros(n) for _ in range(3)]
        self.pot = [np.ascontiguousarray(a, dtype=np.float64) for a in (s.q, s.eps, s.sig)]
        self.frozen = np.zeros(n, np.int32)
        ip = C.POINTER(C.c_int)
        self.list, self.pair, self.order, self.list14 = ip(), ip(), ip(), ip()
        self.excl, self.excl_pair = C.POINTER(ip)(), ip()
        self.makelist()
        # room for the list at any configuration of this density, so that no
        # step has to grow it
        libc = C.CDLL(None)
        libc.calloc.restype, libc.calloc.argtypes = C.c_void_p, [C.c_size_t, C.c_size_t]
        libc.free.argtypes = [C.c_void_p]
        libc.free(C.cast(self.list, C.c_void_p))
        self.room = 640 * n
        self.list = C.cast(libc.calloc(self.room, 4), ip)
        self.neigh.sizeList = self.room
        # rigid molecules: the bonds define the exclusions and carry no energy
        self.rigid = nb.PARAM.from_buffer_copy(self.param)
        self.rigid.nBond = self.rigid.nAngle = 0

    def makelist(self):
        r = C.byref
        self.lib.makelist(r(self.ctrl), r(self.param), r(self.box), r(self.neigh), self.const,
                          self.bond, self.angle, self.none, self.none,
                          *(nb.as_dp(a) for a in self.pos), nb.as_ip(self.frozen), r(self.list),
                          r(self.pair), r(self.order), r(self.list14), r(self.excl),
                          r(self.excl_pair))

    def energy(self):
        r = C.byref
        q, eps, sig = (nb.as_dp(a) for a in self.pot)
        self.lib.init_energy_ptrs(r(self.ctrl))
        self.lib.energy(r(self.ctrl), r(self.rigid), r(self.ener), r(self.ewald), r(self.box),
                        r(self.neigh), self.bond, self.bond, self.angle, self.none, self.none,
                        *(nb.as_dp(a) for a in self.pos), *(nb.as_dp(a) for a in self.vel),
                        *(nb.as_dp(a) for a in self.force), q, eps, sig, eps, sig,
                        nb.as_ip(self.frozen), self.list, self.pair, self.order, self.list14,
                        self.excl, self.excl_pair)

    def view(self, ptr, n):
        """n ints of MDBas's memory as an array that keeps this owner alive."""
        buf = (C.c_int * n).from_address(C.addressof(ptr.contents))
        buf.owner = self
        return np.frombuffer(buf, dtype=np.int32)

    def __del__(self):
        libc = C.CDLL(None)
        libc.free.argtypes = [C.c_void_p]
        rows = self.n if self.ctrl.keyLink else self.n - 1
        for p in [self.excl[i] for i in range(rows)] + [self.excl, self.excl_pair, self.list,
                                                        self.pair, self.order, self.list14]:
            libc.free(C.cast(p, C.c_void_p))


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    f = state["family"]
    if f in ("eval", "fp64"):
        e = state["engine"].evaluate(*state["pos"], *state["force"])
        return {"force": state["force"], "energy": e}
    if f == "device":
        eng = state["engine"]
        eng.set_positions_device(*(t.data_ptr() for t in state["pos"]))
        eng.build()
        eng.compute()
        eng.forces_device(*(t.data_ptr() for t in state["force"]))
        return {"force": state["force"], "energy": eng.energies()}
    if f in ("md_water", "md_chain"):
        eng, bath = state["engine"], state["bath"]
        rows = eng.md_run(state["steps"], energy_every=10, target_temp=bath[0], tau_t=bath[1])
        return {"rows": rows, "pos": eng.positions(), "vel": eng.velocities()}
    if f == "dropin":
        m = state["md"]
        m.makelist()
        m.energy()
        e = m.ener
        return {"force": m.force, "energy": [e.elec, e.vdw, e.virelec, e.virvdw],
                "pair": m.view(m.pair, m.n), "order": m.view(m.order, m.n),
                "list": m.view(m.list, m.room)}
    if f == "spme":
        e, fx, fy, fz, v = nb.spme(state["system"], ALPHA, state["grid"], state["order"])
        return {"energy": e, "force": [fx, fy, fz], "virial": v}
    if f == "ewald":
        e, fx, fy, fz, v, stress = nb.ewald_rec(state["system"], ALPHA, state["mmax"])
        return {"energy": e, "force": [fx, fy, fz], "virial": v, "stress": stress}
    pos, q, eps_t, sig_t = state["args"]
    energy, force = state["model"](pos, q, eps_t, sig_t)
    grads = torch.autograd.grad((energy, force), (pos, q, eps_t, sig_t), state["up"])
    return {"energy": energy.detach(), "force": force.detach(), "grads": list(grads)}


def _sizes(case):
    """(atoms, steps in a pass) of a case."""
    f = case["family"]
    if f == "batch":
        return sum(systems.replica_sizes(case["count"], seed=1)), 1
    if f == "md_chain":
        return 6 * case["side"] ** 3, case["steps"]
    return case["n"], case.get("steps", 1)


def work(case):
    f = case["family"]
    n, steps = _sizes(case)
    if f == "md_chain":
        density = 6 / 6.5 ** 3
    else:
        density = LJ_DENSITY if f == "grad" else 3 * systems.WATER_DENSITY
    pairs = 0.5 * n * density * 4.0 / 3.0 * math.pi * RC ** 3
    listed_pairs = pairs * ((RC + systems.POTENTIAL["delr"]) / RC) ** 3
    if f in ("md_water", "md_chain"):
        # per step: positions, velocities and forces read and written, the
        # parameters read; 77 operations per pair
        w = {"bytes": steps * n * 8 * (2 * 9 + 3), "flops": steps * pairs * 77}
        if f == "md_chain":
            m = _grid(6.5 * case["side"])
            w["flops"] += steps * (10 * m ** 3 * math.log2(m ** 3) + n * 6 ** 3 * 8)
        return w
    if f == "spme":
        m = _grid(_edge(n))
        p = case["order"]
        # two complex transforms, spreading and interpolation
        return {"bytes": n * 8 * 7,
                "flops": 10 * m ** 3 * math.log2(m ** 3) + n * p ** 3 * 8}
    if f == "ewald":
        m = _m_max(_edge(n))
        k = 2.0 / 3.0 * math.pi * (1.05 * m) ** 3
        return {"bytes": n * 8 * 7, "flops": n * k * (14 + 16)}
    w = {"bytes": n * 8 * 9, "flops": pairs * 77}
    if f == "dropin":
        w["bytes"] += listed_pairs * 4 + n * 8
    if f == "grad":
        # forward, the backward's own evaluation and the adjoint
        w = {"bytes": n * 8 * 20, "flops": pairs * (77 + 200)}
    return w


# ---------------------------------------------------------------------------
# The same results in plain 64-bit torch
# ---------------------------------------------------------------------------
def _pairs(pos, box, excl_of):
    """In-cut-off pairs i < j (minimum image) and which of them are excluded."""
    n = pos.shape[0]
    ii, jj = [], []
    chunk = max(1, (1 << 26) // n)
    idx = torch.arange(n, device=pos.device)
    for lo in range(0, n, chunk):
        hi = min(n, lo + chunk)
        r2 = torch.zeros(hi - lo, n - lo, dtype=torch.float64, device=pos.device)
        for k in range(3):
            d = pos[None, lo:, k] - pos[lo:hi, None, k]
            d -= box * torch.round(d / box)
            r2 += d * d
        keep = (r2 <= RC * RC) & (idx[None, lo:] > idx[lo:hi, None])
        a, b = keep.nonzero(as_tuple=True)
        ii.append(a + lo)
        jj.append(b + lo)
    i, j = torch.cat(ii), torch.cat(jj)
    ex = excl_of(i, j)
    return i[~ex], j[~ex]


def _switch(r2):
    a, b = RC * RC, RON * RON
    sw = (a - r2) ** 2 * (a + 2 * r2 - 3 * b) / (a - b) ** 3
    dsw = 12 * r2 * (a - r2) * (b - r2) / (a - b) ** 3  # r dS/dr
    inner = r2 <= b
    return torch.where(inner, 1.0, sw), torch.where(inner, 0.0, dsw)


def _real_space(pos, box, q, eps, sig, excl):
    """Forces (n, 3) and energy terms of the real-space sum; excl: (m, 2)
    excluded pairs."""
    n = pos.shape[0]
    key = torch.sort(excl[:, 0] * n + excl[:, 1])[0] if len(excl) else None

    def excl_of(i, j):
        if key is None:
            return torch.zeros_like(i, dtype=torch.bool)
        k = i * n + j
        at = torch.searchsorted(key, k).clamp(max=len(key) - 1)
        return key[at] == k

    force = torch.zeros_like(pos)
    g0 = 2 * ALPHA / math.sqrt(math.pi)

    def add(i, j, d, s):
        f = s[:, None] * d
        force.index_add_(0, i, f)
        force.index_add_(0, j, -f)

    def disp(i, j):
        d = pos[j] - pos[i]
        d = d - box * torch.round(d / box)
        r2 = (d * d).sum(1)
        return d, r2, torch.sqrt(r2)

    i, j = _pairs(pos, box, excl_of)
    out = {"elec_direct": 0.0, "vdw": 0.0, "vir_direct": 0.0, "vir_vdw": 0.0, "elec_corr": 0.0,
           "vir_corr": 0.0, "n_pairs": float(len(i))}
    for lo in range(0, len(i), 1 << 23):
        a, b = i[lo:lo + (1 << 23)], j[lo:lo + (1 << 23)]
        d, r2, r = disp(a, b)
        qq = CC * q[a] * q[b]
        e = qq * torch.special.erfc(ALPHA * r) / r
        re = -(e + qq * g0 * torch.exp(-(ALPHA * r) ** 2))  # r dE/dr
        s6 = ((sig[a] + sig[b]) / r) ** 6
        ve = eps[a] * eps[b]
        p, rp = 4 * ve * (s6 * s6 - s6), 24 * ve * (s6 - 2 * s6 * s6)
        sw, dsw = _switch(r2)
        rv = rp * sw + p * dsw
        add(a, b, d, (re + rv) / r2)
        out["elec_direct"] += float(e.sum())
        out["vdw"] += float((p * sw).sum())
        out["vir_direct"] += float(re.sum())
        out["vir_vdw"] += float(rv.sum())
    if len(excl):
        a, b = excl[:, 0], excl[:, 1]
        d, r2, r = disp(a, b)
        qq = CC * q[a] * q[b]
        e = -qq * torch.special.erf(ALPHA * r) / r
        re = -(e + qq * g0 * torch.exp(-(ALPHA * r) ** 2))
        add(a, b, d, re / r2)
        out["elec_corr"], out["vir_corr"] = float(e.sum()), float(re.sum())
    out["elec_self"] = float(-CC * ALPHA / math.sqrt(math.pi) * (q * q).sum())
    return force, out


def _water_pairs(n, device):
    o = 3 * torch.arange(n // 3, device=device)
    return torch.cat([torch.stack([o, o + 1], 1), torch.stack([o, o + 2], 1),
                      torch.stack([o + 1, o + 2], 1)])


def _exact_water(s):
    pos = torch.stack(_dev_arrays(s.x, s.y, s.z), 1)
    return _real_space(pos, s.box, *_dev_arrays(s.q, s.eps, s.sig),
                       _water_pairs(s.n, pos.device))


def _columns(f):
    return [f[:, k].cpu().numpy().copy() for k in range(3)]


def _with_tail(erec, s, stress, f1):
    """Energy and stress of a reciprocal sum with the self and non-neutral terms."""
    q = s.q
    self_e = -CC * ALPHA * float((q * q).sum()) / math.sqrt(math.pi)
    non = -0.5 * math.pi * CC * (float(q.sum()) / ALPHA) ** 2 / s.box ** 3
    st = [f1 * v for v in stress]
    for k in (0, 3, 5):
        st[k] += f1 * erec + non
    return f1 * erec + self_e + non, -(st[0] + st[3] + st[5]), st


def _bspline(s, p):
    """Cardinal B-splines of order p at s - j and their derivatives, j < p."""
    fr = s - torch.floor(s)
    b = [fr, 1.0 - fr] + [torch.zeros_like(fr)] * (p - 2)
    d = list(b)
    for k in range(2, p):
        if k == p - 1:
            d = [b[0]] + [b[j] - b[j - 1] for j in range(1, p)]
        new = list(b)
        for j in range(k, 0, -1):
            new[j] = ((fr + j) * b[j] + (k + 1 - fr - j) * b[j - 1]) / k
        new[0] = fr * b[0] / k
        b = new
    if p == 2:
        d = [torch.ones_like(fr), -torch.ones_like(fr)]
    return torch.stack(b, 1), torch.stack(d, 1)


def _moduli(m, p, device):
    b = torch.zeros(p, dtype=torch.float64)
    b[1] = 1.0
    for k in range(2, p):
        for j in range(k, 0, -1):
            b[j] = (j * b[j] + (k + 1 - j) * b[j - 1]) / k
        b[0] = 0.0
    w = torch.arange(m, dtype=torch.float64)[:, None] * torch.arange(p - 1)[None, :]
    c = (b[1:][None, :] * torch.exp(2j * math.pi * w / m)).sum(1)
    return (1.0 / (c.real ** 2 + c.imag ** 2)).to(device)


def _exact_spme(s, m, p):
    pos = torch.stack(_dev_arrays(s.x, s.y, s.z), 1)
    q, = _dev_arrays(s.q)
    u = m * (pos / s.box + 0.5)
    b, d, at = [], [], []
    for k in range(3):
        bk, dk = _bspline(u[:, k], p)
        b.append(bk)
        d.append(dk)
        at.append((torch.floor(u[:, k]).long()[:, None] - torch.arange(p, device=q.device)) % m)
    grid = torch.zeros(m ** 3, dtype=torch.float64, device=q.device)
    cells = []
    for i in range(p):
        for j in range(p):
            cell = ((at[0][:, i] * m + at[1][:, j]) * m)[:, None] + at[2]
            cells.append(cell)
            w = (q * b[0][:, i] * b[1][:, j])[:, None] * b[2]
            grid.index_add_(0, cell.reshape(-1), w.reshape(-1))
    k = torch.arange(m, device=q.device, dtype=torch.float64)
    k = torch.where(k > m // 2, k - m, k) * (2 * math.pi / s.box)
    kx, ky, kz = k[:, None, None], k[None, :, None], k[None, None, :]
    k2 = kx * kx + ky * ky + kz * kz
    rc2 = (m / s.box * 1.05 * 2 * math.pi) ** 2
    ok = (k2 > 2.220446049250313e-16) & (k2 <= rc2)
    k2s = torch.where(ok, k2, 1.0)
    bm = _moduli(m, p, q.device)
    ra = -0.25 / ALPHA ** 2
    infl = torch.where(ok, bm[:, None, None] * bm[None, :, None] * bm[None, None, :]
                       * torch.exp(ra * k2s) / k2s, 0.0)
    ft = torch.fft.fftn(grid.view(m, m, m))
    vam = 2.0 * (1.0 / k2s - ra) * infl * (ft.real ** 2 + ft.imag ** 2)
    ks = (kx, ky, kz)
    stress = [-float((vam * ks[a] * ks[c]).sum()) for a in range(3) for c in range(a, 3)]
    conv = torch.fft.ifftn(infl * ft).real.reshape(-1) * m ** 3
    erec = float((conv * grid).sum())
    g = torch.zeros_like(pos)
    for i in range(p):
        for j in range(p):
            v = conv[cells[i * p + j]]
            sb, sd = (v * b[2]).sum(1), (v * d[2]).sum(1)
            g[:, 0] += d[0][:, i] * b[1][:, j] * sb
            g[:, 1] += b[0][:, i] * d[1][:, j] * sb
            g[:, 2] += b[0][:, i] * b[1][:, j] * sd
    f1 = 2 * math.pi / s.box ** 3 * CC
    force = -2.0 * f1 * q[:, None] * g * (m / s.box)
    force -= force.mean(0)
    e, v, _ = _with_tail(erec, s, stress, f1)
    return {"energy": e, "force": _columns(force), "virial": v}


def _exact_ewald(s, m):
    pos = torch.stack(_dev_arrays(s.x, s.y, s.z), 1)
    q, = _dev_arrays(s.q)
    r = torch.arange(-m, m + 1, device=q.device)
    k = torch.stack(torch.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
    half = (k[:, 0] > 0) | ((k[:, 0] == 0) & ((k[:, 1] > 0) | ((k[:, 1] == 0) & (k[:, 2] > 0))))
    k = k[half].double() * (2 * math.pi / s.box)
    k2 = (k * k).sum(1)
    k = k[k2 <= (m / s.box * 1.05 * 2 * math.pi) ** 2]
    k2 = (k * k).sum(1)
    ra = -0.25 / ALPHA ** 2
    a = torch.exp(ra * k2) / k2
    f1 = 2 * (2 * math.pi / s.box ** 3) * CC
    force = torch.zeros_like(pos)
    sc, ss = torch.zeros_like(k2), torch.zeros_like(k2)
    step = 1024
    for lo in range(0, len(k), step):
        ph = k[lo:lo + step] @ pos.T
        c, sn = torch.cos(ph), torch.sin(ph)
        sc[lo:lo + step], ss[lo:lo + step] = c @ q, sn @ q
        de = a[lo:lo + step, None] * (sn * sc[lo:lo + step, None] - c * ss[lo:lo + step, None])
        force += (de.T @ k[lo:lo + step]) * q[:, None]
    s2 = sc * sc + ss * ss
    vam = 2.0 * a * (1.0 / k2 - ra) * s2
    stress = [-float((vam * k[:, x] * k[:, y]).sum()) for x in range(3) for y in range(x, 3)]
    e, v, st = _with_tail(float((a * s2).sum()), s, stress, f1)
    return {"energy": e, "force": _columns(2 * f1 * force), "virial": v, "stress": st}


def _exact_grad(s, seed):
    rng = np.random.default_rng(seed + 1)
    pos0 = torch.stack(_dev_arrays(s.x, s.y, s.z), 1)
    i, j = _pairs(pos0, s.box, lambda a, b: torch.zeros_like(a, dtype=torch.bool))
    args = [t.requires_grad_() for t in
            [pos0.clone()] + _dev_arrays(s.q, s.type_eps_kcal, s.type_sigma)]
    pos, q, eps_t, sig_t = args
    types = torch.as_tensor(s.types, device=pos.device).long()
    eps, sig = torch.sqrt(eps_t[types] * systems.KCAL_TO_IU), 0.5 * sig_t[types]
    d = pos[j] - pos[i]
    d = d - s.box * torch.round(d / s.box)
    r2 = (d * d).sum(1)
    r = torch.sqrt(r2)
    e = (CC * q[i] * q[j] * torch.special.erfc(ALPHA * r) / r).sum()
    s6 = ((sig[i] + sig[j]) / r) ** 6
    e = e + (4 * eps[i] * eps[j] * (s6 * s6 - s6) * _switch(r2)[0]).sum()
    e = e - CC * ALPHA / math.sqrt(math.pi) * (q * q).sum()
    f = -torch.autograd.grad(e, pos, create_graph=True)[0]
    up_e = torch.tensor(0.01, dtype=torch.float64, device=pos.device)
    up_f, = _dev_arrays(rng.normal(size=(s.n, 3)))
    g = torch.autograd.grad((e, f), args, (up_e, up_f))
    return {"energy": e.detach().cpu(), "force": f.detach().cpu(), "grads": [t.cpu() for t in g]}


def exact(case, seed):
    f = case["family"]
    if f in ("eval", "fp64"):
        if case["n"] > 200000:
            return None
        force, e = _exact_water(_water(case["n"], seed))
        return {"force": _columns(force), "energy": e}
    if f == "batch":
        s = _replicas(case["count"], seed)
        forces, energy = [], {}
        for r in range(case["count"]):
            force, e = _exact_water(systems.replica(s, r))
            forces.append(force)
            for k, v in e.items():
                energy[k] = energy.get(k, 0.0) + v
        return {"force": _columns(torch.cat(forces)), "energy": energy}
    if f == "dropin":
        force, e = _exact_water(_water(case["n"], seed))
        return {"force": _columns(force), "pair": None, "list": None, "order": None,
                "energy": [e["elec_direct"] + e["elec_corr"], e["vdw"],
                           e["vir_direct"] + e["vir_corr"], e["vir_vdw"]]}
    if f == "spme":
        s = _water(case["n"], seed)
        return _exact_spme(s, _grid(s.box), case["order"])
    if f == "ewald":
        s = _water(case["n"], seed)
        return _exact_ewald(s, _m_max(s.box))
    if f == "grad":
        return _exact_grad(_lj(case["n"], seed), seed)
    return None  # dynamics: the rounding of one step travels through the next
