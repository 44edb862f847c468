"""Performance cases of the force path, through the entry points that a
simulation calls: p3mx_forces and p3mx_dp3m_compute on device arrays (the C
ABI a host code binds), System.integrator / System.analysis on host arrays
(scripts), and p3mx_batch_run (many replicas).

A case is a dict of plain values; `prepare` builds its inputs and handles from
a seed, `run` makes one pass, `exact` gives the same outputs in FP64 torch
(the P3M sums written out: same mesh, order, alpha and cutoffs).
"""
import ctypes
import math

import numpy as np
import torch

from espresso_b200 import System, _lib
from espresso_b200.electrostatics import P3M, P3MGPU

ACCURACY = 1e-4
SKIN = 0.4
FENE = dict(k=30.0, r_max=1.5)
DP = ctypes.POINTER(ctypes.c_double)
IP = ctypes.POINTER(ctypes.c_int)


# --- the cases --------------------------------------------------------------

def _ions(name, n, mesh, cao, **kw):
    """Salt or melt system of p3mx_forces: n particles at `density` in a box
    of edge ratios 1 : ay : az, LJ (cutoff 2.5) or WCA, FP32-mixed (P3MGPU)
    or FP64 (P3M); chain > 0: a bead-spring melt with WCA and FENE bonds;
    gap > 0: a slab with the layer correction."""
    mx, my, mz = (mesh, mesh, mesh) if isinstance(mesh, int) else mesh
    c = dict(name=name, kind="forces", n=n, mx=mx, my=my, mz=mz, cao=cao, ay=1.0, az=1.0,
             density=0.5, r_cut=3.5, mixed=True, wca=False, chain=0, gap=0.0, jitter=0.1)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest production run: 2000 ions, where launches and latency count
        _ions("ions_2k_mixed", 2000, 32, 5, density=0.25, r_cut=3.0, wca=True),
        # an oblong box with an odd particle number, ragged bricks and FFT
        # lengths that are no powers of two, at a low assignment order
        _ions("ions_23k_mixed_oblong", 23457, (56, 70, 48), 4, ay=1.25, az=0.85, r_cut=3.9, wca=True),
        # an everyday size on a power-of-two mesh
        _ions("ions_131k_mixed", 131072, 128, 7, wca=True),
        # the benchmark's size: 2^20 ions on a 256^3 mesh, LJ (at this density
        # and jitter no pair lies within rounding of the LJ cutoff)
        _ions("ions_1m_mixed", 1 << 20, 256, 7, density=0.417, jitter=0.05),
        # the same path in plain FP64 (the P3M actor)
        _ions("ions_131k_double", 131072, 120, 6, mixed=False),
        # polyelectrolyte melt: two particle types, WCA, FENE bonds, dense
        _ions("melt_250k_mixed", 250000, 128, 6, density=0.85, r_cut=3.85, wca=True, chain=250),
        # slab between vacuum gaps: P3M plus the layer correction
        _ions("slab_98k_mixed_elc", 98304, (112, 112, 144), 7, az=1.3, gap=14.0, density=0.4,
              wca=True),
        # dipolar P3M, forces and torques, the default FP64 actor
        dict(name="dipoles_16k_double", kind="dipoles", n=16384, mesh=56, cao=7, r_cut=4.7,
             alpha=0.718, mixed=False),
        # ... and its FP32 path at the benchmark's size
        dict(name="dipoles_131k_mixed", kind="dipoles", n=131072, mesh=96, cao=7, r_cut=5.2,
             alpha=0.64, mixed=True),
        # a script's MD run: velocity Verlet on host arrays, lists rebuilt as
        # the particles move
        dict(name="md_12k_system", kind="md", n=12000, mesh=54, cao=5, density=0.4, r_cut=3.6,
             mixed=True, wca=True, steps=10),
        # analysis of stored frames: every frame is a new configuration
        # (forces, energy and pressure tensor of each)
        dict(name="frames_60k_system", kind="frames", n=60000, mesh=90, cao=6, density=0.45,
             r_cut=3.6, mixed=True, wca=True, frames=2),
        # many small systems at once: 48 replicas, Langevin steps in one graph
        dict(name="batch_48_mixed", kind="batch", replicas=48, nmin=1000, nmax=16000, cao=7,
             mesh_max=64, mixed=True, steps=20),
    ]


def _log(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def _mesh(length, spacing):
    """Even FFT length with factors 2, 3, 5, 7 near length / spacing."""
    def smooth(m):
        for p in (2, 3, 5, 7):
            while m % p == 0:
                m //= p
        return m == 1
    m = max(16, 2 * int(length / spacing / 2))
    while not smooth(m):
        m += 2
    return m


def draw(rng):
    # FP32-mixed draws take WCA: the truncated LJ force jumps at its cutoff,
    # and a pair within rounding of it may fall on either side
    kind = rng.choice(["forces"] * 6 + ["dipoles", "dipoles", "md", "frames", "batch"])
    mixed = rng.random() < 0.7
    if kind == "batch":
        return dict(kind=kind, replicas=rng.randint(3, 48), nmin=1000,
                    nmax=_log(rng, 2000, 16000), cao=rng.randint(5, 7), mesh_max=64, mixed=mixed,
                    steps=rng.randint(3, 20))
    cao = rng.randint(3, 7)
    h = rng.uniform(0.5, 0.7)
    if kind == "dipoles":
        n = _log(rng, 3000, 131072 if mixed else 60000)
        mesh = _mesh((n / 0.5) ** (1 / 3), max(h, 0.56))
        return dict(kind=kind, n=n, mesh=mesh, cao=max(cao, 4), r_cut=round(rng.uniform(4, 5.4), 2),
                    alpha=round(rng.uniform(0.6, 0.75), 3), mixed=mixed)
    density = round(rng.uniform(0.3, 0.55), 3)
    r_cut = round(rng.uniform(3.0, 4.2), 2)
    if kind in ("md", "frames"):
        n = _log(rng, 2500, 25000 if kind == "md" else 80000)
        c = dict(kind=kind, n=n, mesh=_mesh((n / density) ** (1 / 3), h), cao=cao,
                 density=density, r_cut=r_cut, mixed=mixed, wca=mixed or rng.random() < 0.4)
        c["steps" if kind == "md" else "frames"] = rng.randint(2, 10 if kind == "md" else 3)
        return c
    form = rng.choice(["salt", "salt", "salt", "melt", "slab"])
    n = _log(rng, 5000 if form == "slab" else 2000, 900000 if mixed and form == "salt" else 200000)
    kw = dict(mixed=mixed, density=density, r_cut=r_cut, ay=round(rng.uniform(0.9, 1.3), 2),
              az=round(rng.uniform(0.9, 1.3), 2), wca=mixed or rng.random() < 0.4)
    if form == "melt":
        kw.update(density=0.85, wca=True, chain=rng.choice([20, 50, 100, 250]))
    elif form == "slab":
        kw.update(gap=round(rng.uniform(8, 14), 1), az=round(rng.uniform(1.2, 1.5), 2))
    c = _ions(None, n, 0, cao, **kw)
    del c["name"]
    c["mx"], c["my"], c["mz"] = (_mesh(b, h) for b in _box(c))
    return c


# --- systems ------------------------------------------------------------------

def _box(c):
    """Box edges; a slab's particles fill the part below the gap."""
    ay, az = c.get("ay", 1.0), c.get("az", 1.0)
    a = (c["n"] / c.get("density", 0.5) / (ay * az)) ** (1.0 / 3.0)
    return [a, a * ay, a * az + c.get("gap", 0.0)]


def _alpha(n_charged, r_cut, box):
    """The splitting parameter at which the real-space error estimate takes
    its share of ACCURACY (unit charges, prefactor 1)."""
    rs = 2.0 * n_charged / math.sqrt(n_charged * r_cut * box[0] * box[1] * box[2])
    return math.sqrt(math.log(math.sqrt(2.0) * rs / ACCURACY)) / r_cut


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gen(seed):
    return torch.Generator(device=_device()).manual_seed(int(seed) * 7919 + 11)


def _sites(n, box, jitter, g, order=None):
    """n places of a jittered lattice that fills the box, in random order or
    in the serpentine order `order` picks from."""
    a = (box[0] * box[1] * box[2] / n) ** (1.0 / 3.0)
    m = [max(1, round(b / a)) for b in box]
    while m[0] * m[1] * m[2] < n:
        k = max(range(3), key=lambda d: box[d] / m[d])
        m[k] += 1
    total = m[0] * m[1] * m[2]
    k = torch.randperm(total, generator=g, device=g.device)[:n] if order is None else order(total, g)
    z, row = k // (m[0] * m[1]), k // m[0]
    y, x = row % m[1], k % m[0]
    if order is not None:  # boustrophedon: consecutive indices are neighbours
        y = torch.where(z % 2 == 0, y, m[1] - 1 - y)
        x = torch.where(row % 2 == 0, x, m[0] - 1 - x)
    cell = torch.tensor([box[d] / m[d] for d in range(3)], dtype=torch.float64, device=g.device)
    p = (torch.stack([x, y, z], 1).double() + 0.5) * cell
    return p + (torch.rand(p.shape, generator=g, dtype=torch.float64, device=g.device) - 0.5) * 2 * jitter


def _system(c, seed):
    """Positions, charges, types, bonds (i, j) and box of an ion case."""
    g, box, n = _gen(seed), _box(c), c["n"]
    dev = g.device
    if c.get("chain"):
        nch = int(0.5 * n / c["chain"])
        nb = nch * c["chain"]

        def order(total, g):
            seg = torch.randperm(total // c["chain"], generator=g, device=dev)[:nch]
            beads = (seg[:, None] * c["chain"] + torch.arange(c["chain"], device=dev)).reshape(-1)
            free = torch.ones(total, dtype=torch.bool, device=dev)
            free[beads] = False
            free = free.nonzero()[:, 0]
            free = free[torch.randperm(len(free), generator=g, device=dev)[:n - nb]]
            return torch.cat([beads, free])
        pos = _sites(n, box, 0.05, g, order)
        k = torch.arange(nb, device=dev)
        bead_q = torch.where((k % c["chain"]) % 2 == 0, -1.0, 0.0).double()
        n_ion = n - nb
        ion_q = torch.where(torch.arange(n_ion, device=dev) % 2 == 0, 1.0, -1.0).double()
        missing = int(round(-float(bead_q.sum()) - float(ion_q.sum())))
        flip = (ion_q < 0).nonzero()[:missing // 2, 0]  # counterions of the chains
        ion_q[flip] = 1.0
        if missing % 2:
            ion_q[-2 if n_ion % 2 else -1] += 1.0
        q = torch.cat([bead_q, ion_q])
        types = torch.cat([torch.zeros(nb), torch.ones(n_ion)]).to(dev, torch.int32)
        first = k.view(nch, -1)
        bonds = torch.stack([first[:, :-1].reshape(-1), first[:, 1:].reshape(-1)], 1)
    else:
        slab = [box[0], box[1], box[2] - c.get("gap", 0.0)]
        pos = _sites(n, slab, c.get("jitter", 0.1), g)
        q = torch.where(torch.arange(n, device=dev) % 2 == 0, 1.0, -1.0).double()
        if n % 2:
            q[-1] = 0.0  # an odd particle number: one neutral particle
        types = torch.zeros(n, dtype=torch.int32, device=dev)
        bonds = torch.zeros((0, 2), dtype=torch.long, device=dev)
    return pos, q, types, bonds, box


def _charged(q):
    return float((q * q).sum())


class _Handle:
    """Owner of a C handle."""

    def __init__(self, ptr, free):
        self.ptr, self._free = ptr, free

    def __del__(self):
        self._free(self.ptr)


def _dbl(a):
    return a.ctypes.data_as(DP)


def _pair_table(c, ntypes):
    tab = (_lib.PairParams * (ntypes * ntypes))()
    for e in tab:
        if c.get("wca"):
            e.wca_eps, e.wca_sig = 1.0, 1.0
        else:
            e.lj_eps, e.lj_sig, e.lj_cut = 1.0, 1.0, 2.5
            e.lj_shift = -((1 / 2.5) ** 12 - (1 / 2.5) ** 6)
    return tab


def _desc(box):
    s = _lib.SystemDesc()
    for d in range(3):
        s.box[d], s.periodic[d] = box[d], 1
    s.skin = SKIN
    return s


# --- prepare and run, by kind -------------------------------------------------

def _prepare_forces(c, seed):
    lib = _lib.load()
    pos, q, types, bonds, box = _system(c, seed)
    p = _lib.Params()
    p.prefactor, p.accuracy, p.cao, p.r_cut = 1.0, ACCURACY, c["cao"], c["r_cut"]
    p.alpha = _alpha(_charged(q), c["r_cut"], box)
    for d in range(3):
        p.mesh[d], p.mesh_off[d] = (c["mx"], c["my"], c["mz"])[d], -1.0
    p.single_precision, p.check_neutrality = int(c["mixed"]), 1
    p.charge_neutrality_tolerance = 2e-12
    ptr = ctypes.c_void_p()
    _lib.check(lib.p3mx_create(ctypes.byref(p), ctypes.byref(ptr)))
    h = _Handle(ptr, lib.p3mx_destroy)
    torch.cuda.current_stream().synchronize()
    _lib.check(lib.p3mx_set_system(ptr, ctypes.byref(_desc(box))), ptr)
    _lib.check(lib.p3mx_activate(ptr, c["n"], _lib.dptr(pos), _lib.dptr(q), _lib.P3MX_DEVICE_PTRS), ptr)
    nt = 2 if c["chain"] else 1
    _lib.check(lib.p3mx_set_pair_params(ptr, nt, _pair_table(c, nt)), ptr)
    if len(bonds):
        fene = (_lib.BondParams * 1)(_lib.BondParams(_lib.P3MX_BOND_FENE, FENE["k"], 0.0, FENE["r_max"]))
        trip = torch.cat([torch.zeros_like(bonds[:, :1]), bonds], 1).to(torch.int32).cpu().numpy()
        trip = np.ascontiguousarray(trip)
        _lib.check(lib.p3mx_set_bonds(ptr, 1, fene, len(trip), trip.ctypes.data_as(IP)), ptr)
    if c["gap"]:
        e = _lib.ElcParams()
        e.maxPWerror, e.gap_size, e.far_cut, e.neutralize = ACCURACY, c["gap"], -1.0, 1
        _lib.check(lib.p3mx_set_elc(ptr, ctypes.byref(e)), ptr)
    return dict(h=h, pos=pos, q=q, types=types, f=torch.zeros_like(pos), n=c["n"])


def _run_forces(s):
    lib, ptr = _lib.load(), s["h"].ptr
    flags = _lib.P3MX_DEVICE_PTRS | _lib.P3MX_FORCES | _lib.P3MX_OVERWRITE
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.p3mx_forces(ptr, s["n"], _lib.dptr(s["pos"]), _lib.dptr(s["q"]),
                               _lib.dptr(s["types"]), _lib.dptr(s["f"]), None, None, flags, stream), ptr)
    return s["f"]


def _dipoles(c, seed):
    g, n = _gen(seed), c["n"]
    edge = (n / 0.5) ** (1.0 / 3.0)
    pos = _sites(n, [edge] * 3, 0.2, g)
    mu = torch.randn((n, 3), generator=g, dtype=torch.float64, device=g.device)
    return pos, mu / mu.norm(dim=1, keepdim=True), edge


def _prepare_dipoles(c, seed):
    lib = _lib.load()
    pos, mu, edge = _dipoles(c, seed)
    p = _lib.Dp3mParams()
    p.prefactor, p.accuracy, p.cao, p.r_cut, p.alpha = 1.0, ACCURACY, c["cao"], c["r_cut"], c["alpha"]
    for d in range(3):
        p.mesh[d], p.mesh_off[d] = c["mesh"], -1.0
    p.timings, p.single_precision = 10, int(c["mixed"])
    ptr = ctypes.c_void_p()
    _lib.check(lib.p3mx_dp3m_create(ctypes.byref(p), ctypes.byref(ptr)), ptr, lib.p3mx_dp3m_last_error)
    h = _Handle(ptr, lib.p3mx_dp3m_destroy)
    torch.cuda.current_stream().synchronize()
    _lib.check(lib.p3mx_dp3m_set_system(ptr, ctypes.byref(_desc([edge] * 3))), ptr, lib.p3mx_dp3m_last_error)
    _lib.check(lib.p3mx_dp3m_activate(ptr, c["n"], _lib.dptr(pos), _lib.dptr(mu), _lib.P3MX_DEVICE_PTRS),
               ptr, lib.p3mx_dp3m_last_error)
    return dict(h=h, pos=pos, mu=mu, f=torch.zeros_like(pos), t=torch.zeros_like(pos), n=c["n"])


def _run_dipoles(s):
    lib, ptr = _lib.load(), s["h"].ptr
    flags = _lib.P3MX_DEVICE_PTRS | _lib.P3MX_FORCES | _lib.P3MX_OVERWRITE
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(lib.p3mx_dp3m_compute(ptr, s["n"], _lib.dptr(s["pos"]), _lib.dptr(s["mu"]),
                                     _lib.dptr(s["f"]), _lib.dptr(s["t"]), None, flags, stream),
               ptr, lib.p3mx_dp3m_last_error)
    return {"force": s["f"], "torque": s["t"]}


def _script_system(c, pos, q, v=None):
    box = _box(c)
    s = System(box_l=box)
    s.time_step = 0.005
    s.cell_system.skin = SKIN
    s.part.add(pos=pos, q=q, v=v)
    ia = s.non_bonded_inter[0, 0]
    if c["wca"]:
        ia.wca.set_params(epsilon=1.0, sigma=1.0)
    else:
        ia.lennard_jones.set_params(epsilon=1.0, sigma=1.0, cutoff=2.5, shift="auto")
    s.electrostatics.solver = (P3MGPU if c["mixed"] else P3M)(
        prefactor=1.0, accuracy=ACCURACY, mesh=c["mesh"], cao=c["cao"], r_cut=c["r_cut"],
        alpha=_alpha(float((q * q).sum()), c["r_cut"], box), tune=False, verbose=False)
    return s


def _script_inputs(c, seed):
    pos, q, _, _, _ = _system(c, seed)
    g = _gen(seed + 1)
    v = torch.randn(pos.shape, generator=g, dtype=torch.float64, device=g.device)
    return pos, q, v


def _prepare_md(c, seed):
    pos, q, v = (x.cpu().numpy() for x in _script_inputs(c, seed))
    return dict(s=_script_system(c, pos, q, v), steps=c["steps"])


def _run_md(st):
    s = st["s"]
    s.integrator.run(st["steps"])
    p = s.part.all()
    return {"pos": p.pos, "v": p.v, "f": p.f}


def _frame_list(c, seed):
    return [_system(c, seed * 31 + k)[0] for k in range(c["frames"])]


def _prepare_frames(c, seed):
    frames = [x.cpu().numpy() for x in _frame_list(c, seed)]
    q = _system(c, seed)[1].cpu().numpy()
    return dict(s=_script_system(c, frames[0], q), frames=frames)


def _run_frames(st):
    s, out = st["s"], []
    for x in st["frames"]:
        s.part.all().pos = x
        s.integrator.run(0)
        e, p = s.analysis.energy(), s.analysis.pressure_tensor()
        out.append({"f": s.part.all().f, "energy": np.array([e["coulomb"], e["non_bonded"]]),
                    "pressure": p["coulomb"] + p["non_bonded"]})
    return out


def _prepare_batch(c, seed):
    lib = _lib.load()
    rng = np.random.default_rng(seed)
    box, pref, off, pos, q = [], [], [0], [], []
    g = _gen(seed)
    for r in range(c["replicas"]):
        # sizes spread over the range alike for every seed
        t = (r + 0.5) / c["replicas"]
        n = int(math.exp((1 - t) * math.log(c["nmin"]) + t * math.log(c["nmax"]))) // 2 * 2
        edge = (n / 0.3) ** (1.0 / 3.0)
        box.append([edge] * 3)
        pref.append(0.5 + 3.5 * ((r * 0.618034) % 1.0))
        off.append(off[-1] + n)
        pos.append(_sites(n, [edge] * 3, 0.1, g).cpu().numpy())
        q.append(rng.permutation(np.repeat([1.0, -1.0], n // 2)) * (1 + r % 2))
    box, pref, off = np.array(box), np.array(pref), np.array(off, dtype=np.int64)
    pos, q = np.ascontiguousarray(np.vstack(pos)), np.concatenate(q)
    d = _lib.BatchDesc()
    d.n_rep, d.box, d.prefactor = c["replicas"], _dbl(box), _dbl(pref)
    d.offset = off.ctypes.data_as(ctypes.POINTER(ctypes.c_longlong))
    d.accuracy, d.skin, d.single_precision = ACCURACY * 10, 0.8, int(c["mixed"])
    d.mesh_min, d.mesh_max, d.cao_min, d.cao_max = 16, c["mesh_max"], c["cao"], c["cao"]
    types = np.zeros(len(q), dtype=np.int32)
    ptr = ctypes.c_void_p()
    _lib.check(lib.p3mx_batch_create(ctypes.byref(d), _dbl(pos), _dbl(q), types.ctypes.data_as(IP), 1,
                                     _pair_table(dict(wca=True), 1), ctypes.byref(ptr)),
               ptr, lib.p3mx_batch_last_error)
    h = _Handle(ptr, lib.p3mx_batch_destroy)
    return dict(h=h, n=len(q), steps=c["steps"], seed=seed % 1000 + 1)


def _run_batch(s):
    """A sampling interval: Langevin steps, then the state is read."""
    lib, ptr = _lib.load(), s["h"].ptr
    _lib.check(lib.p3mx_batch_run(ptr, s["steps"], 0.005, 1.0, 1.0, s["seed"]),
               ptr, lib.p3mx_batch_last_error)
    pos, f, v = (np.empty((s["n"], 3)) for _ in range(3))
    _lib.check(lib.p3mx_batch_get(ptr, _dbl(pos), _dbl(f), _dbl(v)), ptr, lib.p3mx_batch_last_error)
    return {"pos": pos, "f": f, "v": v}


def prepare(case, seed):
    s = globals()["_prepare_" + case["kind"]](case, seed)
    s["kind"] = case["kind"]
    return s


def run(state):
    return globals()["_run_" + state["kind"]](state)


# --- work and tolerance ---------------------------------------------------------

def _evaluation(n, points, cao, r_cut, density, fields=4, assigned=1):
    """Operations of one evaluation: pairs once, stencil terms, transforms."""
    pairs = 0.5 * n * 4.18879 * r_cut ** 3 * density
    return 45.0 * pairs + 2.0 * (assigned + 3 * fields / 4) * n * cao ** 3 + \
        2.5 * (fields + assigned - 1) * points * math.log2(points)


def work(case):
    """Each input read once and each output written once; the operations of
    the P3M sums."""
    c = case
    if c["kind"] == "batch":
        t = [(r + 0.5) / c["replicas"] for r in range(c["replicas"])]
        ns = [c["nmin"] ** (1 - x) * c["nmax"] ** x for x in t]
        n = sum(ns)
        one = sum(_evaluation(k, (k / 0.3) * 4.0, c["cao"], 3.5, 0.3) for k in ns)
        return {"bytes": 72.0 * n + 72.0 * n, "flops": c["steps"] * one}
    n = c["n"]
    if c["kind"] == "dipoles":
        return {"bytes": 96.0 * n, "flops": 2 * _evaluation(n, c["mesh"] ** 3, c["cao"], c["r_cut"], 0.5, 9, 3)}
    mesh = c["mesh"] ** 3 if "mesh" in c else c["mx"] * c["my"] * c["mz"]
    one = _evaluation(n, mesh, c["cao"], c["r_cut"], c["density"])
    if c["kind"] == "md":
        return {"bytes": 132.0 * n, "flops": (c["steps"] + 1) * one}
    if c["kind"] == "frames":
        return {"bytes": c["frames"] * 60.0 * n, "flops": c["frames"] * 2 * one}
    return {"bytes": 60.0 * n, "flops": one}


def tolerance(case):
    """About four times what the paths show against `exact` (the batch: what
    its FP32-mixed and FP64 runs differ by)."""
    if not case["mixed"]:
        # energies and pressures are sums of cancelling terms
        return {"rel": 4e-10, "max": 4e-9} if case["kind"] == "frames" else {"rel": 4e-12, "max": 2e-11}
    return {"rel": 1.2e-5, "max": 1.2e-4}


# --- the same sums in FP64 torch ---------------------------------------------------

def _spline(f, p):
    """M_p(f + k), k = 0 .. p-1, of the cardinal B-spline of order p, for f in
    [0, 1): the recursion on the order."""
    m = [torch.ones_like(f)]
    for n in range(2, p + 1):
        new = []
        for k in range(n):
            a = m[k] if k < n - 1 else 0.0
            b = m[k - 1] if k > 0 else 0.0
            new.append(((f + k) * a + (n - f - k) * b) / (n - 1))
        m = new
    return m


class _Mesh:
    """Assignment to, and interpolation from, a periodic mesh whose points lie
    half a spacing off the box corner."""

    def __init__(self, pos, box, mesh, cao):
        self.mesh, self.cao = mesh, cao
        shift = math.floor((cao - 1) / 2.0) - (cao % 2) / 2.0
        self.i, self.w = [], []
        for d in range(3):
            u = pos[:, d] * (mesh[d] / box[d]) - 0.5 - shift
            c = torch.floor(u)
            m = _spline(u - c, cao)
            self.w.append([m[cao - 1 - k] for k in range(cao)])
            self.i.append([(c.long() + k) % mesh[d] for k in range(cao)])

    def terms(self):
        for a in range(self.cao):
            for b in range(self.cao):
                row = (self.i[0][a] * self.mesh[1] + self.i[1][b]) * self.mesh[2]
                wab = self.w[0][a] * self.w[1][b]
                for k in range(self.cao):
                    yield row + self.i[2][k], wab * self.w[2][k]

    def assign(self, q):
        rho = torch.zeros(self.mesh[0] * self.mesh[1] * self.mesh[2], dtype=torch.float64, device=q.device)
        for idx, w in self.terms():
            rho.index_add_(0, idx, q * w)
        return rho.view(*self.mesh)

    def interpolate(self, fields):
        out = [0.0] * len(fields)
        flat = [x.reshape(-1) for x in fields]
        for idx, w in self.terms():
            out = [o + w * x[idx] for o, x in zip(out, flat)]
        return torch.stack(out, 1)


def _index(m, dev, half=False, dop=False):
    """Signed mesh indices (M/2 -> -M/2), or of the derivative (M/2 -> 0)."""
    k = torch.arange(m // 2 + 1 if half else m, device=dev, dtype=torch.float64)
    k = torch.where(k < m // 2, k, k - m)
    return torch.where(k == -(m // 2), torch.zeros_like(k), k) if dop else k


def _axes(mesh, dev, dop):
    return [_index(m, dev, d == 2, dop).view([-1 if e == d else 1 for e in range(3)])
            for d, m in enumerate(mesh)]


def _all_half(mesh, dev):
    z = [(torch.arange(m // 2 + 1 if d == 2 else m, device=dev) % (m // 2) == 0).view(
        [-1 if e == d else 1 for e in range(3)]) for d, m in enumerate(mesh)]
    return z[0] & z[1] & z[2]


def _u2(n, mesh, cao):
    u = 1.0
    for d in range(3):
        u = u * torch.sinc(n[d] / mesh[d])
    return u ** (2 * cao)


def _kspace(pos, q, box, mesh, cao, alpha, observables=False):
    dev, vol = pos.device, box[0] * box[1] * box[2]
    m = _Mesh(pos, box, mesh, cao)
    rho = torch.fft.rfftn(m.assign(q))
    n = _axes(mesh, dev, False)
    k2 = sum((n[d] * (2 * math.pi / box[d])) ** 2 for d in range(3))
    k2[0, 0, 0] = 1.0
    ex = k2 / (4 * alpha * alpha)
    g = torch.where(ex < 30, torch.exp(-ex) * 4 * math.pi / k2 / _u2(n, mesh, cao), 0.0)
    g = torch.where(_all_half(mesh, dev), 0.0, g)
    kd = [x * (2 * math.pi / box[d]) for d, x in enumerate(_axes(mesh, dev, True))]
    size = mesh[0] * mesh[1] * mesh[2]
    fields = [torch.fft.irfftn(1j * k * (g * rho), s=mesh) * size for k in kd]
    f = -q[:, None] * m.interpolate(fields) / vol
    if not observables:
        return f
    wgt = torch.full((mesh[2] // 2 + 1,), 2.0, dtype=torch.float64, device=dev)
    wgt[0] = wgt[-1] = 1.0
    ek = wgt * g * (rho.real ** 2 + rho.imag ** 2)
    sq, sq2 = float(q.sum()), float((q * q).sum())
    e = float(ek.sum()) / (2 * vol) - sq2 * alpha / math.sqrt(math.pi) - \
        sq * sq * math.pi / (2 * vol * alpha * alpha)
    nsq = sum(k * k for k in kd) + torch.zeros_like(g)
    on = nsq != 0
    pr = torch.where(on, ek * -2.0 * (1 / torch.where(on, nsq, 1.0) + 1 / (4 * alpha * alpha)), 0.0)
    vir = torch.stack([torch.stack([(pr * kd[a] * kd[b]).sum() for b in range(3)]) for a in range(3)])
    vir = vir + torch.eye(3, dtype=torch.float64, device=dev) * torch.where(on, ek, 0.0).sum()
    return f, e, vir / (2 * vol)


def _over_pairs(pos, box, r_cut, term, width):
    """Per particle, the sum over its neighbours within r_cut of
    term(i, j, d, r) (width values, d = x_i - x_j): cells of edge >= r_cut."""
    dev, n = pos.device, len(pos)
    g = [max(3, min(64, int(b / r_cut))) for b in box]
    edge = torch.tensor(box, dtype=torch.float64, device=dev)
    gt = torch.tensor(g, device=dev)
    x = pos - torch.floor(pos / edge) * edge
    c3 = torch.minimum((x / edge * gt).long(), gt - 1)
    cell = (c3[:, 0] * g[1] + c3[:, 1]) * g[2] + c3[:, 2]
    ncell = g[0] * g[1] * g[2]
    order = torch.argsort(cell, stable=True)
    cnt = torch.bincount(cell, minlength=ncell)
    start = torch.cumsum(cnt, 0) - cnt
    m = int(cnt.max())
    table = torch.full((ncell, m), -1, dtype=torch.long, device=dev)
    table[cell[order], torch.arange(n, device=dev) - start[cell[order]]] = order
    out = torch.zeros((n, width), dtype=torch.float64, device=dev)
    step = max(1, (1 << 21) // (m * m))
    for c0 in range(0, ncell, step):
        a = torch.arange(c0, min(ncell, c0 + step), device=dev)
        ia = table[a]
        xa = x[ia]
        ax = [a // (g[1] * g[2]), a // g[2] % g[1], a % g[2]]
        total = torch.zeros((len(a), m, width), dtype=torch.float64, device=dev)
        for o in range(27):
            nb = [ax[0] + o // 9 - 1, ax[1] + o // 3 % 3 - 1, ax[2] + o % 3 - 1]
            wrap = torch.stack([torch.div(nb[d], g[d], rounding_mode="floor") for d in range(3)], 1)
            nb = [nb[d] % g[d] for d in range(3)]
            ib = table[(nb[0] * g[1] + nb[1]) * g[2] + nb[2]]
            d = xa[:, :, None, :] - (x[ib] + (wrap * edge)[:, None, :])[:, None, :, :]
            r2 = (d * d).sum(-1)
            ok = (ia[:, :, None] >= 0) & (ib[:, None, :] >= 0) & (r2 < r_cut * r_cut) & (r2 > 0)
            at = ok.nonzero(as_tuple=True)
            i, j, dv = ia[at[0], at[1]], ib[at[0], at[2]], d[at]
            total.view(-1, width).index_add_(0, at[0] * m + at[1], term(i, j, dv, r2[at].sqrt()))
        live = ia >= 0
        out[ia[live]] = total[live]
    return out


def _coulomb_part(alpha, r):
    """exp(-(alpha r)^2) and erfc(alpha r) / exp of the real-space kernel:
    Abramowitz & Stegun 7.1.26, which the path evaluates by definition."""
    t = 1.0 / (1.0 + 0.3275911 * alpha * r)
    poly = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429))))
    return torch.exp(-(alpha * r) ** 2), poly


def _short(pos, q, box, c, alpha, observables=False):
    """Real-space Coulomb plus LJ or WCA."""
    wca, rc = c.get("wca", False), c["r_cut"]
    lj_cut = 2 ** (1 / 6) if wca else 2.5
    shift = 0.25 if wca else -((1 / 2.5) ** 12 - (1 / 2.5) ** 6)

    def term(i, j, d, r):
        ex, poly = _coulomb_part(alpha, r)
        qq = torch.where(r < rc, q[i] * q[j], 0.0)
        fc = qq * ex * (poly / r + 2 * alpha / math.sqrt(math.pi)) / (r * r)
        s6 = r ** -6
        on = r < lj_cut
        fn = torch.where(on, 48 * s6 * (s6 - 0.5) / (r * r), 0.0)
        f = (fc + fn)[:, None] * d
        if not observables:
            return f
        ec = qq * poly / r * ex
        en = torch.where(on, 4 * (s6 * s6 - s6 + shift), 0.0)
        vir = (f[:, :, None] * d[:, None, :]).reshape(-1, 9)
        return torch.cat([f, 0.5 * ec[:, None], 0.5 * en[:, None], 0.5 * vir], 1)
    return _over_pairs(pos, box, max(rc, lj_cut), term, 14 if observables else 3)


def _bond_forces(pos, bonds, box):
    edge = torch.tensor(box, dtype=torch.float64, device=pos.device)
    d = pos[bonds[:, 0]] - pos[bonds[:, 1]]
    d = d - torch.round(d / edge) * edge
    r = d.norm(dim=1, keepdim=True)
    fd = -FENE["k"] / (1 - (r / FENE["r_max"]) ** 2) * d
    f = torch.zeros_like(pos)
    f.index_add_(0, bonds[:, 0], fd)
    return f.index_add_(0, bonds[:, 1], -fd)


def _elc_far_cut(box, h):
    """Far-formula cutoff of the layer correction at a pairwise error of
    ACCURACY, in steps of the smaller reciprocal edge."""
    ux, uy, lz = 1 / box[0], 1 / box[1], box[2]
    fc = min(ux, uy)
    while True:
        k = 2 * math.pi * fc
        s = k + 2 * (ux + uy)
        err = 0.5 / -math.expm1(-k * lz) * (
            math.exp(k * (h - lz)) * (s + 1 / (lz - h)) / (lz - h) +
            math.exp(-k * (h + lz)) * (s + 1 / (lz + h)) / (lz + h))
        if err <= ACCURACY:
            return fc
        fc += min(ux, uy)


def _elc_forces(pos, q, box, gap):
    """Minus the interaction with the image layers above and below the slab
    (plane waves up to the far cutoff), and the slab's dipole term."""
    far = _elc_far_cut(box, box[2] - gap)
    ux, uy, lz = 1 / box[0], 1 / box[1], box[2]
    f = torch.zeros_like(pos)
    f[:, 2] -= 4 * math.pi * ux * uy / lz * (q * (pos[:, 2] - lz / 2)).sum() * q
    z = pos[:, 2]
    for p in range(0, int(math.ceil(far * box[0]) + 2)):
        for s in range(0, int(math.ceil(far * box[1]) + 2)):
            if (p == 0 and s == 0) or math.hypot(ux * max(p - 1, 0), uy * max(s - 1, 0)) >= far:
                continue
            for sign in ((1,) if p == 0 or s == 0 else (1, -1)):
                kx, ky = 2 * math.pi * ux * p, 2 * math.pi * uy * s * sign
                w = math.hypot(kx, ky)
                ph = torch.polar(torch.ones_like(z), kx * pos[:, 0] + ky * pos[:, 1])
                up, dn = torch.exp(w * z), torch.exp(-w * z)
                su, sd = (q * up * ph).sum(), (q * dn * ph).sum()
                a = 4 * math.pi * ux * uy / (w * math.expm1(w * lz)) * q
                # phi_i ~ Re(conj(ph_i) (up_i S_dn + dn_i S_up)); F = -q grad phi, minus
                c = ph.conj() * (up * sd + dn * su)
                f[:, 0] += a * kx * c.imag
                f[:, 1] += a * ky * c.imag
                f[:, 2] += a * w * (ph.conj() * (up * sd - dn * su)).real
    return f


def _dipole_mesh(pos, mu, edge, m, cao, alpha):
    """k-space fields of dipolar P3M at the particles: E_j and the symmetric
    tensor E_cd (xx, xy, xz, yy, yz, zz)."""
    dev, mesh = pos.device, [m] * 3
    grid = _Mesh(pos, [edge] * 3, mesh, cao)
    n, dop = _axes(mesh, dev, False), _axes(mesh, dev, True)
    mk = sum(dop[d] * torch.fft.rfftn(grid.assign(mu[:, d])) for d in range(3))
    n2 = sum(x * x for x in n)
    dn = sum(a * b for a, b in zip(n, dop))
    dd = sum(x * x for x in dop)
    ex = (math.pi / (alpha * edge)) ** 2 * n2
    on = (ex < 30) & ~_all_half(mesh, dev) & (dd > 0)
    base = 2.0 * m ** 3 / edge ** 2 * torch.exp(-ex) / (torch.where(on, n2, 1.0) * _u2(n, mesh, cao))
    ratio = dn / torch.where(on, dd, 1.0)
    ge = torch.where(on, base * ratio ** 2, 0.0)
    gf = torch.where(on, base * ratio ** 3, 0.0)
    size = m ** 3
    pairs = [(0, 0), (0, 1), (0, 2), (1, 1), (1, 2), (2, 2)]
    e = grid.interpolate([torch.fft.irfftn(dop[j] * ge * mk, s=mesh) * size for j in range(3)])
    t = grid.interpolate([torch.fft.irfftn(-1j * dop[a] * dop[b] * gf * mk, s=mesh) * size for a, b in pairs])
    return e, t


def _dipole_pairs(pos, mu, edge, alpha, r_cut):
    def term(i, j, d, r):
        ex, poly = _coulomb_part(alpha, r)
        co, r2 = 2 * alpha / math.sqrt(math.pi), r * r
        b = (poly / r + co) * ex / r2
        cc = (3 * b + 2 * alpha ** 2 * co * ex) / r2
        dd = (5 * cc + 4 * alpha ** 4 * co * ex) / r2
        mi, mj = mu[i], mu[j]
        mm, mid, mjd = (mi * mj).sum(1), (mi * d).sum(1), (mj * d).sum(1)
        f = (mm * cc - mid * mjd * dd)[:, None] * d + (mjd * cc)[:, None] * mi + (mid * cc)[:, None] * mj
        t = -torch.linalg.cross(mi, mj) * b[:, None] + torch.linalg.cross(mi, d) * (mjd * cc)[:, None]
        return torch.cat([f, t], 1)
    return _over_pairs(pos, [edge] * 3, r_cut, term, 6)


def _mesh3(c):
    return [c["mesh"]] * 3 if "mesh" in c else [c["mx"], c["my"], c["mz"]]


def exact(case, seed):
    c = case
    if c["kind"] == "batch":
        return None  # thermostat noise and parameters chosen by the batch's own tuner
    if c["kind"] == "dipoles":
        pos, mu, edge = _dipoles(c, seed)
        e, t = _dipole_mesh(pos, mu, edge, c["mesh"], c["cao"], c["alpha"])
        ft = _dipole_pairs(pos, mu, edge, c["alpha"], c["r_cut"])
        wn, m3 = 2 * math.pi / edge, float(c["mesh"]) ** 3
        tens = t[:, [0, 1, 2, 1, 3, 4, 2, 4, 5]].view(-1, 3, 3)
        force = wn * wn / m3 * (tens @ mu[:, :, None])[:, :, 0] + ft[:, :3]
        torque = -wn / m3 * torch.linalg.cross(mu, e) + ft[:, 3:]
        return {"force": force, "torque": torque}
    if c["kind"] == "frames":
        q, box = _system(c, seed)[1], _box(c)
        alpha, out = _alpha(_charged(q), c["r_cut"], box), []
        for x in _frame_list(c, seed):
            f, ek, vk = _kspace(x, q, box, _mesh3(c), c["cao"], alpha, True)
            s = _short(x, q, box, c, alpha, True)
            tot = s.sum(0)
            out.append({"f": f + s[:, :3],
                        "energy": torch.stack([tot[3] + ek, tot[4]]),
                        "pressure": (tot[5:].view(3, 3) + vk) / (box[0] * box[1] * box[2])})
        return out
    if c["kind"] == "md":
        pos, q, v = _script_inputs(c, seed)
        box, dt = _box(c), 0.005
        alpha = _alpha(_charged(q), c["r_cut"], box)
        edge = torch.tensor(box, dtype=torch.float64, device=pos.device)

        def forces(x):
            x = x - torch.floor(x / edge) * edge
            return _kspace(x, q, box, _mesh3(c), c["cao"], alpha) + _short(x, q, box, c, alpha)
        f = forces(pos)
        for _ in range(c["steps"]):
            v = v + 0.5 * dt * f
            pos = pos + dt * v
            f = forces(pos)
            v = v + 0.5 * dt * f
        return {"pos": pos, "v": v, "f": f}
    pos, q, _, bonds, box = _system(c, seed)
    edge = torch.tensor(box, dtype=torch.float64, device=pos.device)
    x = pos - torch.floor(pos / edge) * edge
    alpha = _alpha(_charged(q), c["r_cut"], box)
    f = _kspace(x, q, box, _mesh3(c), c["cao"], alpha) + _short(x, q, box, c, alpha)
    if len(bonds):
        f = f + _bond_forces(x, bonds, box)
    if c["gap"]:
        f = f + _elc_forces(x, q, box, c["gap"])
    return f
