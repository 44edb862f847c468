"""GPU tests of the size rules: every path that a rule on sizes, types or
alignment chooses, against the FP64 oracle (or against the same system
computed through another path).

Tolerances: FP64 1e-9 of the largest component (the oracle's own sums); FP32
2e-5, the FP32-mixed mesh and pair arithmetic as in test_gpu_p3m.py.
"""
import ctypes

import numpy as np
import pytest
import torch
from scipy.spatial import cKDTree

import espresso_b200 as eb
from espresso_b200 import _lib
from espresso_b200.electrostatics import P3M, P3MGPU
from espresso_b200.magnetostatics import DipolarP3M
from oracle import oracle as O

pytestmark = pytest.mark.gpu

DP = ctypes.POINTER(ctypes.c_double)
RTOL = {P3M: 1e-9, P3MGPU: 2e-5}


def _ions(n, box, seed=0):
    rng = np.random.default_rng(seed)
    side = int(np.ceil(n ** (1.0 / 3.0)))
    cell = np.asarray(box) / side
    sites = rng.choice(side ** 3, n, replace=False)
    idx = np.stack(np.unravel_index(sites, (side,) * 3), 1)
    pos = (idx + 0.5 + rng.uniform(-0.1, 0.1, (n, 3))) * cell
    return pos, np.where(np.arange(n) % 2 == 0, 1.0, -1.0)


def _actor(cls, box, pos, q, mesh, cao, alpha=1.0, r_cut=2.0):
    act = cls(prefactor=1.0, accuracy=1e-4, mesh=list(mesh), cao=cao, alpha=alpha, r_cut=r_cut,
              tune=False, check_neutrality=False)
    act._set_system(box, 0.4, (True, True, True))
    act._activate(pos, q)
    return act


def _long_range(act, pos, q, mesh):
    lib = _lib.load()
    f = np.zeros((len(q), 3))
    e, v = np.zeros(1), np.zeros(9)
    flags = _lib.P3MX_FORCES | _lib.P3MX_ENERGY | _lib.P3MX_VIRIAL | _lib.P3MX_OVERWRITE
    _lib.check(lib.p3mx_long_range(act._handle, len(q), _lib.dptr(pos), _lib.dptr(q), _lib.dptr(f),
                                   e.ctypes.data_as(DP), v.ctypes.data_as(DP), flags, None),
               act._handle)
    rho = np.zeros(mesh)
    _lib.check(lib.p3mx_copy_mesh(act._handle, rho.ctypes.data_as(DP), rho.size), act._handle)
    return f, e[0], v.reshape(3, 3), rho


# meshes: last super-bricks shorter than the stencil (three covers of the first
# points), one super-brick per axis, 16-point super-bricks (many of them) with
# whole and ragged ends; axis lengths with every transform factor (2..10, 12,
# 14, 15, 16), powers of two, no two factors (22, 34, 200), odd factor pairs;
# brick counts on both sides of 4096 and 32 768 (the three scans)
@pytest.mark.parametrize("cls", [P3M, P3MGPU])
@pytest.mark.parametrize("mesh,cao", [
    ((10, 18, 26), 7), ((8, 8, 8), 7), ((12, 20, 28), 3), ((18, 34, 22), 5), ((30, 42, 54), 6),
    ((64, 32, 48), 4), ((90, 70, 84), 1), ((100, 126, 140), 7), ((130, 98, 120), 7),
    ((144, 150, 210), 2), ((224, 96, 16), 6), ((128, 16, 256), 5), ((200, 50, 36), 7),
    ((128, 128, 128), 6), ((128, 64, 272), 7)])
def test_long_range_meshes(cls, mesh, cao):
    box = np.array([9.0, 10.0, 11.0]) if max(mesh) < 100 else np.array([21.0, 20.0, 23.0])
    pos, q = _ions(700, box, seed=cao)
    # particles on the box faces and corners: stencils that wrap every axis
    pos[:8] = np.stack(np.meshgrid([0, 1], [0, 1], [0, 1]), -1).reshape(-1, 3) * box * (1 - 1e-9)
    alpha = 0.5 * min(mesh) / max(box)
    act = _actor(cls, box, pos, q, mesh, cao, alpha=alpha, r_cut=1.0)
    f, e, v, rho = _long_range(act, pos, q, mesh)
    prm = O.make_params(box, mesh, cao, alpha, 1.0, 1.0)
    fo, eo, vo, rho_o = O.p3m_kspace(prm, pos, q, want_mesh=True)
    tol = RTOL[cls]
    np.testing.assert_allclose(rho, rho_o, rtol=0, atol=tol * np.abs(rho_o).max())
    np.testing.assert_allclose(f, fo, rtol=0, atol=tol * np.abs(fo).max())
    # energies and virials of both actors are FP64 sums (self terms cancel)
    assert abs(e - eo) <= 1e-9 * (abs(eo) + (q * q).sum() * alpha)
    np.testing.assert_allclose(v, vo, rtol=0, atol=1e-9 * np.abs(vo).max())


def _near(pos, box, types, cuts):
    """Particles of pairs within FP32 rounding of a cutoff ({(type, type): r},
    or {None: r} for every pair): such a pair may fall on either side."""
    out = np.zeros(len(pos), bool)
    tree = cKDTree(np.mod(pos, box), boxsize=box)
    for kind, cut in cuts.items():
        i, j = tree.query_pairs(cut + 1e-6, output_type="ndarray").T
        if kind is not None:
            sel = np.isin(types[i], kind) & np.isin(types[j], kind) & (types[i] != types[j])
            i, j = i[sel], j[sel]
        d = pos[i] - pos[j]
        d -= box * np.rint(d / box)
        sel = np.sqrt((d * d).sum(1)) > cut - 1e-6
        out[i[sel]] = out[j[sel]] = True
    return out


# particle numbers for 8, 4, 2 and 1 lanes per particle of the pair kernels, in
# either precision, with and without energies, and for 2 lanes above a wave of
# blocks
@pytest.mark.parametrize("cls", [P3M, P3MGPU])
@pytest.mark.parametrize("n", [3001, 15000, 30000, 45000, 60000, 100001, 116001, 160001])
@pytest.mark.parametrize("form", ["wca", "types", "offset"])
def test_pair_lanes_and_types(cls, n, form):
    box = np.full(3, (n / 0.4) ** (1.0 / 3.0))
    pos, q = _ions(n, box, seed=1)
    if n % 2:
        q[-1] = 0.0
    types = (np.arange(n) % 3 == 0).astype(np.int32) if form != "wca" else np.zeros(n, np.int32)
    s = eb.System(box_l=box)
    s.time_step = 0.01
    s.part.add(pos=pos, q=q, type=types)
    off = 0.2 if form == "offset" else 0.0
    if form == "wca":
        pairs = {(0, 0): dict(wca_eps=1.0, wca_sig=1.0)}
        s.non_bonded_inter[0, 0].wca.set_params(epsilon=1.0, sigma=1.0)
    else:
        lj = dict(lj_eps=1.3, lj_sig=0.9, lj_cut=2.0, lj_shift=0.1, lj_offset=off)
        pairs = {(0, 0): dict(wca_eps=1.0, wca_sig=1.0), (0, 1): lj}  # (1, 1): none
        s.non_bonded_inter[0, 0].wca.set_params(epsilon=1.0, sigma=1.0)
        s.non_bonded_inter[0, 1].lennard_jones.set_params(epsilon=1.3, sigma=0.9, cutoff=2.0,
                                                          shift=0.1, offset=off)
    s.electrostatics.solver = cls(prefactor=1.5, accuracy=1e-3, mesh=32, cao=3, r_cut=2.4,
                                  alpha=1.1, tune=False)
    act = s.electrostatics.solver
    s._sync_pairs(act._handle, types)
    lib = _lib.load()
    prm = O.make_params(box, [32] * 3, 3, 1.1, 2.4, 1.5)
    nt = 1 + int(types.max())
    fo, eo, vc, vn = O.short_range(prm, pos, q, types, nt, O.pair_table(nt, pairs))
    scale = np.abs(fo).max()
    # FP32: a pair within rounding of the LJ cutoff changes two particles by the
    # force there (0.06 at 2.0), one at the Coulomb cutoff by 7.8e-4 = 1.5
    # (erfc(1.1 r) / r^2 + 2.2 / sqrt(pi) exp(-(1.1 r)^2) / r) at r = 2.4; any other
    # particle agrees
    near = np.zeros(n, bool)
    if cls is P3MGPU:
        near = _near(pos, box, types, {None: 2.4} if form == "wca" else
                     {None: 2.4, (0, 1): 2.0 + off})
    # with energies and virials, and the instances without
    for flags in (_lib.P3MX_FORCES | _lib.P3MX_ENERGY | _lib.P3MX_VIRIAL, _lib.P3MX_FORCES):
        f = np.zeros((n, 3))
        e, v = np.zeros(2), np.zeros(18)
        _lib.check(lib.p3mx_short_range(act._handle, n, _lib.dptr(pos), _lib.dptr(q),
                                        _lib.dptr(types), _lib.dptr(f), e.ctypes.data_as(DP),
                                        v.ctypes.data_as(DP), flags | _lib.P3MX_OVERWRITE, None),
                   act._handle)
        d = np.abs(f - fo).max(1)
        assert d[~near].max() <= RTOL[cls] * scale
        assert d.max() <= max(RTOL[cls] * scale, 0.1 if near.any() else 0.0)
        if flags & _lib.P3MX_ENERGY:
            np.testing.assert_allclose(e, eo, rtol=1e-9, atol=1e-9 * n)
            np.testing.assert_allclose(v.reshape(2, 3, 3), [vc, vn], rtol=0,
                                       atol=1e-9 * max(np.abs(vc).max(), np.abs(vn).max()))


# dipolar pair lanes: a 2x2x2 supercell (twice the mesh) gives every copy of a
# dipole the forces and torques of the single cell
@pytest.mark.parametrize("single,tol", [(False, 1e-9), (True, 2e-5)])
@pytest.mark.parametrize("n,mesh", [(500, 10), (3750, 22), (7500, 28), (15000, 36)])
def test_dipole_supercell(single, tol, n, mesh):
    rng = np.random.default_rng(n)
    edge = (n / 0.5) ** (1.0 / 3.0)
    pos, _ = _ions(n, [edge] * 3, seed=n)
    mu = rng.normal(size=(n, 3))
    mu[::7] = 0.0  # non-magnetic particles

    def compute(x, m, length, points):
        act = DipolarP3M(prefactor=1.1, accuracy=1e-4, mesh=points, cao=5, r_cut=3.2, alpha=0.9,
                         tune=False, single_precision=single)
        act._set_system([length] * 3, 0.4, (True, True, True))
        act._activate(x, m)
        f, t, e = np.zeros_like(x), np.zeros_like(x), np.zeros(2)
        flags = _lib.P3MX_FORCES | _lib.P3MX_ENERGY | _lib.P3MX_OVERWRITE
        act._check(_lib.load().p3mx_dp3m_compute(act._handle, len(x), _lib.dptr(x), _lib.dptr(m),
                                                 _lib.dptr(f), _lib.dptr(t), e.ctypes.data_as(DP),
                                                 flags, None))
        # the instances without the energy
        f2, t2, _ = act._compute(x, m)
        np.testing.assert_allclose(f2, f, rtol=0, atol=tol * np.abs(f).max())
        np.testing.assert_allclose(t2, t, rtol=0, atol=tol * np.abs(t).max())
        return f, t, e
    f1, t1, e1 = compute(pos, mu, edge, mesh)
    shifts = np.stack(np.meshgrid(*[[0, edge]] * 3, indexing="ij"), -1).reshape(-1, 3)
    big = np.concatenate([pos + s for s in shifts])
    f8, t8, e8 = compute(big, np.tile(mu, (8, 1)), 2 * edge, 2 * mesh)
    np.testing.assert_allclose(f8.reshape(8, n, 3), np.broadcast_to(f1, (8, n, 3)), rtol=0,
                               atol=tol * np.abs(f1).max())
    np.testing.assert_allclose(t8.reshape(8, n, 3), np.broadcast_to(t1, (8, n, 3)), rtol=0,
                               atol=tol * np.abs(t1).max())
    # the real-space energy is the sum over the copies.  A dipole's part is of order
    # 1 and of either sign, its error below tol and independent of the others': the
    # sum over 8 n dipoles is of order sqrt(8 n), its error below tol 8 sqrt(8 n)
    assert abs(e8[1] - 8 * e1[1]) <= tol * 8 * np.sqrt(8 * n)


@pytest.mark.parametrize("cls", [P3M, P3MGPU])
def test_charge_change_and_table_change(cls):
    """Setting the same pair table keeps the lists; another table, and a
    particle that becomes charged, rebuild them."""
    box = np.full(3, 14.0)
    pos, q = _ions(1000, box, seed=4)
    q[:100] = 0.0
    s = eb.System(box_l=box)
    s.time_step = 0.01
    s.part.add(pos=pos, q=q)
    s.non_bonded_inter[0, 0].wca.set_params(epsilon=1.0, sigma=1.0)
    s.electrostatics.solver = cls(prefactor=1.0, accuracy=1e-3, mesh=24, cao=5, r_cut=2.5,
                                  alpha=1.1, tune=False)
    prm = O.make_params(box, [24] * 3, 5, 1.1, 2.5, 1.0)

    def check(tab):
        s.integrator.run(0)
        fo = O.p3m_kspace(prm, pos, s.part.all().q)[0] + \
            O.short_range(prm, pos, s.part.all().q, None, 1, O.pair_table(1, {(0, 0): tab}))[0]
        np.testing.assert_allclose(s.part.all().f, fo, rtol=0, atol=RTOL[cls] * np.abs(fo).max())
    count = ctypes.c_longlong()
    check(dict(wca_eps=1.0, wca_sig=1.0))
    _lib.load().p3mx_launch_count(s.electrostatics.solver._handle, ctypes.byref(count))
    before = count.value
    check(dict(wca_eps=1.0, wca_sig=1.0))
    _lib.load().p3mx_launch_count(s.electrostatics.solver._handle, ctypes.byref(count))
    assert count.value - before <= 15  # no rebuild: no cell sort, no list build
    q[:100] = np.where(np.arange(100) % 2 == 0, 0.5, -0.5)
    s.part.all().q = q
    check(dict(wca_eps=1.0, wca_sig=1.0))
    s.non_bonded_inter[0, 0].wca.set_params(epsilon=2.0, sigma=1.1)
    check(dict(wca_eps=2.0, wca_sig=1.1))


@pytest.mark.parametrize("cls", [P3M, P3MGPU])
def test_observables_without_forces(cls):
    """p3mx_forces without a force array returns the energies and virials that
    it returns with one."""
    box = np.full(3, 15.0)
    pos, q = _ions(1500, box, seed=5)
    act = _actor(cls, box, pos, q, [32] * 3, 5, alpha=1.2, r_cut=2.5)
    lib = _lib.load()
    out = []
    for force in (np.zeros((1500, 3)), None):
        e, v = np.zeros(3), np.zeros(27)
        _lib.check(lib.p3mx_forces(act._handle, 1500, _lib.dptr(pos), _lib.dptr(q), None,
                                   _lib.dptr(force), e.ctypes.data_as(DP), v.ctypes.data_as(DP),
                                   _lib.P3MX_ENERGY | _lib.P3MX_VIRIAL | _lib.P3MX_OVERWRITE, None),
                   act._handle)
        out.append(np.concatenate([e, v]))
    np.testing.assert_array_equal(out[0], out[1])
    # ... and leaves the mesh of its own positions to p3mx_copy_mesh, as does
    # a call with forces after it
    prm = O.make_params(box, [32] * 3, 5, 1.2, 2.5, 1.0)
    for k, force in enumerate((None, np.zeros((1500, 3)), None)):
        x = np.mod(pos + 0.37 * (k + 1), box)
        _lib.check(lib.p3mx_forces(act._handle, 1500, _lib.dptr(x), _lib.dptr(q), None,
                                   _lib.dptr(force), e.ctypes.data_as(DP), v.ctypes.data_as(DP),
                                   _lib.P3MX_ENERGY | _lib.P3MX_OVERWRITE, None), act._handle)
        rho = np.zeros((32, 32, 32))
        _lib.check(lib.p3mx_copy_mesh(act._handle, rho.ctypes.data_as(DP), rho.size), act._handle)
        rho_o = O.p3m_kspace(prm, x, q, want_mesh=True)[3]
        np.testing.assert_allclose(rho, rho_o, rtol=0, atol=RTOL[cls] * np.abs(rho_o).max())
    # a mesh is copied again as it was, also after a new pair table
    _lib.check(lib.p3mx_forces(act._handle, 1500, _lib.dptr(x), _lib.dptr(q), None, _lib.dptr(force),
                               None, None, _lib.P3MX_OVERWRITE, None), act._handle)
    tab = (_lib.PairParams * 1)()
    tab[0].wca_eps = tab[0].wca_sig = 1.0
    again = []
    for k in range(2):
        rho = np.zeros((32, 32, 32))
        _lib.check(lib.p3mx_copy_mesh(act._handle, rho.ctypes.data_as(DP), rho.size), act._handle)
        again.append(rho)
        _lib.check(lib.p3mx_set_pair_params(act._handle, 1, tab), act._handle)
    np.testing.assert_array_equal(again[1], again[0])
    np.testing.assert_allclose(again[0], rho_o, rtol=0, atol=RTOL[cls] * np.abs(rho_o).max())


def _device_call(lib, act, fn, n, pos, q, types, f):
    flags = _lib.P3MX_DEVICE_PTRS | _lib.P3MX_FORCES | _lib.P3MX_OVERWRITE
    if fn == "forces":
        return lib.p3mx_forces(act._handle, n, pos, q, types, f, None, None, flags, None)
    if fn == "short":
        return lib.p3mx_short_range(act._handle, n, pos, q, types, f, None, None, flags, None)
    return lib.p3mx_long_range(act._handle, n, pos, q, f, None, None, flags, None)


@pytest.mark.parametrize("cls", [P3M, P3MGPU])
@pytest.mark.parametrize("fn", ["forces", "short", "long"])
def test_device_arrays_that_kernels_cannot_read(cls, fn):
    """Device arrays are read by kernels where these can: a NULL array is an
    error and not a fault, and arrays off their alignment are copied."""
    n, box = 1000, np.full(3, 13.0)
    pos, q = _ions(n, box, seed=6)
    types = (np.arange(n) % 2).astype(np.int32)
    act = _actor(cls, box, pos, q, [24] * 3, 5, alpha=1.1, r_cut=2.5)
    lib = _lib.load()
    tab = (_lib.PairParams * 4)()
    tab[1].wca_eps = tab[2].wca_eps = tab[1].wca_sig = tab[2].wca_sig = 1.0
    _lib.check(lib.p3mx_set_pair_params(act._handle, 2, tab), act._handle)
    d = [torch.from_numpy(a).cuda() for a in (pos, q, types)]
    f = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ptr = [_lib.dptr(a) for a in d]
    assert _device_call(lib, act, fn, n, *ptr, _lib.dptr(f)) == 0
    want = f.clone()
    for k in range(2):
        bad = list(ptr)
        bad[k] = None
        assert _device_call(lib, act, fn, n, *bad, _lib.dptr(f)) != 0
    off = []  # the same arrays, 4 and 2 bytes off their alignment
    for a in d:
        raw = a.contiguous().view(torch.uint8).reshape(-1)
        buf = torch.empty(len(raw) + 16, dtype=torch.uint8, device="cuda")
        shift = a.element_size() // 2
        buf[shift:shift + len(raw)] = raw
        off.append((buf, ctypes.c_void_p(buf.data_ptr() + shift)))
    f.zero_()
    torch.cuda.synchronize()
    assert _device_call(lib, act, fn, n, *[p for _, p in off], _lib.dptr(f)) == 0
    assert torch.equal(f, want)


# axis lengths whose backward z pass takes one line per block: 2048 points in
# FP64 (two lines would need 241 568 bytes of shared memory), 3840 in FP32
@pytest.mark.parametrize("cls,mz,energy", [(P3M, 2048, True), (P3MGPU, 2048, True),
                                           (P3MGPU, 3840, False)])
def test_long_z_axis(cls, mz, energy):
    mesh, box = (8, 6, mz), np.array([6.0, 5.0, 0.4 * mz])
    pos, q = _ions(700, box, seed=9)
    act = _actor(cls, box, pos, q, mesh, 3, alpha=0.9, r_cut=1.0)
    lib = _lib.load()
    f, e = np.zeros((len(q), 3)), np.zeros(1)
    flags = _lib.P3MX_FORCES | _lib.P3MX_OVERWRITE | (_lib.P3MX_ENERGY if energy else 0)
    _lib.check(lib.p3mx_long_range(act._handle, len(q), _lib.dptr(pos), _lib.dptr(q), _lib.dptr(f),
                                   e.ctypes.data_as(DP), None, flags, None), act._handle)
    fo, eo, _ = O.p3m_kspace(O.make_params(box, mesh, 3, 0.9, 1.0, 1.0), pos, q)
    np.testing.assert_allclose(f, fo, rtol=0, atol=RTOL[cls] * np.abs(fo).max())
    if energy:
        assert abs(e[0] - eo) <= 1e-9 * (abs(eo) + (q * q).sum() * 0.9)


@pytest.mark.parametrize("cls", [P3M, P3MGPU])
def test_device_arrays_on_a_stream(cls):
    """Device arrays on the caller's stream, staged by the first kernel: small
    moves, moves beyond skin / 2, other types and other charges between calls give
    bitwise the forces of the host-array calls."""
    n, box = 4001, np.full(3, 20.0)
    pos, q = _ions(n, box, seed=8)
    q[-1] = 0.0
    rng = np.random.default_rng(8)
    types = (np.arange(n) % 2).astype(np.int32)
    lib = _lib.load()
    tab = (_lib.PairParams * 4)()
    tab[0].wca_eps = tab[0].wca_sig = 1.0
    tab[1].lj_eps, tab[1].lj_sig, tab[1].lj_cut = 1.0, 0.9, 2.2
    tab[2] = tab[1]
    acts = []
    for _ in range(2):
        act = _actor(cls, box, pos, q, [40] * 3, 5, alpha=1.1, r_cut=2.6)
        _lib.check(lib.p3mx_set_pair_params(act._handle, 2, tab), act._handle)
        acts.append(act)
    stream = torch.cuda.Stream()
    flags = _lib.P3MX_FORCES | _lib.P3MX_OVERWRITE
    f_dev = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for step in range(6):
        if step in (1, 3):
            pos = pos + rng.uniform(-0.05, 0.05, pos.shape)
        elif step == 2:
            pos = pos + rng.uniform(-0.5, 0.5, pos.shape)
        elif step == 4:
            types = 1 - types
        elif step == 5:
            q = np.roll(q, 7)  # another particle is the neutral one
        f = np.zeros((n, 3))
        _lib.check(lib.p3mx_forces(acts[0]._handle, n, _lib.dptr(pos), _lib.dptr(q),
                                   _lib.dptr(types), _lib.dptr(f), None, None, flags, None),
                   acts[0]._handle)
        with torch.cuda.stream(stream):
            d = [torch.from_numpy(a).cuda() for a in (pos, q, types)]
            _lib.check(lib.p3mx_forces(acts[1]._handle, n, *[_lib.dptr(a) for a in d],
                                       _lib.dptr(f_dev), None, None,
                                       flags | _lib.P3MX_DEVICE_PTRS,
                                       ctypes.c_void_p(stream.cuda_stream)), acts[1]._handle)
        np.testing.assert_array_equal(f_dev.cpu().numpy(), f)


@pytest.mark.parametrize("single", [False, True])
def test_dipoles_with_little_memory(single):
    """Where the device memory does not hold three field meshes, one serves the
    three field sets in turn: the same forces and torques, bitwise."""
    n, mesh, edge = 3000, 160, 18.0
    pos, _ = _ions(n, [edge] * 3, seed=2)
    mu = np.random.default_rng(2).normal(size=(n, 3))
    lib = _lib.load()

    def compute():
        act = DipolarP3M(prefactor=1.1, accuracy=1e-4, mesh=mesh, cao=5, r_cut=3.0, alpha=1.0,
                         tune=False, single_precision=single)
        act._set_system([edge] * 3, 0.4, (True, True, True))
        act._activate(pos, mu)
        f, t, _ = act._compute(pos, mu)
        count = ctypes.c_longlong()
        lib.p3mx_dp3m_launch_count(act._handle, ctypes.byref(count))
        return act, f, t, count.value
    act = compute()[0]  # kernels loaded, caches filled
    del act
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    act, f, t, launches = compute()
    used = before - torch.cuda.mem_get_info()[0]
    del act
    # leave one field mesh less than the actor took
    field = 4 * (4 if single else 8) * (mesh + 4) ** 3
    ballast = torch.empty(before - used + field, dtype=torch.uint8, device="cuda")
    try:
        act, f1, t1, launches1 = compute()
    finally:
        del ballast
        torch.cuda.empty_cache()
    assert launches1 == launches + 4
    np.testing.assert_array_equal(f1, f)
    np.testing.assert_array_equal(t1, t)
