"""GPU tests of calls after a configuration that failed: the error is raised
again by every call until the parameters are valid, and the forces after that
are those of a fresh actor (no state of the failed configuration is left)."""
import ctypes

import numpy as np
import pytest

import espresso_b200 as eb
from espresso_b200 import _lib
from espresso_b200.electrostatics import P3M, P3MGPU
from oracle import oracle as O
from tests.test_gpu_dispatch import RTOL, _ions

pytestmark = pytest.mark.gpu

IP = ctypes.POINTER(ctypes.c_int)
N, EDGE, MESH, CAO, ALPHA, R_CUT = 900, 12.0, 24, 5, 1.1, 2.5


def _system(cls):
    box = np.full(3, EDGE)
    pos, q = _ions(N, box, seed=3)
    s = eb.System(box_l=box)
    s.time_step = 0.01
    s.part.add(pos=pos, q=q)
    s.non_bonded_inter[0, 0].lennard_jones.set_params(epsilon=1.0, sigma=0.8, cutoff=1.8,
                                                      shift=0.0)
    s.electrostatics.solver = cls(prefactor=1.0, accuracy=1e-3, mesh=MESH, cao=CAO, r_cut=R_CUT,
                                  alpha=ALPHA, tune=False)
    return s, pos, q


def _check(s, pos, q, cls, bond=None):
    s.integrator.run(0)
    prm = O.make_params(np.full(3, EDGE), [MESH] * 3, CAO, ALPHA, R_CUT, 1.0)
    tab = O.pair_table(1, {(0, 0): dict(lj_eps=1.0, lj_sig=0.8, lj_cut=1.8)})
    fo = O.p3m_kspace(prm, pos, q)[0] + O.short_range(prm, pos, q, None, 1, tab)[0]
    if bond is not None:  # harmonic, k = 3, r_0 = 0
        d = pos[bond[0]] - pos[bond[1]]
        d -= EDGE * np.rint(d / EDGE)
        fo[bond[0]] -= 3.0 * d
        fo[bond[1]] += 3.0 * d
    np.testing.assert_allclose(s.part.all().f, fo, rtol=0, atol=RTOL[cls] * np.abs(fo).max())


@pytest.mark.parametrize("before", [False, True])  # the failure first, or after a good call
@pytest.mark.parametrize("cls", [P3M, P3MGPU])
def test_pair_cutoff_beyond_the_box(cls, before):
    s, pos, q = _system(cls)
    if before:
        _check(s, pos, q, cls)
    lj = s.non_bonded_inter[0, 0].lennard_jones
    # longer than the box: no cell grid holds it
    lj.set_params(epsilon=1.0, sigma=0.8, cutoff=2 * EDGE, shift=0.0)
    lib, h = _lib.load(), s.electrostatics.solver._handle
    f = np.zeros((N, 3))
    for _ in range(2):
        with pytest.raises(_lib.P3MXError, match="larger than the box"):
            s.integrator.run(0)
        # ... and by a force call that does not set the table
        rc = lib.p3mx_forces(h, N, _lib.dptr(pos), _lib.dptr(q), None, _lib.dptr(f), None, None,
                             _lib.P3MX_FORCES | _lib.P3MX_OVERWRITE, None)
        with pytest.raises(_lib.P3MXError, match="larger than the box"):
            _lib.check(rc, h)
        # a stage profile fails too, and leaves no profiling mode behind
        assert lib.p3mx_profile(h, 1, None, None, 0, None) != 0
    # bonds set meanwhile are used once the engine is configured again
    kind = (_lib.BondParams * 1)(_lib.BondParams(_lib.P3MX_BOND_HARMONIC, 3.0, 0.0, 0.0))
    trip = np.array([0, 17, 40], dtype=np.int32)
    assert lib.p3mx_set_bonds(h, 1, kind, 1, trip.ctypes.data_as(IP)) == 0
    s.electrostatics.solver._bonds_of = s
    s.electrostatics.solver._bond_version = s._bond_version
    lj.set_params(epsilon=1.0, sigma=0.8, cutoff=1.8, shift=0.0)
    _check(s, pos, q, cls, bond=(17, 40))


@pytest.mark.parametrize("cls", [P3M, P3MGPU])
def test_box_too_small(cls):
    """The mesh part scales with the box, the pair cutoff does not: a box
    below it fails, and the old box works again."""
    s, pos, q = _system(cls)
    _check(s, pos, q, cls)
    with pytest.raises(_lib.P3MXError, match="larger than the box"):
        s.box_l = [1.5] * 3
    for _ in range(2):
        with pytest.raises(_lib.P3MXError, match="larger than the box"):
            s.integrator.run(0)
    s.box_l = [EDGE] * 3
    _check(s, pos, q, cls)
