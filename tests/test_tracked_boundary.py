"""A boundary face whose two end points lie on one tracked surface: the exact
Riemann solution between its cell and its boundary state, in every moving-grid
form."""
import numpy as np
import pytest

import gelios_2d_b200 as g
from gelios_2d_b200 import _native as N
from gelios_2d_b200 import workloads as W
from gelios_2d_b200.mesh import AXIS, EXTERN, INPUT, P_CONTACT, UPPER_WALL
from oracle import oracle as O

DIMS = (9, 5, 3, 17, 25, 7, 11, 6)


def _mesh():
    """One face of every outer boundary type that the grid has, its points
    declared contact points."""
    m = g.Mesh.setka(*DIMS)
    types = []
    for t in (EXTERN, INPUT, AXIS, UPPER_WALL):
        on = [f for f in m["gran"] if m["face_type"][f] == t and
              m["point_type"][m["face_A"][f]] < P_CONTACT and m["point_type"][m["face_B"][f]] < P_CONTACT]
        if on:
            f = on[len(on) // 2]
            m["point_type"][[m["face_A"][f], m["face_B"][f]]] = P_CONTACT
            types.append(t)
    return m, types


def test_the_grid_has_such_faces():
    m, types = _mesh()
    assert EXTERN in types and AXIS in types
    f = m["gran"]
    on = (m["point_type"][m["face_A"][f]] == P_CONTACT) & (m["point_type"][m["face_B"][f]] == P_CONTACT)
    assert np.count_nonzero(on & (m["face_type"][f] != 0)) >= len(types)


@pytest.mark.gpu
def test_five_fluids_against_the_oracle():
    """The parity bound of the form, 1e-12 per step, after two steps."""
    m, _ = _mesh()
    st0, h0 = W.init_conditions_reference(m), W.hydrogen_fields(m, seed=3)
    dev, ora = g.Setka(m, N.reference_params()), O.Oracle(O.reference_params(), m)
    for b in (0, 1):
        dev.set_par(b, st0)
        dev.set_hydrogen(b, h0)
        ora.set_state(b, st0)
        ora.set_hydrogen(b, h0)
    s = dev.Go_5_komponent(2)
    ora.five_komponent(2)
    for b in (0, 1):
        for x, y in ((dev.par(b), ora.get_state(b)), (dev.hydrogen(b), ora.get_hydrogen(b))):
            assert np.max(np.abs(x - y).max(axis=1) / np.abs(y).max(axis=1)) <= 1e-12
    st = ora.status()
    assert s.n_ro_clamp == st[1] and s.n_p_clamp == st[2]


@pytest.mark.gpu
def test_mk2_against_the_oracle():
    m, _ = _mesh()
    st0, mc = W.init_conditions_reference(m), W.mc_fields(m, seed=3)
    dev, ora = g.Setka(m, N.reference_params()), O.Oracle(O.reference_params(), m)
    for b in (0, 1):
        dev.set_par(b, st0)
        ora.set_state(b, st0)
    dev.set_mc(*mc)
    ora.set_mc(*mc)
    dev.Go_5_komponent__MK2(2)
    ora.mk2(2)
    for b in (0, 1):
        x, y = dev.par(b), ora.get_state(b)
        assert np.max(np.abs(x - y).max(axis=1) / np.abs(y).max(axis=1)) <= 1e-12
