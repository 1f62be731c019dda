"""A cell whose density and pressure are both negative before the first step
(a caller's own state is not floored): its sound speed is the positive root of
gamma p / ro, as the reference takes it."""
import numpy as np
import pytest

import gelios_2d_b200 as g
from gelios_2d_b200 import _native as N
from gelios_2d_b200 import workloads as W
from oracle import oracle as O


def _go(p):
    return O.GoParams(**{n: getattr(p, n) for n, _ in O.GoParams._fields_ if n != "pad_"}, pad_=0)


def _case(form):
    if form == "plain":
        m, P = W.plain_mesh(36, 24), W.plain_params()
        st = W.plain_initial(m, P, seed=5)
    else:
        m, P = g.Mesh.setka(9, 5, 3, 17, 25, 7, 11, 6), N.reference_params()
        st = W.init_conditions_reference(m)
    # a cell of the outer flow, none of whose faces is tracked; the magnitude
    # makes it the one that decides the time step
    r = np.hypot(m["x"], m["y"])[m["contour"][m["contour_start"][:-1]]]
    tracked = np.isin(m["point_type"], (6, 7, 8))
    near = np.array([tracked[m["contour"][a:b]].any() for a, b in
                     zip(m["contour_start"][:-1], m["contour_start"][1:])])
    c = np.flatnonzero((m["cell_type"] != 5) & ~near & (r > 0.5 * r.max()))[7]
    st[0][c] = -st[0][c]
    st[1][c] = -1e8
    return m, P, st, c


def _oracle(form, m, P, st, mc, steps):
    o = O.Oracle(_go(P), m)
    o.set_state(0, st)
    o.set_state(1, st)
    if form == "mk2":
        o.set_mc(*mc)
    (o.stationary if form == "plain" else o.mk2)(steps)
    return o


@pytest.mark.parametrize("form", ["plain", "mk2"])
def test_the_cell_decides_the_step(form):
    """The oracle: the second step, whose dt the first one set, moves the state
    differently when the cell is left as it was."""
    m, P, st, c = _case(form)
    mc = W.mc_fields(m, seed=3)
    a = _oracle(form, m, P, st, mc, 2).get_state(0)
    st2 = st.copy()
    st2[0][c], st2[1][c] = -st[0][c], 1.0
    b = _oracle(form, m, P, st2, mc, 2).get_state(0)
    far = np.ones(m.n_cells, bool)
    far[max(0, c - 300):c + 300] = False
    assert np.isfinite(a).all()
    assert np.max(np.abs(a - b)[:, far].max(axis=1) / np.abs(b).max(axis=1)) > 1e-9


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["plain", "mk2"])
@pytest.mark.parametrize("timing", [False, True])
def test_against_the_oracle(form, timing):
    """1e-12 per step, the parity bound of the forms.  One step of the moving
    grid: its wave speeds enter the HLL flux itself, while after a second one
    the floored cell's velocity, a difference of momenta of 1e5 over a density
    of 1e-5, keeps only 11 digits in any arithmetic."""
    m, P, st, _ = _case(form)
    n = 2 if form == "plain" else 1
    mc = W.mc_fields(m, seed=3)
    S = g.Setka(m, P)
    S.set_par(0, st)
    S.set_par(1, st)
    if form == "mk2":
        S.set_mc(*mc)
    S.set_phase_timing(timing)  # the plain form's one launch per phase
    (S.Go_stationary if form == "plain" else S.Go_5_komponent__MK2)(n)
    o = _oracle(form, m, P, st, mc, n)
    x, y = S.par(n % 2), o.get_state(n % 2)
    S.close()
    assert np.max(np.abs(x - y).max(axis=1) / np.abs(y).max(axis=1)) <= 1e-12 * n
