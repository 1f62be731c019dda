"""The plain and inner forms run all steps of a call in one launch: the launch
count does not grow with the steps, whatever the order in which parameters and
list were set."""
import numpy as np
import pytest

import gelios_2d_b200 as g
from gelios_2d_b200 import _native as N
from gelios_2d_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _counts(go, launches):
    n = []
    for steps in (2, 9):
        go(steps)
        n.append(launches())
    return n


@pytest.mark.parametrize("dims", [(33, 17), (185, 128), (186, 128)])
@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_FP32_WAVES, N.PREC_FP32_FLUX])
def test_plain(dims, prec):
    mesh, P = g.Mesh.polar(*dims), W.plain_params(precision=prec)
    st = W.plain_initial(mesh, P)
    S = g.Setka(mesh, P)
    S.set_par(0, st)
    S.set_par(1, st)
    S.Go_stationary(1)  # the geometry's own launches
    assert _counts(S.Go_stationary, S.launches) == [2, 2]  # the words, the steps
    S.set_phase_timing(True)
    a, b = _counts(S.Go_stationary, S.launches)
    assert b - a == 3 * 7
    S.close()


def _inner(mesh, st, mc, prec):
    S = g.Setka(mesh, N.reference_params(precision=prec))
    S.set_par(0, st)
    S.set_par(1, st)
    S.set_mc(*mc)
    return S


@pytest.mark.parametrize("share", [0.05, 0.16, 0.17, 0.39, 0.41, 1.0])
@pytest.mark.parametrize("first", [N.PREC_FP64, N.PREC_FP32_FLUX])
def test_inner(share, first):
    """Lists within and beyond the flux rows (a sixth of the cells) and the unit
    geometry behind them (0.4), set while the fluxes were FP64 or FP32: FP64 steps take the lanes either way, and give
    the same bits as a context that never changed."""
    mesh = g.Mesh.setka(*W.SETKA_SMALL)
    st, mc = W.init_conditions_reference(mesh), W.mc_fields(mesh, seed=8)
    cells = np.random.RandomState(3).permutation(mesh.n_cells)[:int(share * mesh.n_cells)].astype(np.int32)
    out = []
    for prec in (first, N.PREC_FP64):
        S = _inner(mesh, st, mc, prec)
        N.check(S._L.gelios_set_inner_cells(S._h, cells.ctypes.data_as(N._IP), len(cells)), "gelios_set_inner_cells")
        if prec != N.PREC_FP64:
            S.set_params(N.reference_params(precision=N.PREC_FP64))
        S.Go_stationary_5_komponent_inner_MK2(3)
        assert _counts(S.Go_stationary_5_komponent_inner_MK2, S.launches) == [3, 3]  # words, table, steps
        out.append((S.par(0), S.par(1)))
        S.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("share", [0.05, 0.39])
def test_plain_between_inner_calls(share):
    """A long list's table overwrites the plain form's unit geometry: the plain
    steps that follow compute it again."""
    mesh = g.Mesh.setka(*W.SETKA_SMALL)
    st, mc = W.init_conditions_reference(mesh), W.mc_fields(mesh, seed=8)
    cells = np.arange(int(share * mesh.n_cells), dtype=np.int32)
    S, T = _inner(mesh, st, mc, N.PREC_FP64), _inner(mesh, st, mc, N.PREC_FP64)
    N.check(S._L.gelios_set_inner_cells(S._h, cells.ctypes.data_as(N._IP), len(cells)), "gelios_set_inner_cells")
    for k in range(2):
        S.Go_stationary(3)
        T.Go_stationary(3)
        for b in (0, 1):
            assert np.array_equal(S.par(b), T.par(b))
        S.Go_stationary_5_komponent_inner_MK2(2)
        for b in (0, 1):
            T.set_par(b, S.par(b))
    S.close()
    T.close()


def test_inner_between_moving_grid_calls():
    """The table lies in the moving grid's flux rows: calls of both forms in
    turn against a context whose inner calls use no table (phase timing: one
    thread per cell; they refresh the geometry cache alike) and that takes over
    the inner results."""
    mesh = g.Mesh.setka(*W.SETKA_SMALL)
    st, mc = W.init_conditions_reference(mesh), W.mc_fields(mesh, seed=8)
    S = _inner(mesh, st, mc, N.PREC_FP64)
    S.build_inner_list()
    T = _inner(mesh, st, mc, N.PREC_FP64)
    T.build_inner_list()
    for k in range(3):
        S.Go_5_komponent__MK2(4)
        T.Go_5_komponent__MK2(4)
        for b in (0, 1):
            assert np.array_equal(S.par(b), T.par(b))
        S.Go_stationary_5_komponent_inner_MK2(2 + k)
        T.set_phase_timing(True)
        T.Go_stationary_5_komponent_inner_MK2(2 + k)
        T.set_phase_timing(False)
        for b in (0, 1):
            T.set_par(b, S.par(b))
    S.close()
    T.close()
