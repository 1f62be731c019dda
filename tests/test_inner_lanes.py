"""The inner form's lane kernel (four lanes per listed cell, one launch for
all steps) against its one-thread-per-cell kernel, which phase timing uses."""
import numpy as np
import pytest

from gelios_2d_b200 import _native as N
from gelios_2d_b200 import workloads as W
from gelios_2d_b200.mesh import Mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 63, 64, 65, 1000, None])
@pytest.mark.parametrize("steps", [1, 4])
def test_lanes_equal_threads(n, steps):
    """The same formulas with factors of the fixed grid computed once: the
    per-step parity bound, 1e-12, per step."""
    import gelios_2d_b200 as g

    mesh = Mesh.setka(*W.SETKA_SMALL)
    st0 = W.init_conditions_reference(mesh)
    mc = W.mc_fields(mesh, seed=8)
    mc[0][::97] = 0.0  # cells without hydrogen
    out = []
    for timing in (False, True):
        S = g.Setka(mesh, N.reference_params())
        S.set_par(0, st0)
        S.set_par(1, st0)
        S.set_mc(*mc)
        S.build_inner_list()
        # any cells may be listed, in any order: spread over the grid, C_centr
        # and axis cells among them
        cells = S.All_Cells_Inner
        if n is not None:
            cells = np.random.RandomState(n).permutation(mesh.n_cells)[:n].astype(np.int32)
        S._L.gelios_set_inner_cells(S._h, cells.ctypes.data_as(N._IP), len(cells))
        S.set_phase_timing(timing)
        r = S.Go_stationary_5_komponent_inner_MK2(steps)
        out.append((S.par(0), S.par(1), r.dt, r.flags, r.n_ro_clamp, r.n_p_clamp))
        S.close()
    a, b = out
    for x, y in zip(a[:2], b[:2]):
        # as the oracle parity tests measure it: each row against its largest value
        assert np.max(np.abs(x - y).max(axis=1) / np.abs(y).max(axis=1)) <= 1e-12 * steps
    assert abs(a[2] - b[2]) <= 1e-12 * b[2] and a[3:] == b[3:]
