"""The four-fluid step's face-unit groups and three-phase update on grids whose
groups and cells end inside a block and a warp."""
import numpy as np
import pytest

import gelios_2d_b200 as g
from gelios_2d_b200 import _native as N
from gelios_2d_b200 import workloads as W
from oracle import oracle as O


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(5, 3, 4, 9, 23, 6, 7, 9), (9, 5, 3, 17, 25, 7, 11, 6), (13, 4, 6, 20, 40, 9, 13, 17)])
def test_odd_grids_against_the_oracle(dims):
    """Two steps (the second on the moved grid, from the cached geometry); the
    parity bound of the form, 1e-12 per step."""
    m = g.Mesh.setka(*dims)
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
