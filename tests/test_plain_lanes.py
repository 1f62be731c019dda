"""The plain form's one-launch kernels at the sizes where their split changes:
four lanes per cell (up to 640 lanes per SM), two phases beyond that, one
thread-block cluster per instance in a batch."""
import ctypes as C

import numpy as np
import pytest

from gelios_2d_b200 import _native as N
from gelios_2d_b200 import warmstart as W
from gelios_2d_b200.mesh import Mesh
from gelios_2d_b200.workloads import SETKA_SMALL, init_conditions_reference, plain_initial, plain_params

pytestmark = pytest.mark.gpu


def _run(mesh, prm, st, steps, one_launch):
    import gelios_2d_b200 as g

    S = g.Setka(mesh, prm)
    S.set_par(0, st)
    S.set_par(1, st)
    S.set_phase_timing(not one_launch)  # phase timing: one launch per phase and step
    r = S.Go_stationary(steps)
    out = S.par(0), S.par(1), r.dt, r.n_ro_clamp, r.n_p_clamp, r.flags
    S.close()
    return out


# 185 x 128 cells are the most that 640 lanes on each of 148 SMs hold
@pytest.mark.parametrize("grid", [(2, 2), (3, 7), (33, 17), (185, 128), (186, 128), "rails"])
@pytest.mark.parametrize("prec", [N.PREC_FP64, N.PREC_FP32_WAVES])
def test_one_launch_equals_one_launch_per_phase(grid, prec):
    """Same fixed operations in every kernel: at most the last bits of the
    geometry differ, 1e-13 after seven steps (2^-53 times the ~1e3 operations
    a value passes)."""
    prm = plain_params(precision=prec)
    if grid == "rails":  # triangles and the central fan (C_centr)
        mesh = Mesh.setka(*SETKA_SMALL)
        st = init_conditions_reference(mesh)
    else:
        mesh = Mesh.polar(*grid)
        st = plain_initial(mesh, prm)
    a, b = (_run(mesh, prm, st, 7, k) for k in (True, False))
    for x, y in zip(a[:2], b[:2]):
        scale = np.abs(y).max(axis=1, keepdims=True)
        assert np.max(np.abs(x - y) / np.maximum(np.abs(y), 1e-6 * scale)) <= 1e-13
    assert abs(a[2] - b[2]) <= 1e-13 * b[2] and a[3:] == b[3:]


@pytest.mark.parametrize("n", [1, 9, 19, 40, 300])
def test_batch_clusters_equal_single_contexts(n):
    """Cluster sizes 16 down to 1 (a block per instance); odd step count."""
    import gelios_2d_b200 as g

    mesh = Mesh.polar(13, 11, 1.0, 600.0)
    th = W.sample_inflows(n, 5)
    sts = [W.cold_state(mesh, W.inflow_params(t)) for t in th]
    ss = [g.Setka(mesh, W.inflow_params(t)) for t in th]
    try:
        for S, st in zip(ss, sts):
            S.set_par(0, st)
            S.set_par(1, st)
        b = C.c_void_p()
        hs = (C.c_void_p * n)(*[S._h for S in ss])
        N.check(N.lib().gelios_plain_batch_create(C.byref(b), hs, n), "gelios_plain_batch_create")
        got = (N.GeliosStatus * n)()
        try:
            N.check(N.lib().gelios_plain_batch_step(b, 9, got), "gelios_plain_batch_step")
        finally:
            N.lib().gelios_plain_batch_destroy(b)
        for i in sorted({0, n // 2, n - 1}):
            ref = _run(mesh, W.inflow_params(th[i]), sts[i], 9, True)
            assert np.array_equal(ss[i].par(0), ref[0]) and np.array_equal(ss[i].par(1), ref[1])
            assert got[i].dt == ref[2]
    finally:
        for S in ss:
            S.close()


@pytest.mark.parametrize("dims,n", [((60, 50), 2), ((60, 50), 3), ((186, 128), 2)])
def test_few_instances_of_a_large_mesh(dims, n):
    """One instance after the other up to 2 instances of 3000 cells (lanes) and
    of 23808 (two phases), clusters from 3 instances on: the same bits as
    single contexts where the kernel is the same, else 1e-13 (as above)."""
    import gelios_2d_b200 as g

    mesh = Mesh.polar(*dims, 1.0, 600.0)
    th = W.sample_inflows(n, 9)
    sts = [W.cold_state(mesh, W.inflow_params(t)) for t in th]
    ss = [g.Setka(mesh, W.inflow_params(t)) for t in th]
    try:
        for S, st in zip(ss, sts):
            S.set_par(0, st)
            S.set_par(1, st)
        b = C.c_void_p()
        hs = (C.c_void_p * n)(*[S._h for S in ss])
        N.check(N.lib().gelios_plain_batch_create(C.byref(b), hs, n), "gelios_plain_batch_create")
        got = (N.GeliosStatus * n)()
        try:
            for _ in range(2):  # the second call arms the accumulators again
                N.check(N.lib().gelios_plain_batch_step(b, 6, got), "gelios_plain_batch_step")
        finally:
            N.lib().gelios_plain_batch_destroy(b)
        for i in range(n):
            S = g.Setka(mesh, W.inflow_params(th[i]))
            S.set_par(0, sts[i])
            S.set_par(1, sts[i])
            S.Go_stationary(6)
            r = S.Go_stationary(6)
            for x, y in ((ss[i].par(0), S.par(0)), (ss[i].par(1), S.par(1))):
                scale = np.abs(y).max(axis=1, keepdims=True)
                assert np.max(np.abs(x - y) / np.maximum(np.abs(y), 1e-6 * scale)) <= 1e-13
            assert abs(got[i].dt - r.dt) <= 1e-13 * r.dt
            S.close()
    finally:
        for S in ss:
            S.close()
