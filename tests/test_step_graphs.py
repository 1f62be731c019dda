"""Two steps of a moving-grid form as one graph: when it is formed, and that
calls of any length give what direct launches give."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

import gelios_2d_b200 as g
from gelios_2d_b200 import _native as N
from gelios_2d_b200 import workloads as W

ROOT = Path(__file__).resolve().parent.parent
CSRC = ROOT / "gelios_2d_b200" / "csrc"

RULE = r"""
#include <cstdio>
#include <cstdlib>
#include "graph_capture.cuh"
// argv: direct?, steps of every call; prints the call that forms the graph of two steps
int main(int, char** v) {
    const bool direct = std::atoi(v[1]) != 0;
    const int n = std::atoi(v[2]);
    int uses = 0;
    for (int call = 1; call <= 1000; call++)
        for (int st = 1; st + 1 < n; st += 2) {
            if (gelios::pair_graph_worth(direct, (n - st) / 2, uses)) { std::printf("%d\n", call); return 0; }
            uses++;
        }
    std::printf("0\n");
}
"""


@pytest.fixture(scope="module")
def rule(tmp_path_factory):
    d = tmp_path_factory.mktemp("rule")
    (d / "rule.cpp").write_text(RULE)
    inc = next((p for p in ("/usr/local/cuda/include",) if (Path(p) / "cuda_runtime_api.h").exists()), None)
    if inc is None:
        pytest.skip("CUDA headers not found")
    # the capture helper of the same header is a template: nothing of the runtime is linked
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", f"-I{inc}", str(d / "rule.cpp"), "-o", str(d / "rule")], check=True)
    return lambda direct, n: int(subprocess.run([str(d / "rule"), str(int(direct)), str(n)], capture_output=True,
                                                text=True, check=True).stdout)


@pytest.mark.parametrize("direct", [False, True])
def test_short_first_calls_form_no_graph_of_two_steps(rule, direct):
    """A call that would replay it less than three (seven, against direct
    launches) times does not pay for it; a program of such calls forms it once,
    after at least 64 missed uses."""
    at_once = 17 if direct else 9
    for n in range(3, at_once):
        call = rule(direct, n)
        assert call > 1 and (call - 1) * ((n - 1) // 2) <= 64 < call * ((n - 1) // 2) + 1
    for n in (at_once, at_once + 1, 60):
        assert rule(direct, n) == 1
    assert rule(direct, 1) == 0 and rule(direct, 2) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["mk2", "k5", "mhd"])
@pytest.mark.parametrize("calls", [(1, 2, 3, 4), (3, 20, 2, 5, 9, 1), (19, 19, 4), (2,) * 40])
def test_calls_of_any_length_equal_direct_launches(form, calls):
    """Odd and even lengths, before and after the two-step graph is formed; the
    same kernels in the same order: the same bits."""
    mesh = g.Mesh.setka(9, 5, 3, 17, 25, 7, 11, 6)
    st = W.init_conditions_reference(mesh)
    mp = W.mhd_params()
    out = []
    for timing in (False, True):  # phase timing launches directly, unpipelined
        S = g.Setka(mesh, N.reference_params())
        S.set_par(0, st)
        S.set_par(1, st)
        if form == "mk2":
            S.set_mc(*W.mc_fields(mesh, seed=1))
        if form == "k5":
            for b in (0, 1):
                S.set_hydrogen(b, W.hydrogen_fields(mesh, seed=2))
        if form == "mhd":
            S.set_mhd_params(mp)
            for b in (0, 1):
                S.set_mhd(b, W.mhd_initial(mesh, st, mp))
            S.set_sources(*W.mhd_sources(mesh, seed=3))
        S.set_phase_timing(timing)
        go = {"mk2": S.Go_5_komponent__MK2, "k5": S.Go_5_komponent, "mhd": S.Go_MHD_pickup}[form]
        dts = [go(n).dt for n in calls]
        extra = [S.hydrogen(0), S.hydrogen(1)] if form == "k5" else [S.mhd(0), S.mhd(1)] if form == "mhd" else []
        out.append([S.par(0), S.par(1), *S.points(), np.array(dts), *extra])
        S.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


@pytest.mark.gpu
def test_rail_table_follows_the_parameters():
    """n_inner is a constant of the rails' table: a context whose parameters
    change between calls moves the grid as a new one does."""
    mesh = g.Mesh.setka(9, 5, 3, 17, 25, 7, 11, 6)
    st, mc = W.init_conditions_reference(mesh), W.mc_fields(mesh, seed=1)
    p0 = N.reference_params()
    p1 = N.reference_params(n_inner=p0.n_inner - 1)

    def ctx(p):
        S = g.Setka(mesh, p)
        S.set_par(0, st)
        S.set_par(1, st)
        S.set_mc(*mc)
        return S

    ref = ctx(p1)
    ref.Go_5_komponent__MK2(3)
    S = ctx(p0)
    S.Go_5_komponent__MK2(3)
    assert not np.array_equal(S.points()[0], ref.points()[0])
    S.TVD_prepare()  # the topology again: the points of the mesh, not the moved ones
    S.set_par(0, st)
    S.set_par(1, st)
    S.set_mc(*mc)
    S.Go_5_komponent__MK2(1)
    S.set_params(p1)
    S.TVD_prepare()
    S.set_par(0, st)
    S.set_par(1, st)
    S.set_mc(*mc)
    S.Go_5_komponent__MK2(3)
    for a, b in zip((*S.points(), S.par(0), S.par(1)), (*ref.points(), ref.par(0), ref.par(1))):
        assert np.array_equal(a, b)
    ref.close()
    S.close()


@pytest.mark.gpu
def test_batch_before_and_after_its_graphs():
    """Calls of one to three steps of a batch, 46 in all: directly launched
    steps and the graphs formed at the sixteenth of each parity give the bits of
    single contexts that make the same calls."""
    from gelios_2d_b200.sweep import Sweep

    meshes = [g.Mesh.setka(9, 5, 3, 17, 25, 7, 11, 6), g.Mesh.setka(5, 3, 4, 9, 23, 6, 7, 9)]
    mp = W.mhd_params()
    inst = []
    for k, m in enumerate(meshes):
        st = W.init_conditions_reference(m)
        inst.append((m, N.reference_params(), st, (mp, W.mhd_initial(m, st, mp), W.mhd_sources(m, seed=k))))
    B = Sweep(inst, form=N.FORM_MHD_PUI, batched=True)
    ref = Sweep(inst, form=N.FORM_MHD_PUI, batched=False)
    for n in (1, 2, 3) * 7 + (1, 3):
        got = B.batch_step(n, statuses=True)
        for i, S in enumerate(ref.items):
            assert S.Go_MHD_pickup(n).dt == got[i].dt
    for i, S in enumerate(ref.items):
        for b in (0, 1):
            assert np.array_equal(B.par(i, b), S.par(b))
        assert np.array_equal(B.items[i].points()[0], S.points()[0])
