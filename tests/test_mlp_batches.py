"""Batches smaller than the network's largest: the partial sums of the weight
gradients of every batch fit the workspace that the largest one sized."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from gelios_2d_b200 import warmstart as W
from oracle import mlp_oracle as O

CSRC = Path(__file__).resolve().parent.parent / "gelios_2d_b200" / "csrc"

PLAN = r"""
#include <algorithm>
#include <cstdio>
#include "mlp_plan.cuh"
int main() {
    int most = 0, bad = 0;
    for (int m = 1; m <= 1 << 20; m++) {
        most = std::max(most, gelios::splits_of(m));  // most slices of any batch up to m rows
        const int kc = gelios::tc_split_len(m, gelios::split_target(m));
        if (gelios::reserved_splits(m) < most || kc % gelios::kGemmBK || gelios::splits_of(m) * kc < m ||
            gelios::reserved_splits(m) > gelios::kMaxSplit)
            if (bad++ < 5) std::printf("max_batch %d: %d reserved, %d needed\n", m, gelios::reserved_splits(m), most);
    }
    return bad != 0;
}
"""


def test_workspace_holds_every_batch(tmp_path):
    """The split arithmetic of the library, compiled for the host: for every
    largest batch up to 2^20 rows the reserved slices hold those of every
    smaller batch."""
    (tmp_path / "plan.cpp").write_text(PLAN)
    exe = tmp_path / "plan"
    subprocess.run(["g++", "-O2", "-std=c++17", f"-I{CSRC}", str(tmp_path / "plan.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [8192, 7000])
def test_gradients_of_a_smaller_batch(rows):
    """A network made for 8193 rows (26 slices) on batches of 32 and 28: the
    gradients of one made for 8192, and 2e-3 of a tensor's norm from the
    float64 restatement, as in the other gradient tests."""
    rng = np.random.default_rng(rows)
    x = rng.uniform(-1, 1, (rows, 7)).astype(np.float32)
    t = rng.normal(size=(rows, 5)).astype(np.float32)
    got = []
    for max_batch in (8193, 8192):
        net = W.Mlp(7, 6, 64, 2, 5, max_batch)
        try:
            p = net.init_params(3)
            got.append(net.loss_grad(x, t))
        finally:
            net.close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])
    lay = O.layout(7, 6, 64, 2, 5)
    _, gb = O.loss_grad(p.astype(np.float64), x, t, 6, lay, bf16_mode=True)
    din, dout, w_off, b_off, _ = lay
    g = got[0][1]
    for l in range(len(din)):
        for a, n in ((w_off[l], din[l] * dout[l]), (b_off[l], dout[l])):
            assert np.linalg.norm(g[a:a + n] - gb[a:a + n]) <= 2e-3 * np.linalg.norm(gb[a:a + n])
