"""When the warm-start network takes its workspaces: what a gradient needs at
the first gradient, pinned staging once predictions have moved enough."""
import subprocess
from pathlib import Path

import numpy as np
import pytest

from gelios_2d_b200 import warmstart as W

CSRC = Path(__file__).resolve().parent.parent / "gelios_2d_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "mlp_plan.cuh"
using namespace gelios;
int main() {
    int bad = 0;
    const int64_t staging = 2 * stage_rows(8192, 7, 5) * 12 * 4;
    // one prediction of any grid of the warm start does not pin
    for (int64_t rows : {1LL, 5400LL, 86400LL, 200000LL}) bad += staging_worth(1, rows * 48, staging);
    // a program that predicts again and again does
    bad += staging_worth(30, 30 * 5400LL * 48, staging) || !staging_worth(100, 100 * 5400LL * 48, staging);
    bad += staging_worth(100, 100 * 48, staging) || !staging_worth(300, 300 * 48, staging);
    // chunks: at most the largest batch and 16 MB, at least 1024 rows of wide networks
    bad += stage_rows(8192, 7, 5) != 8192 || stage_rows(1 << 20, 7, 5) * 12 > (4 << 20) || stage_rows(100, 4096, 4096) != 100 ||
           stage_rows(1 << 20, 4096, 4096) != 1024;
    Carve c;
    for (size_t n : {1, 256, 257, 0, 100000}) {
        const size_t at = c.take(n);
        bad += at % 256 != 0 || c.bytes < at + n;
    }
    return bad;
}
"""


def test_rules(tmp_path):
    (tmp_path / "rules.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", f"-I{CSRC}", str(tmp_path / "rules.cpp"), "-o", str(tmp_path / "rules")],
                   check=True)
    assert subprocess.run([str(tmp_path / "rules")]).returncode == 0


@pytest.mark.gpu
@pytest.mark.parametrize("rows", [1, 512, 513, 1500, 1537])
def test_predictions_before_and_after_staging(rows):
    """One to three chunks of 512 rows through the driver's staging, then (a
    prediction of 16 MB later) through its own; the same bits."""
    net = W.Mlp(7, 6, 64, 2, 5, 512)
    try:
        net.init_params(2)
        x = np.random.default_rng(rows).uniform(-1, 1, (rows, 7)).astype(np.float32)
        first = net.predict(x)
        assert np.array_equal(net.predict(x), first)
        net.predict(np.zeros((350000, 7), np.float32))
        for _ in range(3):
            assert np.array_equal(net.predict(x), first)
        assert net.predict(x[:0]).shape == (0, 5)
    finally:
        net.close()


@pytest.mark.gpu
@pytest.mark.parametrize("width,n_out", [(64, 5), (20, 5), (64, 33)])
def test_gradient_memory_comes_with_the_first_gradient(width, n_out):
    """A network that only predicts holds no gradient workspace; the first
    gradient takes it, a second one nothing more."""
    import torch

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, (300, 7)).astype(np.float32)
    t = rng.normal(size=(300, n_out)).astype(np.float32)
    net = W.Mlp(7, 6, width, 3, n_out, 200000)
    try:
        net.init_params(5)
        net.predict(x)
        a = free()
        l1, g1 = net.loss_grad(x, t)
        b = free()
        l2, g2 = net.loss_grad(x, t)
        assert b < a - (8 << 20) and free() == b
        assert l1 == l2 and np.array_equal(g1, g2)
    finally:
        net.close()
