"""K to pageable host arrays: the rule that chooses pinned pieces (pmsim_b200/csrc/pms_host_copy.h, compiled here
without CUDA), and the values either way."""
import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "pms_host_copy.h"
int main() {
    const size_t sizes[] = {0, pms::STAGE_PIECE - 8, pms::STAGE_PIECE, size_t(16) << 20, (size_t(16) << 20) + 8, size_t(240) << 20};
    for (int nt : {1, 2, 8})
        for (size_t b : sizes) std::printf("%d", pms::pieces_pay(b, nt) ? 1 : 0);
    return 0;
}
"""


def test_one_thread_leaves_large_arrays_to_the_driver(tmp_path):
    src, exe = tmp_path / "t.cpp", tmp_path / "t"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "pmsim_b200", "csrc"), "-o", str(exe), str(src)], check=True)
    assert subprocess.run([str(exe)], capture_output=True, text=True, timeout=60).stdout == "001100" + 2 * "001111"


VALUES = r"""
import numpy as np, torch
from pmsim_b200 import mesh as M
from pmsim_b200.elements import Elements, Material
for n in ((7, 6, 5), (11, 11, 10)):  # several pieces; more than one thread moves on
    m = M.structured_3d(M.HEX20, *n, *map(float, n))
    g = Elements(m, Material.von_mises(2e5, 0.3, 1e3, 250.0))
    g.initialize_internal_values()
    g.backup_secondary_values()
    ddu = np.random.default_rng(1).normal(0.0, 1e-3, g.ndof)
    ff, kk = np.zeros(g.ndof), np.zeros(g.nnz)
    d_ff, d_kk = (torch.zeros(k, dtype=torch.float64, device="cuda") for k in (g.ndof, g.nnz))
    torch.cuda.synchronize()
    g.update_and_assemble(torch.tensor(ddu, device="cuda"), d_ff, d_kk)
    g.sync()
    g.update_and_assemble(ddu, ff, kk)
    assert np.array_equal(kk, d_kk.cpu().numpy()) and np.array_equal(ff, d_ff.cpu().numpy())
print("same")
"""


@pytest.mark.gpu
@pytest.mark.parametrize("threads", ["1", "2"])
def test_values_with_few_host_threads(threads):
    env = dict(os.environ, OMP_NUM_THREADS=threads)
    r = subprocess.run([sys.executable, "-c", VALUES], cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "same", r.stderr[-2000:]
