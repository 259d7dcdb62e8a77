"""GPU: the grid-wide conjugate gradient gives the same bits with its rows in
registers (one to four per thread) and in memory, when each thread owns the
same rows: the search direction that a thread forms for itself and the one it
forms for its neighbours are the same number."""
import os
import subprocess

import pytest

from giftbte_b200 import build

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
EXE = os.path.join(ROOT, "giftbte_b200", "_build", "tests", "cg_grid")


@pytest.fixture(scope="module")
def driver():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    src = os.path.join(ROOT, "tests", "cpp", "cg_grid_main.cu")
    subprocess.check_call([build.nvcc(), *build.ARCH, "-std=c++17", "-O3", "-I", build.CSRC, src, "-o", EXE])
    return EXE


@pytest.mark.parametrize("w,h,rows", [(23, 31, 1), (200, 201, 1), (200, 201, 2), (307, 401, 3), (307, 401, 4),
                                      (500, 500, 4)])
def test_rows_in_registers_and_in_memory(driver, w, h, rows):
    r = subprocess.run([driver, str(w), str(h), str(rows)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    f = r.stdout.split()
    assert int(f[3]) == int(f[4]) > 0
    assert int(f[6]) == 0, r.stdout
