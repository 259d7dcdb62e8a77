"""Host checks of the wall table (no GPU): which boundary sides the wall kernels
walk, and that its index check passes on built tables and catches planted
entries."""
import os
import subprocess

import pytest

from giftbte_b200 import decks
from test_gpu_repeated_walls import twice

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "giftbte_b200", "csrc")
EXE = os.path.join(ROOT, "giftbte_b200", "_build", "tests", "wall_check")


@pytest.fixture(scope="module")
def driver():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    srcs = [os.path.join(ROOT, "tests", "cpp", "wall_check_main.cpp")] + [
        os.path.join(CSRC, f) for f in ("mesh.cpp", "angles.cpp", "deck.cpp")]
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, *srcs, "-o", EXE])
    return EXE


@pytest.mark.parametrize("make,slots,walls", [
    (lambda: decks.config1_deck(6), 24, 24),
    (lambda: decks.interface_deck(8), 32 + 16, 32 + 16),  # an interface wall has two sides, of two cell faces
    (lambda: twice(decks.config1_deck(6), [1, 3]), 24, 36),
    (lambda: decks.config3_deck(h_nm=25.0, size_nm=(50.0, 50.0, 50.0), n_bands=2), 48, 48),
], ids=["square", "interface", "twice", "block"])
def test_table_and_its_check(driver, tmp_path, make, slots, walls):
    make().write(str(tmp_path))
    r = subprocess.run([driver, str(tmp_path)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    last = r.stdout.split("\n")[-2].split()
    assert (int(last[1]), int(last[3])) == (slots, walls)
