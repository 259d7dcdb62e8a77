"""Host checks of the global face list (no GPU): which meshes have paired
faces, the condition of the face-value transport, and that every cell face
keeps its own centre where they are not."""
import os
import subprocess

import pytest

from giftbte_b200 import decks
from test_gpu_shared_faces import notched_square
from tests.golden import make_golden

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "giftbte_b200", "csrc")
EXE = os.path.join(ROOT, "giftbte_b200", "_build", "tests", "face_pairs")


@pytest.fixture(scope="module")
def driver():
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    srcs = [os.path.join(ROOT, "tests", "cpp", "face_pairs_main.cpp")] + [
        os.path.join(CSRC, f) for f in ("mesh.cpp", "angles.cpp", "deck.cpp")]
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, *srcs, "-o", EXE])
    return EXE


@pytest.mark.parametrize("make,paired", [
    (lambda: notched_square(4, 2), 0),
    (lambda: decks.config1_deck(6), 1),
    (lambda: decks.interface_deck(8), 1),
    (lambda: make_golden.load("quad_heat_specular")[0], 1),
    (lambda: decks.config3_deck(h_nm=25.0, size_nm=(50.0, 50.0, 50.0), n_bands=2), 1),
], ids=["notched", "square", "interface", "quads", "block"])
def test_paired_faces_and_centres(driver, tmp_path, make, paired):
    make().write(str(tmp_path))
    r = subprocess.run([driver, str(tmp_path)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    f = dict(zip(r.stdout.split()[0::2], r.stdout.split()[1::2]))
    assert int(f["paired"]) == paired
    # the mean of two or three coordinates, written to the deck and read back
    # at full precision: a few roundings of coordinates up to 64 faces away
    assert float(f["centre_error"]) <= 64 * 1e-15
