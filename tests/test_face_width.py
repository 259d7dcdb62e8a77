"""Host checks of the face-value gradient's block width (no GPU) on the meshes
of test_gpu_face_width.py, whose cells' order gets worse: the widest block of
which two fit on an SM, else the widest that fits at all; both kinds, and
several widths, are among them."""
import os
import subprocess

import pytest

from test_gpu_face_width import shuffled

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "giftbte_b200", "csrc")
EXE = os.path.join(ROOT, "giftbte_b200", "_build", "tests", "face_width")


@pytest.fixture(scope="module")
def widths(tmp_path_factory):
    os.makedirs(os.path.dirname(EXE), exist_ok=True)
    srcs = [os.path.join(ROOT, "tests", "cpp", "face_width_main.cpp")] + [
        os.path.join(CSRC, f) for f in ("mesh.cpp", "angles.cpp", "deck.cpp")]
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I", CSRC, *srcs, "-o", EXE])
    out = {}
    for window in (1, 60, 120, 4200):
        d = shuffled(window)
        d.mesh.cell_region[:] = 0  # one region, so that the deck lists the cells in this order
        d.region_heat = [0.0]
        root = tmp_path_factory.mktemp(f"w{window}")
        d.write(str(root))
        r = subprocess.run([EXE, str(root)], capture_output=True, text=True)
        assert r.returncode == 0, r.stdout + r.stderr
        rows = [list(map(int, line.split())) for line in r.stdout.splitlines()]
        out[window] = [(row[0], dict(zip(row[2::2], row[3::2]))) for row in rows]
    return out


@pytest.mark.parametrize("form,paired_widths", [(0, {32, 24}), (1, {24, 20})], ids=["fp32", "fp64"])
def test_width_by_what_fits(widths, form, paired_widths):
    seen = set()
    for width, smem in (w[form] for w in widths.values()):
        pairs = [b for b in smem if 2 * (smem[b] + 1024) <= 227 * 1024]
        alone = [b for b in smem if smem[b] <= 220 * 1024]
        # (a lone block is not given up for pairs of fewer than 16 cells)
        if max(alone) >= 16:
            pairs = [b for b in pairs if b >= 16]
        assert width == (max(pairs) if pairs else max(alone))
        seen.add((width, bool(pairs)))
    assert {w for w, paired in seen if paired} == paired_widths
    assert any(not paired for w, paired in seen)
