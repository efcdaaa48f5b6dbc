"""The tile size of the face passes: tiles smaller than the largest size all run at once, whatever the species
count leaves resident, and no size is larger than that asks for (tests/tile_rule_check.cpp, compiled with g++)."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
SPECIES = [0, 2, 3, 5, 9, 16, 64, 128]
CELLS = [1, 31, 500, 9471, 9472, 9473, 14208, 14209, 18944, 18945, 28416, 28417, 30000, 37888, 37889, 75776, 75777, 2_000_000, 3_000_000_000]


def test_small_tiles_run_in_one_wave(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    exe = tmp_path / "tile_rule_check"
    subprocess.run([gxx, "-std=c++17", "-I", str(ROOT / "ablate_b200" / "csrc"), "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "tile_rule_check.cpp"), "-o", str(exe)], check=True)
    cases = [(n, ns, sm) for n in CELLS for ns in SPECIES for sm in (148, 20)]
    out = subprocess.run([str(exe), *(str(x) for c in cases for x in c)], capture_output=True, text=True, check=True).stdout.split()
    for (n, ns, sm), tile, ctas in zip(cases, map(int, out[0::2]), map(int, out[1::2])):
        top = 128 if ns else 256
        assert 32 <= tile <= top and top % tile == 0
        assert ctas == (4 if ns <= 2 else 3 if ns <= 5 else 2)  # the register budgets of MinBlocks
        if tile < top:
            assert -(-n // tile) <= ctas * sm, (n, ns, sm, tile)
        if tile > 32:
            assert -(-n // (tile // 2)) > ctas * sm, (n, ns, sm, tile)
