"""The digit scheme's tile width and cluster are its own, not the residue GEMM's.

The residue GEMM has a CTA per (tile, modulus) and takes 256-wide tiles and CTA
pairs where they suit it; the digit GEMM has a CTA per tile and keeps 128-wide
tiles up to m n k = 3.04e9 and single CTAs up to 2.43e10, and its table entry's
pairs above, whatever the shape. Read through phpc_tuning with PHPC_MODULI=0.
"""
import os
import subprocess
import sys
from pathlib import Path

import pytest

PKG = Path(__file__).resolve().parent.parent / "hpc-multigpu-matrixmult_gb300"

PROBE = """
import sys, ctypes as ct
L = ct.CDLL(sys.argv[1])
cfg = (ct.c_int * 10)()
for shape in sys.argv[2:]:
    assert L.phpc_tuning(*(int(x) for x in shape.split("x")), cfg) == 0
    print(cfg[0], cfg[2], cfg[4])
"""


def _tuning(shapes, **env):
    env = {**{k: v for k, v in os.environ.items() if not k.startswith("PHPC_")}, **env}
    r = subprocess.run([sys.executable, "-c", PROBE, str(PKG / "lib" / "libphpc_gemm.so"),
                        *("x".join(map(str, s)) for s in shapes)], env=env, capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    return [tuple(int(x) for x in line.split()) for line in r.stdout.splitlines()]


SHAPES = [((192, 320, 160), 128, 1), ((1024, 1024, 1024), 128, 1), ((1448, 1448, 1448), 128, 1),
          ((1449, 1449, 1449), 256, 1), ((2048, 2048, 2048), 256, 1), ((4096, 512, 4096), 256, 1),
          ((3000, 3000, 3000), 256, 2), ((8192, 520, 8192), 256, 2), ((4096, 4096, 4096), 256, 2),
          ((8192, 8192, 8192), 256, 1)]


def test_digit_scheme_keeps_its_tiles(built):
    got = _tuning([s for s, _, _ in SHAPES], PHPC_MODULI="0")
    assert got == [(0, bn, cluster) for _, bn, cluster in SHAPES]


@pytest.mark.parametrize("lines,want", [
    ("{0} 7 256 8 2 0\n", (256, 2)),                                # an entry of its own decides alone
    ("{0} 7 256 8 2 0\ndigits 1000 256 1\n", (256, 2)),             # no "digits" line covers it
    ("{0} 7 256 8 2 0\ndigits {0} 128 1\ndigits {0} 256 2\n", (128, 1)),  # the first that does
    ("{0} 7 128 8 1 13\ndigits {0} 512 1\ndigits {0} 256 3\n", (128, 1)),  # malformed lines are passed over
])
def test_digit_entries_of_a_table(built, tmp_path, lines, want):
    table = tmp_path / "table.txt"
    table.write_text(lines.format(2 ** 62))
    assert _tuning([(700, 700, 700)], PHPC_TUNE_TABLE=str(table), PHPC_MODULI="0") == [(0, *want)]


def test_environment_overrides(built):
    got = _tuning([(700, 700, 700)], PHPC_MODULI="0", PHPC_OZAKI_BN="256", PHPC_CLUSTER="2")
    assert got == [(0, 256, 2)]
