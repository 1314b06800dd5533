"""CTA pairs are chosen by the call's own moduli: from 80 K-steps an SM on, where
the table names them (1024 x 2048 x 1024 has 54, 88 and 101 with 8, 13 and 15)."""
import pytest

from test_digit_tuning import _tuning


@pytest.mark.parametrize("moduli,cluster", [(8, 1), (10, 1), (12, 2), (13, 2), (15, 2)])
def test_pairs_by_moduli(built, tmp_path, moduli, cluster):
    table = tmp_path / "table.txt"
    table.write_text(f"{2 ** 62} 7 256 8 2 {moduli}\n")
    shapes = [(1024, 2048, 1024), (4096, 4096, 4096), (4096, 520, 4096)]
    got = _tuning(shapes, PHPC_TUNE_TABLE=str(table))
    assert [g[0] for g in got] == [moduli] * 3
    assert [g[2] for g in got] == [cluster, 2, 1]
