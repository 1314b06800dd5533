"""phpc_tuning reports the tile width that the device calls take: 128 where the
modular scheme's rule narrows the table's 256 (n <= 128 on any machine)."""
import pytest

from test_digit_tuning import _tuning

Q13 = {"PHPC_MODULI": "13"}


@pytest.mark.parametrize("shape,bn", [((8000, 1000, 100), 128), ((2000, 2000, 128), 128), ((4096, 4096, 4096), 256)])
def test_modular_tile_width(built, shape, bn):
    assert _tuning([shape], **Q13)[0][:2] == (13, bn)
    assert _tuning([shape], **Q13, PHPC_OZAKI_BN="256")[0][:2] == (13, 256)
