"""Geometries with more lines than 32-bit numbers hold are refused before anything is written."""
import pytest

pytestmark = pytest.mark.gpu


def test_more_lines_than_32_bits_find_no_memory(omni):
    """64^3 cells, lines a hundredth of a cell apart: 5e7 to 7e7 lines a direction, 80 directions."""
    with pytest.raises(omni.Omni3DError) as e:
        omni.Omni3D((64, 64, 64), 1.0, omni.icosphere(3)[:80], line_spacing=0.01)
    assert e.value.code == -4 and "2^32 lines" in str(e.value)
    # the device is as before
    with omni.Omni3D((64, 64, 64), 1.0, omni.icosphere(2), line_spacing=0.5) as s:
        assert s.geometry_info()["walk_errors"] == 0
