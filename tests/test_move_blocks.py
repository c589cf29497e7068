"""How the FP32 mover's blocks follow from the parcels and the faces they crossed:
one round of the resident blocks for ordinary populations, three for large ones
and for those that cross many faces."""
import pytest

from picfoam_gb300 import build, native


@pytest.mark.parametrize("parcels, faces, per_sm", [
    (1, 0.0, 5), (100_000, 2e4, 5), (1_000_000, 2e5, 5), (3_000_000, 7e5, 5), (10_000_000, 2.2e6, 5),
    (12_000_000, 0.0, 15), (26_000_000, 6e6, 15), (300_000, 6.4e6, 5), (1_000_000, 5.7e6, 5),
    (1_000_000, 2.1e7, 15), (1_638_400, 1.04e8, 15), (8_000_000, 4.5e7, 5)])
def test_blocks(parcels, faces, per_sm):
    build.build()
    assert native.load().picgpu_test_move_blocks(parcels, faces, 152) == per_sm * 152
