"""pfa3d_footprint is the device memory that a 3D handle allocates."""
import pytest


@pytest.mark.parametrize("nx,ny,nz", [(3, 3, 3), (34, 35, 36), (66, 130, 19)])
def test_3d_footprint_is_the_handles_buffers(pfa, nx, ny, nz):
    ghost, cells = nx * ny * nz, (nx - 2) * (ny - 2) * (nz - 2)
    # the events (48 bytes) and their sort keys, four counters, the status and
    # call words, and the list of cells
    nuc = (48 + 8) * 2 ** 14 + 4 * 4 + 4 + 8 + 8 * max(1024, cells // 4)
    recs = (nx - 2 + 31) // 32 * 32 * (ny - 2) * (nz - 2)
    assert pfa.Grid3D.footprint((nz, ny, nx), "fp64") == 2 * 4 * ghost * 8 + nuc
    assert pfa.Grid3D.footprint((nz, ny, nx), "fp32") == 4 * ghost * 8 + 2 * recs * (16 + 8) + nuc
