"""Bytes of a first-order stage: no reconstruction, the averages once per cell
(and, above 38,912 faces, a row of 64 bytes per cell written and read), the
face geometry and flux, the update's rows."""

import pytest

import mallard_gb300 as mg
from cases import GAS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, side_rows", [(20, 0), (140, 128)])
def test_first_order_stage(n, side_rows):
    m = mg.Mesh.generate("cartesian", n, n, 1.0, 1.0)
    with mg.Solver(m, face_reconstruction="FO", boundaries=[dict(name=z, type="extrapolation") for z in m.zone_names[1:]],
                   **GAS) as s:
        _, stage = s.traffic_model()
    cells, faces = m.n_cells, len(m.zone_faces)
    assert (faces > 38912) == bool(side_rows)
    flux = cells * (32 + side_rows) + faces * (32 + 8 + 16 + 8 + 1)
    update = cells * (16 + 8 + 4 * 32) + faces * 2 * 32
    assert stage == flux + update
