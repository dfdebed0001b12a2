"""Velocities recovered from the conserved state are quotients, not products
with a rounded reciprocal: a supersonic row of cells whose momenta are exact
multiples of their densities has fluxes that are exact whole numbers, in both
FP64 forms and on both sides of the face flux's dispatch by size."""

import numpy as np
import pytest

import mallard_gb300 as mg
from cases import GAS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "fp64_fast"])
@pytest.mark.parametrize("nx, ny", [(64, 1), (200, 120)])
@pytest.mark.parametrize("solver", ["HLL", "HLLC"])
def test_whole_number_mass_fluxes(solver, nx, ny, precision):
    m = mg.Mesh.generate("cartesian", nx, ny, float(nx), float(ny))  # unit cells
    col = np.round(m.cell_coords[:, 0] - 0.5).astype(int)
    r = np.random.default_rng(3)
    rho, u = r.integers(1, 500, nx).astype(float), np.full(nx, 7.0)
    # a reciprocal loses the velocity's last bit in some of the cells
    assert ((rho * u) * (1.0 / rho) != u).any()
    p = 0.25  # sound speeds under 0.6, contacts between the cells
    U = np.stack([rho, rho * u, 0 * rho, p / 0.4 + 0.5 * rho * u * u], 1)[col]
    bcs = [dict(name=z, type="extrapolation" if z in ("left", "right") else "symmetry") for z in m.zone_names[1:]]
    with mg.Solver(m, face_reconstruction="FO", riemann_solver=solver, boundaries=bcs, precision=precision, **GAS) as s:
        R = s.calc_rhs(U)[:, 0]
    flux = np.concatenate([rho[:1] * u[:1], rho * u])
    np.testing.assert_array_equal(R, (flux[:-1] - flux[1:])[col])
