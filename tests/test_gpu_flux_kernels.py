"""The FP64 face flux on both sides of its dispatch by size against the oracle.

Up to 38,912 face points the flux runs with one lane per side of a point, above
with one lane per point (and, at first order, each cell's states recovered
once): two statements of every boundary condition and Riemann solver, each
compared here, with every order of the reconstruction."""

import functools

import numpy as np
import pytest

import mallard_gb300 as mg
from cases import make_pair, perturbed
from test_gpu_fast import FAST_STAGE_TOL
from test_gpu_parity import STAGE_TOL, assert_close, tri_mesh

pytestmark = pytest.mark.gpu

LIMIT = 38912
# (reconstruction, order, n, points per face): the last mesh under the limit and the first above
SIZES = [("FO", 3, 113, 1), ("FO", 3, 114, 1), ("TENO", 1, 114, 1), ("TENO", 2, 114, 1), ("TENO", 3, 80, 2),
         ("TENO", 3, 81, 2)]
ALL_KINDS = {"left": "upt", "right": "p_out", "top": "symmetry", "bottom": "wall_adiabatic"}


@functools.lru_cache(maxsize=4)
def mesh_and_state(n):
    m = tri_mesh(n, seed=12)
    return m, perturbed(m, seed=9)[0]


@functools.lru_cache(maxsize=1)
def expected(recon, p, n, riemann, bcs):
    m, U = mesh_and_state(n)
    return make_pair(m, recon=recon, poly_order=p, riemann=riemann, variant="corrected", bcs=dict(bcs),
                     gpu=False)[1].calc_rhs(U)


def test_sizes_are_at_the_line():
    faces = {n: len(mesh_and_state(n)[0].zone_faces) for n in (113, 114, 80, 81)}
    assert faces[113] <= LIMIT < faces[114] and 2 * faces[80] <= LIMIT < 2 * faces[81]


@pytest.mark.parametrize("recon, p, n, nq", SIZES)
@pytest.mark.parametrize("riemann", ["Rusanov", "HLL", "HLLC"])
@pytest.mark.parametrize("bcs", ["all kinds", "extrapolation"])
@pytest.mark.parametrize("precision", ["fp64", "fp64_fast"])
def test_residual(recon, p, n, nq, riemann, bcs, precision):
    m, U = mesh_and_state(n)
    kinds = tuple((ALL_KINDS if bcs == "all kinds" else {z: "extrapolation" for z in ALL_KINDS}).items())
    s, _ = make_pair(m, recon=recon, poly_order=p, riemann=riemann, variant="corrected", bcs=dict(kinds),
                     precision=precision)
    with s:
        assert s.nq == nq
        R = s.calc_rhs(U)
    Ro = expected(recon, p, n, riemann, kinds)
    if precision == "fp64":
        assert_close(R, Ro, STAGE_TOL, min_exact=0.95, what=f"{recon} p={p} {riemann}")
    else:
        assert_close(R, Ro, FAST_STAGE_TOL, what=f"fast {recon} p={p} {riemann}")


@pytest.mark.parametrize("n", [113, 114])
@pytest.mark.parametrize("riemann", ["Rusanov", "HLL", "HLLC"])
def test_first_order_quads(n, riemann):
    """Quads with every kind of boundary: 113 x 171 has 38,930 faces, 113 x 170 under the limit."""
    m = mg.Mesh.generate("cartesian", 113, 171 if n == 114 else 170, 1.0, 1.0)
    assert (len(m.zone_faces) > LIMIT) == (n == 114)
    U = perturbed(m, seed=9)[0]
    s, oc = make_pair(m, recon="FO", riemann=riemann, bcs=ALL_KINDS)
    with s:
        R = s.calc_rhs(U)
    assert_close(R, oc.calc_rhs(U), STAGE_TOL, min_exact=0.99, what=f"quads {riemann}")
