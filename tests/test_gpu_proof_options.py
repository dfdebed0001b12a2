"""The proof of the central decision with the options that change its tables
(basis, cell quadrature), and the batch's default launch where it takes the
proof form."""

import numpy as np
import pytest

import mallard_gb300 as mg
from cases import BC_DATA, GAS, four_quadrant
from oracle import OracleCase, OracleMesh
from test_gpu_central import wavy
from test_gpu_parity import STAGE_TOL, assert_close

pytestmark = pytest.mark.gpu

# the last one's oscillation indicator is too close to singular for the proof:
# every cell runs the full kernel
OPTIONS = [("monomial", 1, 0), ("monomial", 2, 0), ("monomial", 3, 0), ("legendre", 3, 5), ("legendre", 2, 4),
           ("monomial", 3, 5), ("monomial", 3, 1)]


@pytest.mark.parametrize("basis, p, q_cell", OPTIONS)
@pytest.mark.parametrize("state", ["jump", "waves", "weak"])
def test_masks_and_face_values(basis, p, q_cell, state):
    m = mg.Mesh.generate("cartesian_tri", 23, 19, 1.0, 1.0)
    m.permute_cells(5)
    U = {"jump": four_quadrant, "waves": lambda x: wavy(x, 0.1), "weak": lambda x: wavy(x, 3e-6)}[state](m)[0]
    bcs = [dict(name=z, type="extrapolation", **BC_DATA["extrapolation"]) for z in m.zone_names[1:]]
    om = OracleMesh.from_arrays(m)
    oc = OracleCase(om, basis=basis, poly_order=p, q_cell=q_cell, **GAS)
    oc.set_teno_variant(1)
    for b in bcs:
        oc.add_boundary(m.zone_index(b["name"]), b["type"], ())
    with mg.Solver(m, basis_type=basis, basis_order=p, quadrature_order_cell=q_cell, teno_variant="corrected",
                   boundaries=bcs, **GAS) as s:
        F, M = s.calc_face_values(U, masks=True)
    Fo, Mo = oc.face_values(U, masks=True)
    np.testing.assert_array_equal(M, Mo)
    f = m.zone_faces
    assert_close(F[f][:, :, 0], Fo[f][:, :, 0], STAGE_TOL, min_exact=0.99, what=f"{basis} p={p} q={q_cell}")


@pytest.mark.parametrize("basis, q_cell", [("monomial", 0), ("legendre", 5), ("monomial", 1)])
def test_fp32_shapes(basis, q_cell):
    """The FP32 proof kernels against the direct kernel, whose tables are the same."""
    m = mg.Mesh.generate("cartesian_tri", 223, 225, 1.0, 1.0)
    bcs = [dict(name=z, type="extrapolation") for z in m.zone_names[1:]]
    with mg.Solver(m, basis_type=basis, quadrature_order_cell=q_cell, teno_variant="corrected", boundaries=bcs,
                   precision="fp32", **GAS) as s:
        for U in (wavy(m, 0.1)[0], four_quadrant(m)[0]):
            out = []
            for shape in (0, 4, 5, 6, 7):
                s.set_launch_shape(shape)
                out.append(s.calc_face_values(U, masks=True))
            for F, M in out[1:]:
                np.testing.assert_array_equal(M, out[0][1])
                np.testing.assert_array_equal(F, out[0][0])


def test_batch_default_launch_with_large_cases():
    """Cases of 25,312 cells on average (the batch's default is the proof form
    from 25,000) against the direct kernel."""
    from mallard_gb300.batch import Batch
    meshes = [mg.Mesh.generate("cartesian_tri", n, n, 1.0, 1.0) for n in (112, 114)]
    counts = [3, 1]
    assert 25000 <= sum(m.n_cells * c for m, c in zip(meshes, counts)) / 4 < 25500
    out = []
    for shape in (None, 0):
        with Batch(meshes, counts, boundaries=[dict(name=z, type="extrapolation") for z in meshes[0].zone_names[1:]],
                   teno_variant="robust", **GAS) as b:
            if shape is not None:
                b.set_launch_shape(shape)
            for g, m in enumerate(meshes):
                for i in range(counts[g]):
                    b.set_state(g, i, (four_quadrant(m) if i % 2 else wavy(m, 0.1, seed=i))[0])
            b.run(0.4, 4)
            flags, t = b.status()
            assert (flags == 0).all()
            out.append((t, [b.get_state(g, i)[0] for g in (0, 1) for i in range(counts[g])]))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for a, c in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, c)
