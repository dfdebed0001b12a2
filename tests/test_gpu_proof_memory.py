"""Tables of the central-decision proof are held where a kernel reads them: an
FP32 solver reads them from 100,000 cells."""

import pytest

import mallard_gb300 as mg
from cases import GAS

pytestmark = pytest.mark.gpu


def test_small_fp32_solver_holds_no_proof_tables():
    import torch
    held = []
    for n in ((223, 225), (223, 224), (223, 225)):  # the first one also loads the kernels
        m = mg.Mesh.generate("cartesian_tri", *n, 1.0, 1.0)
        free = torch.cuda.mem_get_info()[0]
        with mg.Solver(m, boundaries=[dict(name=z, type="extrapolation") for z in m.zone_names[1:]], precision="fp32",
                       teno_variant="corrected", **GAS):
            held.append((m.n_cells, free - torch.cuda.mem_get_info()[0]))
    (_, _), (small, a), (large, b) = held
    assert small < 100000 <= large
    assert b - a > 400 * small  # 492 bytes a cell in the larger one alone
