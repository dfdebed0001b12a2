"""The staged reconstruction shapes that the proof form's numbers cover on large
meshes (8-10): the direct kernel's bits with and without a selector, reachable by
number and by the autotuner."""

import ctypes as C

import numpy as np
import pytest

import mallard_gb300 as mg
from cases import GAS, four_quadrant
from mallard_gb300 import _native as N
from mallard_gb300.selector import Selector, default_weights_path
from test_gpu_central import shapes_agree, wavy

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, tuned", [((41, 39), 8), ((223, 225), 11)])
@pytest.mark.parametrize("learned", [False, True])
def test_staged_shapes(n, tuned, learned):
    m = mg.Mesh.generate("cartesian_tri", *n, 1.0, 1.0)
    m.permute_cells(5)
    with Selector() as sel:
        sel.load(default_weights_path())
        attach = (lambda s: s.attach_selector(sel, threshold=0.9)) if learned else None
        for U in (wavy(m, 0.05)[0], four_quadrant(m)[0]):
            shapes_agree(m, U, (8, 9, 10), attach=attach, teno_variant="robust")
    with mg.Solver(m, boundaries=[dict(name=z, type="extrapolation") for z in m.zone_names[1:]], precision="fp32",
                   teno_variant="robust", **GAS) as s:
        s.set_state(four_quadrant(m)[0])
        best, ms = s.autotune()
        assert (ms > 0).sum() == tuned and (ms[:tuned] > 0).all() and ms[best] == ms[:tuned].min()
        with pytest.raises(RuntimeError, match="out of range"):
            s.set_launch_shape(11)
        # the entry that knows eight shapes writes eight times and picks among them
        eight, first = np.full(11, -1.0), C.c_int(-1)
        N.check(N.lib().mgpu_autotune(s._h, N.ptr(eight), C.byref(first)))
        assert (eight[:8] > 0).all() and (eight[8:] == -1.0).all()
        assert 0 <= first.value < 8 and eight[first.value] == eight[:8].min()
