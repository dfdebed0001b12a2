"""HLL and HLLC fluxes across contacts and shear layers whose pressure and
normal velocity jumps are rounding noise.  The two-rarefaction star pressure is
its own rounding noise there and the FP64 path may leave it out where the flux
cannot see it; HLL, which spreads the whole jump of the state over its waves,
does see it across a contact.  Against the oracle, which evaluates the
reference's formula.

Tolerance, in units of rho (|u| + a) to the component's power: the GPU's and the
C library's pow() differ by 2 ulps at most, the estimate takes three of them
and a seventh power, 2e-15 of the pressure; a wave speed moves by 0.43 of that,
the flux by a quarter of a wave speed's change times the jump: under 1e-15, and
a few ulps of the sums."""

import numpy as np
import pytest

import mallard_gb300 as mg
from cases import GAS, make_pair
from oracle import Oracle
from test_gpu_parity import tri_mesh

pytestmark = pytest.mark.gpu

TOL = 2e-15


@pytest.mark.parametrize("solver", ["HLL", "HLLC"])
@pytest.mark.parametrize("kind", ["contact", "shear", "both"])
@pytest.mark.parametrize("noise", [1e-13, 1e-12, 1e-11])
def test_flux(solver, kind, noise):
    r = np.random.default_rng(5)
    n = 1000
    th = r.uniform(0, 2 * np.pi, n)
    nn = np.stack([np.cos(th), np.sin(th)], 1)
    rho_l, p_l = r.uniform(0.2, 3, n), r.uniform(0.1, 3, n)
    rho_r = rho_l * (1.0 if kind == "shear" else np.exp(r.uniform(-1.35, 1.35, n)))
    p_r = p_l * (1 + noise * r.uniform(-0.4, 0.4, n))
    a_l, a_r = np.sqrt(1.4 * p_l / rho_l), np.sqrt(1.4 * p_r / rho_r)
    u_l = r.uniform(-0.5, 0.5, (n, 2)) * a_l[:, None]
    u_r = u_l + (noise * r.uniform(0, 1, n) * np.minimum(a_l, a_r))[:, None] * nn
    if kind != "contact":
        u_r += (r.uniform(-1, 1, n) * a_l)[:, None] * np.stack([-nn[:, 1], nn[:, 0]], 1)
    g = np.full(n, 1.4)
    args = (nn, rho_l, u_l, p_l, g, 3.5 * p_l / rho_l, rho_r, u_r, p_r, g, 3.5 * p_r / rho_r)
    F = mg.riemann_flux(solver, *args)
    o = Oracle()
    Fo = np.array([o.riemann_flux(solver, *(x[i] for x in args)) for i in range(n)])
    c = np.maximum(a_l, a_r) + np.sqrt(np.maximum((u_l ** 2).sum(1), (u_r ** 2).sum(1)))
    scale = np.maximum(rho_l, rho_r)[:, None] * np.stack([c, c * c, c * c, c ** 3], 1)
    assert (np.abs(F - Fo) / scale).max() <= TOL


@pytest.mark.parametrize("precision", ["fp64", "fp64_fast"])
@pytest.mark.parametrize("n", [24, 120])
@pytest.mark.parametrize("solver", ["HLL", "HLLC"])
def test_residual(solver, n, precision):
    """The face flux kernels (both sides of their dispatch by size) on cells of
    random density at one pressure and velocity."""
    m = tri_mesh(n, seed=6)
    r = np.random.default_rng(7)
    noise = lambda: 1e-11 * r.uniform(-0.35, 0.35, m.n_cells)  # noqa: E731
    rho = 1.5 * np.exp(r.uniform(-0.65, 0.65, m.n_cells))
    U, _ = mg.state_from_primitives(rho, 0.3 + noise(), -0.2 + noise(), 0.8 * (1 + noise()), **GAS)
    s, oc = make_pair(m, recon="FO", riemann=solver, precision=precision)
    with s:
        R = s.calc_rhs(U)
    Ro = oc.calc_rhs(U)
    c = np.sqrt(1.4 * 0.8 / rho.min()) + 0.37
    # three faces of a cell, each off by TOL (the fast form's own rounding: 20
    # ulps a flux), over the volume h^2 / 2 with faces of h, h and 1.42 h
    tol = TOL if precision == "fp64" else 20 * 2.3e-16
    scale = rho.max() * np.array([c, c * c, c * c, c ** 3]) * 3.42 * 2 * n
    assert (np.abs(R - Ro) / scale).max() <= tol
