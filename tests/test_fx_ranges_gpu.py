"""The FP64 mode's right-hand side at the limits of its fixed-point sums."""
import numpy as np
import pytest

from cudanavierstokes_gb300 import Solver
from cudanavierstokes_gb300.batch import Batch
from cudanavierstokes_gb300.params import Derived, boundary_layer_params
from tests._util import field_errors, state_errors

pytestmark = pytest.mark.gpu

TOL64 = 1e-12   # the FP64 path's bar (norm-wise)


def _energy(p, rho, u, v, w, T):
    return rho * Derived.of(p).Rgas * T / (p.gam - 1.0) + 0.5 * rho * (u * u + v * v + w * w)


def _saw_tooth(S):
    """A boundary layer on a uniform grid with nearly the largest difference of theta across an
    extrapolated end that fields and ghosts of one size can give (7.2 of at most 9 times one
    direction's largest part): zero in the last plane, in the planes before it u along x and v
    along y with the signs of the first-derivative weights about a point, alternating with the
    plane, w along z with those signs about the last plane. The spacing makes theta's scale factor
    just less than a power of two."""
    n = {4: 840, 2: 12}[S]
    h = 2.0 ** np.ceil(np.log2(n)) / (1.99 * n)   # (1/h) / n = 1.99 times a power of two
    p = boundary_layer_params(17, 16, 15).copy(stencil_size=S, stencil_visc=S, nonuniform_x=0, perturbed=0, Re=10.0)
    p = p.copy(Lx=p.mx * h, Ly=p.my * h, Lz=p.mz * h)
    sign = {4: [1, -1, 1, -1], 2: [1, -1]}[S]
    u, v, w = np.zeros(p.shape), np.zeros(p.shape), np.zeros(p.shape)
    amp = np.zeros(p.mz)
    for m in range(1, 9):
        amp[-1 - m] = (-1.0) ** m
    for l, s in enumerate(sign, 1):
        u[:, :, 6 + l], u[:, :, 6 - l] = s, -s
        v[:, 8 + l, :], v[:, 8 - l, :] = s, -s
        w[p.mz - 1 - l] = -0.999 * s
    u, v = (0.999 * amp[:, None, None] * f for f in (u, v))
    one = np.ones(p.shape)
    return p, [one, u, v, w, _energy(p, one, u, v, w, one)]


@pytest.mark.parametrize("S", [4, 2])
def test_dilatation_at_extrapolated_ends(gpu_lib, oracle_mod, S):
    p, f = _saw_tooth(S)
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    s = Solver(p)
    s.copy_field_in(*f)
    errs = field_errors(s.calc_rhs(), o.rhs())
    assert max(errs) <= TOL64, errs
