"""Blocks fitted to the plane just above the two-threads-per-point switch, and the screened
time-step reduction where the screen cannot decide or the fastest point is the last."""
import numpy as np
import pytest

from cudanavierstokes_gb300 import Solver
from cudanavierstokes_gb300.params import Derived, channel_params, tgv_params
from tests._util import field_errors, smooth_random_state, state_errors, wall_state

pytestmark = pytest.mark.gpu

TOL64 = 1e-12   # the FP64 path's bar (norm-wise)


@pytest.mark.parametrize("mx,my,mz", [(25, 9, 90), (65, 8, 40), (75, 10, 33)])
@pytest.mark.parametrize("S,V", [(4, 4), (3, 1)])
def test_fitted_blocks(gpu_lib, oracle_mod, mx, my, mz, S, V):
    """25, 13 and 25 columns per block (the last warp ragged), more than 152 blocks: one thread a point."""
    p = channel_params(mx, my, mz).copy(stencil_size=S, stencil_visc=V)
    f = wall_state(p, oracle_mod.Oracle(p).grid()["x"])
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    s = Solver(p)
    s.copy_field_in(*f)
    errs = field_errors(s.calc_rhs(), o.rhs())
    assert max(errs) <= TOL64, errs
    o.run(2)
    s.run(2)
    errs = state_errors(s.copy_field_out(), o.get_state())
    assert max(errs) <= TOL64, errs


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("kind", ["cold", "last"])
def test_time_step_where_the_screen_is_at_its_limit(gpu_lib, oracle_mod, kind, prec):
    """`cold`: an internal energy below a tenth of the total at the fast points, which FP32 cannot
    tell from it closely enough. `last`: fluid at rest but for the last point of a ragged box."""
    p = tgv_params(13, Ma=8.0 if kind == "cold" else 0.1).copy(my=11, mz=10, cfl=0.05)   # (0.5: T < 0 after a step)
    d = Derived.of(p)
    one = np.ones(p.shape)
    if kind == "cold":
        u, v, w = smooth_random_state(p, seed=3)[1:4]
        u = 3.0 * u
    else:
        u, v, w = 0 * one, 0 * one, 0 * one
        v[-1, -1, -1] = 0.25
    e = d.Rgas / (p.gam - 1.0) * one + 0.5 * (u * u + v * v + w * w)
    o = oracle_mod.Oracle(p)
    o.set_state(one, u, v, w, e)
    o.run(1)
    s = Solver(p.copy(precision=prec))
    s.copy_field_in(one, u, v, w, e)
    s.run(1)
    a, b = s.scalars()["dt"], o.scalars()["dt"]
    assert abs(a - b) <= 1e-13 * b, (a, b)
