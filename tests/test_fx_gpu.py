"""Fixed-point stencil sums of the FP64 mode against the CPU oracle where the number format is
at its edges: fields at rest, large and small magnitudes, values just below a power of two,
wall ghosts above every interior value, strongly stretched grids, batches in both modes.

Tolerance: the FP64 path's bar of 1e-12 (norm-wise). The format keeps 2^-62 of a field's
largest value and the sums 2^-59 of their largest possible one, a few hundred times the
typical value of a resolved derivative: below 2^-50 = 1e-15 of it.
"""
import numpy as np
import pytest

from cudanavierstokes_gb300 import Solver
from cudanavierstokes_gb300.batch import Batch
from cudanavierstokes_gb300.params import Derived, channel_params, tgv_params
from tests._util import field_errors, smooth_random_state, state_errors, wall_state

pytestmark = pytest.mark.gpu

TOL64 = 1e-12


def _fields(p, rho, u, v, w, T):
    d = Derived.of(p)
    e = rho * d.Rgas * T / (p.gam - 1.0) + 0.5 * rho * (u * u + v * v + w * w)
    return [np.ascontiguousarray(a) for a in (rho, u, v, w, e)]


def _rest(oracle_mod):
    """A pressure wave at rest: every velocity zero, growing from the first stage on."""
    p = tgv_params(18).copy(my=14, mz=21)
    s = smooth_random_state(p, seed=3)
    z = np.zeros(p.shape)
    return p, _fields(p, s[0], z, z, z, 1.0 + 0.1 * s[1])


def _low_mach(oracle_mod):
    p = tgv_params(16).copy(Ma=0.01)
    return p, smooth_random_state(p, seed=4)


def _top_of_binade(oracle_mod):
    """The largest values of rho, u and w just below powers of two."""
    p = tgv_params(17).copy(my=13, mz=19, Ma=0.5)
    s = smooth_random_state(p, seed=5)
    r, u, w = s[0].copy(), s[1].copy(), s[3].copy()
    r[3, 4, 5] = r[7, 4, 5] = np.nextafter(2.0, 0.0)
    u[3, 4, 5], u[3, 4, 9] = np.nextafter(1.0, 0.0), -np.nextafter(1.0, 0.0)
    w[3, 4, 5], w[8, 4, 5] = np.nextafter(2.0, 0.0), np.nextafter(2.0, 0.0)
    return p, _fields(p, r, u, s[2], w, np.ones(p.shape))


def _hot_walls(oracle_mod):
    """T = 2 Tw - T at the ghosts far above the interior's largest T (and rho below)."""
    p = channel_params(21, 12, 14).copy(twall_bot=2.9, twall_top=1.7)
    s = wall_state(p, oracle_mod.Oracle(p).grid()["x"])
    return p, _fields(p, s[0], s[1], s[2], s[3], 0.6 + 0.05 * s[3])


def _stretched(oracle_mod):
    p = channel_params(40, 9, 10).copy(stretch=4.0, Re=200.0, stencil_visc=2)
    return p, wall_state(p, oracle_mod.Oracle(p).grid()["x"])


@pytest.mark.parametrize("make", [_rest, _low_mach, _top_of_binade, _hot_walls, _stretched])
def test_range_edges(gpu_lib, oracle_mod, make):
    p, f = make(oracle_mod)
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    s = Solver(p)
    s.copy_field_in(*f)
    if make is not _rest:   # (from rest the mass equation's RHS is rounding alone)
        errs = field_errors(s.calc_rhs(), o.rhs())
        assert max(errs) <= TOL64, errs
    o.run(3)
    s.run(3)
    errs = state_errors(s.copy_field_out(), o.get_state())
    assert max(errs) <= TOL64, errs


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("mx", [13, 33])
def test_batch_modes(gpu_lib, oracle_mod, mode, mx):
    """Odd edges (ghost cells beside interior ones) through the persistent and the concurrent mode."""
    p = tgv_params(mx).copy(my=11, mz=10)
    f = smooth_random_state(p, seed=mx)
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    o.run(3)
    b = Batch(precision=0)
    b.set_mode(mode)
    i = b.add(p, f, max_steps=8)
    b.step(3)
    errs = state_errors(b.fields(i), o.get_state())
    assert max(errs) <= TOL64, errs


@pytest.mark.parametrize("mx,my,mz", [(9, 8, 9), (33, 7, 38), (32, 8, 76), (32, 8, 77), (31, 9, 50), (65, 6, 29)])
@pytest.mark.parametrize("S,V", [(4, 4), (3, 1)])
def test_small_box_kernel(gpu_lib, oracle_mod, mx, my, mz, S, V):
    """Both sides of the switch between two threads and one thread per point (152 blocks of 32 x
    4 points: 32 x 8 x 76 is the last box below it), with ragged tiles, on channel walls."""
    if my < 2 * S:
        pytest.skip("fewer points than the stencil")
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


@pytest.mark.parametrize("V", [1, 4])
def test_dilatation_planes_per_block(gpu_lib, V):
    """FP32: boxes repeated along z take 1, 2 and 8 planes per block of the dilatation kernel (6
    tiles a plane, the last block ragged); each copy of the box has the same RHS bit for bit."""
    def rhs(r):
        p = tgv_params(33).copy(my=20, mz=14 * r, precision=1, stencil_visc=V)
        p = p.copy(Lz=p.Lz / 32 * r)
        s = Solver(p)
        s.copy_field_in(*[np.tile(f, (r, 1, 1)) for f in base])
        return s.calc_rhs()
    base = smooth_random_state(tgv_params(33).copy(my=20, mz=14), seed=3)
    one = rhs(1)
    for r in (8, 32):
        for a, b in zip(one, rhs(r)):
            assert np.array_equal(np.tile(a, (r, 1, 1)), b)
