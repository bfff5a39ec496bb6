"""The FP64 mode's right-hand side at the limits of its fixed-point sums."""
import numpy as np
import pytest

from cudanavierstokes_gb300 import Solver
from cudanavierstokes_gb300.batch import Batch
from cudanavierstokes_gb300.native import CnsError
from cudanavierstokes_gb300.params import Derived, boundary_layer_params, channel_params, tgv_params
from tests._rhs_ref import derived, rhs
from tests._util import field_errors, smooth_random_state, state_errors

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


def _uniform_pressure(p, u, v, w):
    """rho = 1 and an internal energy of 64, with velocities whose squares the energy holds exactly: the
    recovered T, p and mu are the same number at every point, and a small component's equation is its own terms alone."""
    one = np.ones(p.shape)
    f = [one, *(np.ascontiguousarray(a * one) for a in (u, v, w))]
    return f + [64.0 + 0.5 * (f[1] * f[1] + f[2] * f[2] + f[3] * f[3])]


def _modes(p, rng, n=3, along=(1, 1, 1)):
    z, y, x = np.meshgrid(*(2 * np.pi * (np.arange(m) + 0.5) / m for m in p.shape), indexing="ij")
    f = np.zeros(p.shape)
    for _ in range(n):
        k, ph = rng.integers(1, 3, size=3), rng.uniform(0, 2 * np.pi, size=3)
        for a, q, c in zip((x, y, z), range(3), along):
            f += c * rng.uniform(0.1, 0.3) * np.sin(k[q] * a + ph[q])
        f += rng.uniform(-0.3, 0.3) * np.sin(along[0] * k[0] * x + ph[0]) * np.sin(along[2] * k[2] * z + ph[2]) * (
            np.cos(k[1] * y + ph[1]) if along[1] else 1.0)
    return f


def _grain(f, bits):
    return np.round(f * 2.0 ** bits) * 2.0 ** -bits


def _small_component(kind):
    """`thin`: a shear layer with a wall-normal spacing 24 and 96 times finer than the others and
    cross velocities 2^-10 of the stream. `span`: a two-dimensional flow with a spanwise velocity
    2^-15 of it."""
    p = tgv_params(16).copy(my=16, mz=24, Re=100.0, viscexp=1.0)
    p = p.copy(Ma=float(np.sqrt(1.0 / (p.gam * (p.gam - 1.0) * 64.0))))   # T = 1
    rng = np.random.default_rng(5)
    if kind == "thin":
        p = p.copy(Lx=p.Lz * 16 / 24 / 96, Ly=p.Lz * 16 / 24 / 4)
        u, v = (_grain(_modes(p, rng), 10) * 2.0 ** -10 for _ in range(2))
        w = _grain(1.0 + 0.1 * _modes(p, rng), 20)
    else:
        u, w = (_grain(0.5 * _modes(p, rng, along=(1, 0, 1)), 10) for _ in range(2))
        v = _grain(_modes(p, rng), 7) * 2.0 ** -15
    return p, _uniform_pressure(p, u, v, w)


@pytest.mark.parametrize("kind", ["thin", "span"])
def test_small_components_keep_their_own_scale(gpu_lib, kind):
    """Each equation against the same sums in extended precision, relative to its own maximum: no
    further off than twice the sums in plain FP64 are, or than 8 roundings of that maximum."""
    p, f = _small_component(kind)
    t = derived(p, f, np.float64)[4]
    assert (t == t.flat[0]).all()   # the state is what it is meant to be
    exact = rhs(p, f)
    plain = field_errors(rhs(p, f, np.float64), exact)
    s = Solver(p)
    s.copy_field_in(*f)
    errs = field_errors(s.calc_rhs(), exact)
    assert all(a <= max(2 * b, 8 * 2.0 ** -53) for a, b in zip(errs, plain)), (errs, plain)


def _local_error(A, B):
    """The largest error of each field relative to its largest value within two points."""
    out = []
    for a, b in zip(A, B):
        scale = np.abs(np.asarray(b))
        for axis in range(3):
            scale = np.max([np.roll(scale, s, axis) for s in range(-2, 3)], axis=0)
        out.append(float(np.max(np.abs(a - b) / scale)))
    return out


def _spot(p, peak, width):
    z, y, x = np.meshgrid(*((np.arange(n) + 0.5) / n for n in p.shape), indexing="ij")
    return 1.0 + (peak - 1.0) * np.exp(-((x - 0.5) ** 2 + (y - 0.5) ** 2 + (z - 0.5) ** 2) / width)


def _uneven(kind, p):
    """rho, u, v, w, T with a hot spot (density or pressure even), one outlier cell, or a jet far
    above the speed of sound beside fluid almost at rest."""
    q = [smooth_random_state(p, seed=n) for n in (3, 4)]
    r, u, v, w = q[0][:4]
    T = np.ones(p.shape)
    if kind == "hot":
        T = _spot(p, 1e3, 0.012)
    elif kind == "pressure":
        T, r = _spot(p, 1e6, 0.008), np.ones(p.shape)
    elif kind == "density":
        r = _spot(p, 1e4, 0.008)
        T = 1.0 / r
    elif kind == "cell":
        r = r.copy()
        r[5, 6, 7] *= 1e-5
    else:
        u = u * 1e-3 + 300.0 * (_spot(p, 2.0, 0.008) - 1.0)
    return [r, u, v, w, _energy(p, r, u, v, w, T)]


@pytest.mark.parametrize("kind", ["hot", "pressure", "density", "cell", "jet"])
@pytest.mark.parametrize("n", [(16, 16, 24), (40, 33, 24)])
def test_uneven_fields_keep_their_quiet_regions(gpu_lib, kind, n):
    """Values far below a field's maximum, point by point, against extended precision: no further off
    than four times the sums in plain FP64 are. (Both sizes of the RHS kernel.)"""
    p = tgv_params(n[0]).copy(my=n[1], mz=n[2], Re=100.0, Ma=0.3, viscexp=0.7)
    f = _uneven(kind, p)
    exact = rhs(p, f)
    plain = _local_error(rhs(p, f, np.float64), exact)
    s = Solver(p)
    s.copy_field_in(*f)
    errs = _local_error(s.calc_rhs(), exact)
    assert all(a <= 4 * b for a, b in zip(errs, plain)), (errs, plain)


@pytest.mark.parametrize("which", [0, 1])
def test_magnitudes_beyond_the_formats_range(gpu_lib, oracle_mod, which):
    """Densities of 2^310 and 2^-310 with everything else of order one: a step and the dissipation."""
    p = tgv_params(16).copy(my=9, mz=11, Re=1e3)
    f = smooth_random_state(p, seed=6)
    scale = 2.0 ** (310 if which == 0 else -310)
    f = [f[0] * scale, f[1], f[2], f[3], f[4] * scale]
    if which == 1:
        p = p.copy(Re=1e3 / scale)   # mu with it
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


def test_dissipation_of_large_velocities(gpu_lib, oracle_mod):
    """Velocities of 2^305 (and T to match): the dissipation's gradients beyond the format's range."""
    p = tgv_params(16).copy(my=9, mz=11)
    f = smooth_random_state(p, seed=7)
    s305 = 2.0 ** 305
    f = [f[0] * 2.0 ** -300, f[1] * s305, f[2] * s305, f[3] * s305, f[4] * 2.0 ** 310]
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    s = Solver(p)
    s.copy_field_in(*f)
    a, b = s.dissipation(), o.dissipation()
    assert abs(a["enstrophy"] - b["enstrophy"]) <= 1e-12 * abs(b["enstrophy"])


def test_a_failing_point_spoils_its_neighbourhood_alone(gpu_lib, oracle_mod):
    """A cell that the first stage drives to a negative temperature: NaN spreads by the stencils of the
    stages that follow, the far end of the box goes on as in the oracle."""
    p = tgv_params(96).copy(my=9, mz=9, cfl=60.0, viscexp=0.7, Ma=0.5)
    p = p.copy(Lx=p.Lx * 10)
    one = np.ones(p.shape)
    T = one.copy()
    T[4, 4, 10] = 50.0
    f = [one, 0 * one, 0 * one, 0 * one, _energy(p, one, 0 * one, 0 * one, 0 * one, T)]
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    o.run(1)
    s = Solver(p)
    s.copy_field_in(*f)
    with pytest.raises(CnsError) as e:
        s.run(1)
    assert e.value.code == 4
    got, want = s.copy_field_out(), o.get_state()
    assert any(np.isnan(a).any() for a in want)
    for a, b in zip(got, want):
        assert np.isfinite(b[:, :, 50:80]).all()
        np.testing.assert_allclose(a[:, :, 50:80], b[:, :, 50:80], rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("kind", ["channel", "bl"])
def test_uneven_fields_at_walls_and_open_ends(gpu_lib, oracle_mod, kind):
    """FP64 sums on a stretched grid with wall images and with extrapolated ones, over some steps in
    which the box calms down or not."""
    if kind == "channel":
        p = channel_params(21, 12, 14).copy(Re=200.0)
    else:
        p = boundary_layer_params(18, 10, 150).copy(pert_amp1=0.01)
    f = smooth_random_state(p, seed=8)
    T = _spot(p, 40.0, 0.02)
    f[4] = _energy(p, *f[:4], T)
    o = oracle_mod.Oracle(p)
    o.set_state(*f)
    s = Solver(p)
    s.copy_field_in(*f)
    errs = field_errors(s.calc_rhs(), o.rhs())
    assert max(errs) <= TOL64, errs
    o.run(4)
    s.run(4)
    errs = state_errors(s.copy_field_out(), o.get_state())
    assert max(errs) <= TOL64, errs


@pytest.mark.parametrize("mode", [0, 1])
def test_uneven_member_of_a_batch(gpu_lib, oracle_mod, mode):
    """Beside an even member: each by its own rule."""
    b = Batch(precision=0)
    b.set_mode(mode)
    ids, want = [], []
    for q in range(2):
        p = tgv_params(13 + 20 * q).copy(my=10, mz=9, Re=100.0, Ma=0.3, viscexp=0.7)
        f = smooth_random_state(p, seed=9)
        if q == 0:
            f[4] = _energy(p, *f[:4], _spot(p, 40.0, 0.05))
        o = oracle_mod.Oracle(p)
        o.set_state(*f)
        o.run(3)
        want.append(o.get_state())
        ids.append(b.add(p, f, max_steps=8))
    b.step(3)
    for i, x in zip(ids, want):
        errs = state_errors(b.fields(i), x)
        assert max(errs) <= TOL64, errs
