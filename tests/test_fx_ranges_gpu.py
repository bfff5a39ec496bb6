"""The FP64 mode's right-hand side at the limits of its fixed-point sums."""
import numpy as np
import pytest

from cudanavierstokes_gb300 import Solver
from cudanavierstokes_gb300.params import Derived, boundary_layer_params, tgv_params
from tests._rhs_ref import derived, rhs
from tests._util import field_errors

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
