"""Batches of uneven members: the persistent kernel, whose later phases read what earlier ones of
the same launch wrote, against the members' own kernels; the member that a failing step names.
"""
import numpy as np
import pytest

from cudanavierstokes_gb300.batch import Batch
from cudanavierstokes_gb300.native import CnsError
from cudanavierstokes_gb300.params import channel_params, tgv_params
from tests._util import smooth_random_state, wall_state

pytestmark = pytest.mark.gpu


def _members(oracle_mod):
    """Edges whose ghost cells share memory sectors with interior ones (13, 33), walls, an even box."""
    ps = [tgv_params(13).copy(my=11, mz=10), tgv_params(33).copy(my=9, mz=12), channel_params(21, 10, 9),
          tgv_params(32).copy(my=8, mz=9, Ma=0.5)]
    return [(p, smooth_random_state(p, seed=q) if p.periodic_x else wall_state(p, oracle_mod.Oracle(p).grid()["x"]))
            for q, p in enumerate(ps)]


def test_fp64_modes_agree_bit_for_bit(gpu_lib, oracle_mod):
    """The FP64 sums are integers, the same in both modes, and the rest of a point's arithmetic is
    shared: the states are equal to the last bit."""
    out = []
    for mode in (0, 1):
        b = Batch(precision=0)
        b.set_mode(mode)
        ids = [b.add(p, f, max_steps=16) for p, f in _members(oracle_mod)]
        b.step(12)
        out.append([b.fields(i) for i in ids])
    for a, c in zip(*out):
        for x, y in zip(a, c):
            assert np.isfinite(x).all()
            assert np.array_equal(x, y)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("mode", [0, 1])
def test_non_finite_member_is_named(gpu_lib, prec, mode):
    """Of three members the middle one runs at a CFL number far beyond the scheme's limit."""
    b = Batch(precision=prec)
    b.set_mode(mode)
    ids = []
    for q in range(3):
        p = tgv_params(16, precision=prec).copy(cfl=50.0 if q == 1 else 0.5)
        ids.append(b.add(p, smooth_random_state(p, seed=q), max_steps=32))
    with pytest.raises(CnsError) as e:
        b.step(20)
    assert e.value.code == 4 and f"batch member {ids[1]}:" in str(e.value)
    for i in (ids[0], ids[2]):
        assert all(np.isfinite(f).all() for f in b.fields(i))
