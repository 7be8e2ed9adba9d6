"""The reference-arithmetic predictor divides by grid values through their reciprocals: every
quotient must be the rounded one, so the predicted velocities equal the oracle's bit for bit
on values of every size, zeros of both signs, denormals and infinities, and on spacings so
far apart that the divisors' reciprocals cannot be used."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(shape, kind, seed):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal(shape)
    if kind == "sizes":
        a = np.ldexp(a, rng.integers(-1060, 300, shape))
        pick = rng.integers(0, 12, shape)
        a[pick == 0] = 0.0
        a[pick == 1] = -0.0
    elif kind == "infinite":
        a[rng.integers(0, 300, shape) == 0] = np.inf
        a[rng.integers(0, 300, shape) == 0] = -np.inf
        a[rng.integers(0, 300, shape) == 0] = np.nan
    return np.asfortranarray(a)


@pytest.mark.parametrize("ab", [0, 1])
@pytest.mark.parametrize("kind", ["plain", "sizes", "infinite"])
@pytest.mark.parametrize("shape,scale", [((5, 4, 4), 1.0), ((33, 6, 7), 1.0), ((20, 31, 9), 1.0),
                                         ((12, 9, 10), 2.0 ** -230)])
def test_predictor_divides_exactly(ib3d, grids, oracle_mod, shape, scale, kind, ab):
    x, y, z = (grids.tanh_axis(n) * scale for n in shape)
    s = ib3d.Solver(x, y, z, ib3d.default_params(re=100.0, deltat=0.01, momentum=ab))
    o = oracle_mod.Oracle(x, y, z, 100.0, 0.01, momentum=ab)
    o.no_body()
    for k, f in enumerate(("u", "v", "w", "p", "ut", "vt", "wt")):
        a = _field(s.shape, kind, 10 + k)
        s.set_field(f, a)
        o.set_field(f, a)
    for _ in range(2):   # the second predictor of the Adams-Bashforth form reads the first one's terms
        for x in (s, o):
            (x.ns_momentum_ab if ab else x.ns_momentum)()
        for f in ("ut", "vt", "wt"):
            np.testing.assert_array_equal(s.get_field(f), o.get_field(f), f)
    s.close()


# nz: slabs of four planes that end full and one to three planes short
@pytest.mark.parametrize("ab", [0, 1])
@pytest.mark.parametrize("shape", [(5, 4, 4), (33, 6, 5), (20, 31, 6), (9, 14, 7), (130, 7, 12)])
def test_contracted_predictor_agrees_to_rounding(ib3d, grids, shape, ab):
    """150 operations on terms of at most ten times the largest result (time step 0.01, spacings
    of 1/200 and more): 150 * 2^-53 * 10 < 2e-13 of it; 1e-12 is allowed."""
    x, y, z = (grids.tanh_axis(n) for n in shape)
    s = ib3d.Solver(x, y, z, ib3d.default_params(re=100.0, deltat=0.01, momentum=ab))
    for k, f in enumerate(("u", "v", "w", "p")):
        s.set_field(f, _field(s.shape, "plain", 20 + k))
    out = []
    for precision in (ib3d.PREC_FP64, ib3d.PREC_FP32DC):
        s.set_params(precision=precision)
        for f in ("ut", "vt", "wt"):
            s.set_field(f, np.zeros(s.shape))
        (s.ns_momentum_ab if ab else s.ns_momentum)()
        (s.ns_momentum_ab if ab else s.ns_momentum)()
        out.append([s.get_field(f) for f in ("ut", "vt", "wt")])
    for ref, got in zip(*out):
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()
        assert np.any(got != 0.0)
    s.close()


@pytest.mark.parametrize("ab", [0, 1])
@pytest.mark.parametrize("kind", ["sizes", "infinite"])
def test_predictor_keeps_the_signs_of_zeros(ib3d, grids, oracle_mod, kind, ab):
    """Bit patterns, with one for all NaNs: fields of signed zeros almost everywhere, so that
    predicted values are zeros of both signs too."""
    x, y, z = (grids.tanh_axis(n) for n in (33, 12, 9))
    s = ib3d.Solver(x, y, z, ib3d.default_params(re=100.0, deltat=0.01, momentum=ab))
    o = oracle_mod.Oracle(x, y, z, 100.0, 0.01, momentum=ab)
    o.no_body()
    rng = np.random.default_rng(7)
    for k, f in enumerate(("u", "v", "w", "p", "ut", "vt", "wt")):
        a = _field(s.shape, kind, 40 + k)
        a = np.where(rng.integers(0, 40, s.shape) == 0, a, np.copysign(0.0, rng.standard_normal(s.shape)))
        a[:, :, :5] = np.copysign(0.0, -1.0)   # a region of negative zeros alone
        a = np.asfortranarray(a)
        s.set_field(f, a)
        o.set_field(f, a)

    def bits(a):
        return np.where(np.isnan(a), np.uint64(0x7FF8000000000000), a.view(np.uint64))
    for _ in range(2):
        for m in (s, o):
            (m.ns_momentum_ab if ab else m.ns_momentum)()
        for f in ("ut", "vt", "wt"):
            got, want = s.get_field(f), o.get_field(f)
            np.testing.assert_array_equal(bits(got), bits(want), f)
    inner = want[1:-1, 1:-1, 1:-1]
    assert np.any((inner == 0) & np.signbit(inner)) or np.any((inner == 0) & ~np.signbit(inner))
    s.close()
