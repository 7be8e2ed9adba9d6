"""The sweep forms that a grid's size selects, against the one-array FP32 sweep
(sweep_kernel 1) or the oracle: all perform the same operations in the same order, so
the corrections agree bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _capped(ib3d, grids, shape, sweeps, b, **kw):
    """pc after `sweeps` FP32 sweeps (the solve stops at the cap; the residual goal is out of reach)."""
    x, y, z = (grids.tanh_axis(n) for n in shape)
    p = ib3d.default_params(re=100.0, deltat=1.0, omega=1.85, eps=1e-30, max_sweeps=sweeps)
    p.precision, p.criterion, p.inner_sweeps = ib3d.PREC_FP32DC, 1, 35
    for k, v in kw.items():
        setattr(p, k, v)
    s = ib3d.Solver(x, y, z, p)
    s.set_field("b", b)
    st = s.redblack_sor(allow_noconv=True)
    pc = s.get_field("pc")
    s.close()
    return st["sweeps"], pc


# sizes whose sweeps run on chip (blocks split both ways, along one axis, with several planes
# a thread) and beyond; odd nx (the second colour's rows end in the ghost cell), odd ny (a row pair's second row is
# the ghost row), nz no multiple of a slab; the last two exceed what the blocks hold on chip,
# and the last one streams its right-hand side and alternates the direction of its passes
@pytest.mark.parametrize("kernel,shape", [(0, (129, 21, 19)), (0, (37, 18, 45)), (0, (5, 4, 4)), (0, (7, 5, 301)),
                                          (0, (9, 203, 6)), (0, (126, 130, 97)), (3, (129, 21, 19)),
                                          (4, (67, 9, 11)), (0, (1201, 41, 78)), (0, (271, 225, 202))])
def test_packed_sweeps_match_the_padded_layout(ib3d, grids, kernel, shape):
    b = np.zeros(tuple(n + 2 for n in shape), order="F")
    b[1:-1, 1:-1, 1:-1] = np.random.default_rng(5).standard_normal(shape)
    want = _capped(ib3d, grids, shape, 75, b, sweep_kernel=1, smooth_sweeps=2, ramp_sweeps=5)
    got = _capped(ib3d, grids, shape, 75, b, sweep_kernel=kernel, smooth_sweeps=2, ramp_sweeps=5)
    assert got[0] == want[0]
    bad = np.argwhere(got[1] != want[1])
    assert bad.size == 0, f"{len(bad)} pc mismatches, first {bad[0]}"
    assert np.any(got[1] != 0.0)


def test_fused_sweep_still_needs_an_even_nx(ib3d, grids):
    b = np.zeros((23, 10, 10), order="F")
    with pytest.raises(ib3d.IB3DError) as e:
        _capped(ib3d, grids, (21, 8, 8), 10, b, sweep_kernel=2)
    assert e.value.code == ib3d.ERR_ARG
