"""The one-launch boundary conditions on the smallest and on ragged grids, where the faces'
edges and corners make up most of the cells, and the drag/lift sums in either order."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import _same

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("outlet", [0, 1])
@pytest.mark.parametrize("shape", [(5, 4, 4), (6, 5, 4), (33, 6, 7), (8, 130, 5)])
def test_velocity_bc_on_random_fields_bit_exact(ib3d, grids, oracle_mod, shape, outlet):
    x, y, z = (grids.tanh_axis(n) for n in shape)
    s = ib3d.Solver(x, y, z, ib3d.default_params(re=100.0, deltat=0.01, outlet=outlet))
    o = oracle_mod.Oracle(x, y, z, 100.0, 0.01, outlet=outlet)
    o.no_body()
    rng = np.random.default_rng(3)
    for f in ("u", "v", "w", "ut", "vt", "wt"):
        a = np.asfortranarray(rng.standard_normal(s.shape))
        s.set_field(f, a)
        o.set_field(f, a)
    assert s.calculate_uc() == o.calculate_uc()
    for _ in range(2):
        s.velocity_bc()
        o.velocity_bc()
    for f in ("ut", "vt", "wt"):
        _same(s.get_field(f), o.get_field(f), f)
    s.close()


@pytest.mark.parametrize("sub", [0, 2, 4])
def test_drag_sums_in_tree_order_agree_with_the_serial_ones(ib3d, grids, sub):
    """20, 320 and 5,120 terms a sum. A sum of n terms is off by at most n 2^-53 times the sum of
    their sizes in any order; the coefficients divide by areas of the body's own size."""
    import dataclasses
    cs = dataclasses.replace(grids.case("tiny"), subdivisions=sub)
    s = ib3d.setup_case(cs)
    rng = np.random.default_rng(1)
    for f in ("ut", "vt", "wt", "p"):
        s.set_field(f, np.asfortranarray(rng.standard_normal(s.shape)))
    serial = s.stress(True)
    for precision in (ib3d.PREC_FP32DC, ib3d.PREC_FP64_FAST):
        s.set_params(precision=precision)
        tree = s.stress(False)
        n = 20 * 4 ** sub
        assert np.max(np.abs(tree - serial)) <= 2 * n * 2.0 ** -53 * 100.0, (tree, serial)
    s.close()
