"""The search's FP32 filter (groups of elements by their spheres, then elements by their
distance) must leave the reference's nearest element, bit for bit, whatever the mesh's
size, place and ties."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_parity import _same

pytestmark = pytest.mark.gpu


# 20 elements (one group, not full) to 20,480 (groups of 96); the body centred, where cells lie
# at equal distances from several elements, and off the centre; a grid far from the origin,
# where the coordinates have few digits left for the distances
@pytest.mark.parametrize("sub,shift,far", [(0, 0.0, 0.0), (1, 0.0, 0.0), (2, 0.013, 0.0), (3, 0.0, 0.0), (5, 0.0, 0.0),
                                           (3, 0.021, 4096.0), (2, -0.017, 1.0e9)])
def test_nearest_elements_match_the_oracle(ib3d, grids, oracle_mod, sub, shift, far):
    cs = grids.case("tiny")
    nodes, tris = grids.icosphere(sub, 0.5)
    nodes = nodes + shift * np.array([1.0, -0.5, 0.25]) + far
    x, y, z = cs.x + far, cs.y + far, cs.z + far
    s = ib3d.Solver(x, y, z, ib3d.default_params(re=cs.re, deltat=cs.dt))
    o = oracle_mod.Oracle(x, y, z, cs.re, cs.dt)
    for m in (s, o):
        m.set_mesh(nodes, tris)
    assert s.search(cs.box) == o.search(cs.box)
    got, want = s.get_search(), o.get_search()
    for key in ("cell", "ib", "nelp", "normdis"):
        _same(got[key], want[key], key)
    # a smaller mesh after a larger one, in the room that the larger one left
    nodes, tris = grids.icosphere(1, 0.4)
    for m in (s, o):
        m.set_mesh(nodes + far, tris)
    assert s.search(cs.box) == o.search(cs.box)
    got, want = s.get_search(), o.get_search()
    for key in ("cell", "ib", "nelp", "normdis"):
        _same(got[key], want[key], key)
    s.close()
