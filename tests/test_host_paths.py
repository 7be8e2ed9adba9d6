"""Host code that a GPU test cannot reach -- allocations that fail, launches of several threads
that interleave -- on a CUDA runtime that runs no kernel (fake_cuda.cpp)."""
from __future__ import annotations

import ctypes as C
import pathlib
import subprocess

import numpy as np
import pytest


@pytest.fixture(scope="session")
def fake_path(ib3d, tmp_path_factory):
    pkg = pathlib.Path(ib3d.__file__).resolve().parent
    from ib3d_gpu_gb300 import buildlib
    objs = [pkg / "_build" / (pathlib.Path(s).stem + ".o") for s in buildlib.SOURCES]
    newest = max(f.stat().st_mtime for f in buildlib.CSRC.iterdir())
    if not all(o.exists() and o.stat().st_mtime >= newest for o in objs):
        ib3d.build()
    out = tmp_path_factory.mktemp("fake") / "libib3d_fake.so"
    include = pathlib.Path(buildlib.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-O1", "-Wl,-Bsymbolic", "-Wl,--no-undefined", "-I",
                    str(include), "-I", str(buildlib.CSRC), "-o", str(out),
                    str(pathlib.Path(__file__).resolve().parent / "fake_cuda.cpp"), *map(str, objs)], check=True)
    return out


@pytest.fixture
def fake(ib3d, fake_path, monkeypatch):
    """The package on the library linked with the fake runtime."""
    monkeypatch.setattr(ib3d, "_lib", None)
    monkeypatch.setattr(ib3d, "LIB_PATH", fake_path)
    L = ib3d.lib()
    L.fake_launches.restype = C.c_char_p
    L.fake_quad_item.restype = C.c_uint
    L.fake_launches()
    return L


def _solver(ib3d, grids, shape, precision=0, **kw):
    p = ib3d.default_params(deltat=1.0, omega=1.7, eps=1e-6, max_sweeps=1000, precision=precision, criterion=1, **kw)
    return ib3d.Solver(*(grids.tanh_axis(n) for n in shape), p)


def test_shared_memory_limits_never_fall(ib3d, grids, fake):
    """A kernel's limit of dynamic shared memory holds for all contexts and threads: a launch that
    lowered it could have another thread's refused between its own two calls."""
    before = fake.fake_lowered(), fake.fake_refused()
    for shape in ((96, 64, 64), (24, 24, 24), (100, 75, 51), (5, 4, 4)):
        for precision in (ib3d.PREC_FP64, ib3d.PREC_FP32DC, ib3d.PREC_FP64_FAST):
            with _solver(ib3d, grids, shape, precision) as s:
                s.redblack_sor()
    net = ib3d.Net(seed=1)
    for size in (32, 4):
        x = np.zeros((1, size, size, size, 4), np.float32)
        net.loss_grad(x, x[..., 0])
    net.close()
    names = fake.fake_launches().decode()
    for kernel in ("k_resident32", "k_resident64", "k_conv3", "k_wgrad_tc"):
        assert kernel in names
    assert (fake.fake_lowered(), fake.fake_refused()) == before


@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_failed_allocation_of_one_form_leaves_the_others_sound(ib3d, grids, fake, nth):
    """The on-chip forms share the exchange buffer, the two FP64 forms the second array and the
    recorded measures. The n-th allocation of the first FP64 solve fails: that form launches per
    pass, the others run on chip with every buffer they take."""
    before = fake.fake_null_exchange()
    with _solver(ib3d, grids, (21, 18, 16), ib3d.PREC_FP32DC) as s:
        def solve(precision, kernel):
            s.set_params(precision=precision)
            s.redblack_sor()
            assert kernel in fake.fake_launches().decode()

        solve(ib3d.PREC_FP32DC, "k_resident32")
        fake.fake_fail_in(nth)
        solve(ib3d.PREC_FP64, "k_sor64")
        assert fake.fake_pending_failure() == 0
        solve(ib3d.PREC_FP32DC, "k_resident32")
        solve(ib3d.PREC_FP64_FAST, "k_resident64")
        solve(ib3d.PREC_FP64, "k_sor64")
        solve(ib3d.PREC_FP32DC, "k_resident32")
    assert fake.fake_null_exchange() == before


# the first cells, the ones around 2^30 and the last cell of the largest box
@pytest.mark.parametrize("cell", [0, 63, 64, 2 ** 30 - 1, 2 ** 30, 2 ** 30 + 12345, 2 ** 31 - 1])
def test_four_threads_a_cell_reach_every_cell_of_a_large_box(fake, cell):
    """k_tagging's numbering of cells, with its 256 threads a block."""
    block = cell // 64
    for lane in range(4):
        assert fake.fake_quad_item(block, 256, 4 * (cell % 64) + lane) == cell


def _forcing_is_refused(ib3d, s):
    for call in (s.velocity_forcing, s.pressure_forcing, lambda: s.stress(True), lambda: s.step(True)):
        with pytest.raises(ib3d.IB3DError) as e:
            call()
        assert e.value.code == ib3d.ERR_ARG


@pytest.mark.parametrize("nth", [1, 4, 7])
def test_failed_mesh_ends_the_earlier_search(ib3d, grids, fake, nth):
    """A larger mesh whose arrays cannot be allocated leaves none: what was searched for the
    earlier mesh must not be run on them. The next mesh that fits is searched as ever."""
    cs = grids.case("tiny")
    with ib3d.Solver(cs.x, cs.y, cs.z, ib3d.default_params()) as s:
        s.set_mesh(*grids.icosphere(1, 0.5))
        s.search(cs.box)
        s.velocity_forcing()
        fake.fake_fail_in(nth)
        with pytest.raises(ib3d.IB3DError) as e:
            s.set_mesh(*grids.icosphere(2, 0.5))
        assert e.value.code == ib3d.ERR_CUDA
        _forcing_is_refused(ib3d, s)
        s.set_mesh(*grids.icosphere(2, 0.5))
        s.search(cs.box)
        s.velocity_forcing()


@pytest.mark.parametrize("nth", [1, 2])
def test_failed_search_ends_the_earlier_search(ib3d, grids, fake, nth):
    """The same for a search whose larger box finds no room for its cells' nearest elements, or for
    its scan."""
    z = np.arange(161) * 0.05
    small = [10, 20, 10, 20, 10, 20]
    with ib3d.Solver(z, z, z, ib3d.default_params()) as s:
        s.set_mesh(*grids.icosphere(1, 0.5))
        s.search(small)
        fake.fake_fail_in(nth)
        with pytest.raises(ib3d.IB3DError) as e:
            s.search([1, s.nx + 2, 1, s.ny + 2, 1, s.nz + 2])
        assert e.value.code == ib3d.ERR_CUDA and fake.fake_pending_failure() == 0
        _forcing_is_refused(ib3d, s)
        s.search(small)
        s.velocity_forcing()


@pytest.mark.parametrize("nth", [1, 2, 3, 4])
def test_odd_rows_fall_back_to_the_padded_layout(ib3d, grids, fake, nth):
    """A grid of odd nx needs no packed arrays: where one of the four finds no room, the context is
    created without them and solves in the padded layout. An even nx is refused, as ever."""
    import re
    axes = lambda *n: [grids.tanh_axis(k) for k in n]
    kw = dict(precision=ib3d.PREC_FP32DC, criterion=1, inner_sweeps=32, max_sweeps=100)
    packed = []   # the allocations that may fail
    for k in range(1, 60):
        fake.fake_fail_in(k)
        try:
            ib3d.Solver(*axes(21, 18, 16), **kw).close()
            if fake.fake_pending_failure() == 0:
                packed.append(k)
        except ib3d.IB3DError as e:
            assert e.code == ib3d.ERR_MEMORY
    assert len(packed) == 4, packed
    fake.fake_fail_in(packed[nth - 1])
    with ib3d.Solver(*axes(21, 18, 16), **kw) as s:
        assert fake.fake_pending_failure() == 0
        fake.fake_launches()
        s.redblack_sor()
        names = fake.fake_launches().decode()
        assert re.search(r"k_sor32ILi0", names) and "k_resident32" not in names
    fake.fake_fail_in(packed[nth - 1])
    with pytest.raises(ib3d.IB3DError) as e:
        ib3d.Solver(*axes(20, 18, 16), **kw)
    assert e.value.code == ib3d.ERR_MEMORY
