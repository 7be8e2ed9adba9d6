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
# and the last one L2, where the sweeps go through parts
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


def _rhs(shape, seed=5):
    b = np.zeros(tuple(n + 2 for n in shape), order="F")
    b[1:-1, 1:-1, 1:-1] = np.random.default_rng(seed).standard_normal(shape)
    return b


# blocks of two rows, of several, split along one axis only; odd extents; the test met inside a
# batch (of 16, 32, ... sweeps), at its end, and not at all; residuals checked at every sweep
# and between; a given pc, which the zero start replaces
@pytest.mark.parametrize("shape,criterion,every,eps,cap", [
    ((21, 9, 8), 0, 1, 1e-7, 100000), ((37, 18, 25), 1, 3, 1e-6, 100000), ((8, 41, 5), 1, 1, 1e-6, 100000),
    ((7, 5, 61), 0, 1, 1e-30, 77), ((16, 12, 12), 1, 8, 1e-30, 48), ((16, 12, 12), 1, 5, 1e-30, 33),
    ((130, 40, 31), 0, 1, 1e-30, 40)])
def test_fp64_sweeps_on_chip_are_bit_exact(ib3d, grids, oracle_mod, shape, criterion, every, eps, cap):
    x, y, z = (grids.tanh_axis(n) for n in shape)
    b, pc0 = _rhs(shape), np.asfortranarray(np.random.default_rng(9).standard_normal(tuple(n + 2 for n in shape)))
    o = oracle_mod.Oracle(x, y, z, 100.0, 1.0, omega=1.7, eps=eps, criterion=criterion, max_sweeps=cap,
                          check_every=every)
    o.no_body()
    o.set_field("b", b)
    r = o.redblack_sor(allow_noconv=True)
    p = ib3d.default_params(re=100.0, deltat=1.0, omega=1.7, eps=eps, max_sweeps=cap)
    p.criterion, p.check_every = criterion, every
    s = ib3d.Solver(x, y, z, p)
    s.set_field("b", b)
    s.set_field("pc", pc0)
    g = s.redblack_sor(allow_noconv=True)        # a zero start replaces the given pc
    assert (g["sweeps"], g["final_err"]) == (r["sweeps"], r["final_err"])
    want = o.get_field("pc")
    assert np.array_equal(s.get_field("pc"), want)
    # the fast form: the same method within rounding, amplified by the sweeps
    s.set_params(precision=ib3d.PREC_FP64_FAST)
    f = s.redblack_sor(allow_noconv=True)
    assert abs(f["sweeps"] - r["sweeps"]) <= max(1, every)
    if f["sweeps"] == r["sweeps"]:
        assert np.max(np.abs(s.get_field("pc") - want)) <= 1e-13 * r["sweeps"] * np.max(np.abs(want))
    s.close()


def test_noalloc_solve_on_rows_too_long_for_a_block(ib3d, grids, oracle_mod):
    """Launch per colour pass, capped, against the context's one-array kernel on the same sweeps
    (the two round b/dt - A pc differently)."""
    import torch
    shape = (4200, 9, 7)
    b = _rhs(shape)
    n, want = _capped(ib3d, grids, shape, 48, b, sweep_kernel=1, inner_sweeps=24)
    o = oracle_mod.Oracle(*(grids.tanh_axis(n) for n in shape), 100.0, 1.0)
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v.ravel(order="F"))).cuda()
    A, bd, cd = [dev(np.asarray(o.acoef(q))) for q in range(3)], dev(b), dev(np.zeros(b.shape, np.uint8))
    pc = torch.zeros(b.size, dtype=torch.float64, device="cuda")
    rc = ib3d.lib().ib3d_pressure_solve_noalloc(*shape, *(v.data_ptr() for v in A), cd.data_ptr(), bd.data_ptr(), 1.0,
                                                pc.data_ptr(), 1.85, 1e-30, 48, 24, None, None, None)
    assert (rc, n) == (ib3d.ERR_NOCONV, 48)
    got = pc.cpu().numpy().reshape(b.shape, order="F")
    assert np.max(np.abs(got - want)) <= 1e-6 * np.max(np.abs(want))


# even and odd rows of the on-chip sweeps
@pytest.mark.parametrize("shape", [(21, 10, 13), (64, 33, 31)])
def test_noalloc_solve_meets_the_residual(ib3d, grids, oracle_mod, shape):
    import ctypes as C
    import torch
    x, y, z = (grids.tanh_axis(n) for n in shape)
    o = oracle_mod.Oracle(x, y, z, 100.0, 1.0)
    a = [np.asfortranarray(o.acoef(q)) for q in range(3)]
    b = _rhs(shape)
    cell = np.zeros(b.shape, np.uint8, order="F")
    cell[shape[0] // 3:shape[0] // 3 + 3, 3:5, 3:5] = 1
    dev = lambda v: torch.from_numpy(np.ascontiguousarray(v.ravel(order="F"))).cuda()
    A, bd, cd = [dev(v) for v in a], dev(b), dev(cell)
    pc = torch.zeros(b.size, dtype=torch.float64, device="cuda")
    sweeps, res = np.zeros(1, np.int64), np.zeros(1)
    rc = ib3d.lib().ib3d_pressure_solve_noalloc(
        *shape, A[0].data_ptr(), A[1].data_ptr(), A[2].data_ptr(), cd.data_ptr(), bd.data_ptr(), 1.0, pc.data_ptr(), 1.6,
        1e-6, 2000000, 24, None, sweeps.ctypes.data_as(C.POINTER(C.c_int64)), res.ctypes.data_as(C.POINTER(C.c_double)))
    assert rc == ib3d.OK and res[0] < 1e-6 and sweeps[0] % 24 == 0
    q = pc.cpu().numpy().reshape(b.shape, order="F")
    i = np.s_[1:-1]
    Ap = (a[0][:, 0][:, None, None] * q[:-2, i, i] + a[0][:, 2][:, None, None] * q[2:, i, i]
          + a[1][:, 0][None, :, None] * q[i, :-2, i] + a[1][:, 2][None, :, None] * q[i, 2:, i]
          + a[2][:, 0][None, None, :] * q[i, i, :-2] + a[2][:, 2][None, None, :] * q[i, i, 2:]
          + (a[0][:, 1][:, None, None] + a[1][:, 1][None, :, None] + a[2][:, 1][None, None, :]) * q[i, i, i])
    fluid = cell[i, i, i] == 0
    # the kernel's own residual and this one differ by the rounding of their sums
    scale = np.abs(a[0]).max() + np.abs(a[1]).max() + np.abs(a[2]).max()
    assert np.max(np.abs(b[i, i, i] - Ap)[fluid]) < 1e-6 + 1e-14 * scale * np.max(np.abs(q))
    assert np.all(q[cell != 0] == 0.0)


# launch-per-pass sweeps: whole tiles (256 x 192 x 192; in parts: 512 x 128 x 304), odd ny and nz
# (the march ends on the ghost plane), enough passes in a row
# that a value left over from an earlier pass would show
@pytest.mark.parametrize("shape", [(256, 192, 192), (256, 193, 193), (250, 191, 191), (512, 128, 304), (271, 225, 201)])
def test_passes_read_the_last_pass_only(ib3d, grids, shape):
    b = _rhs(shape)
    want = _capped(ib3d, grids, shape, 75, b, sweep_kernel=1, smooth_sweeps=2, ramp_sweeps=5)
    for kernel in (0, 0, 3, 4):
        got = _capped(ib3d, grids, shape, 75, b, sweep_kernel=kernel, smooth_sweeps=2, ramp_sweeps=5)
        assert got[0] == want[0]
        assert np.array_equal(got[1], want[1]), kernel


# sweeps in parts (grids beyond L2): two parts and more, wide planes (a part is four planes, one sweep
# a group, more blocks than one wave), parts that end off the grid; odd nz; groups cut short
@pytest.mark.parametrize("shape,sweeps", [((1500, 1100, 9), 7), ((384, 256, 255), 43), ((512, 400, 151), 36),
                                          ((300, 290, 301), 17)])
def test_sweeps_in_parts_match_whole_passes(ib3d, grids, shape, sweeps):
    b = _rhs(shape)
    want = _capped(ib3d, grids, shape, sweeps, b, sweep_kernel=3, smooth_sweeps=2, ramp_sweeps=5)
    got = _capped(ib3d, grids, shape, sweeps, b, sweep_kernel=0, smooth_sweeps=2, ramp_sweeps=5)
    assert got[0] == want[0] == sweeps
    assert np.array_equal(got[1], want[1])


# several cells of a colour per thread, so that the warps of a block finish the residual of a
# check apart: a red pass that began before all had read its cells would change the recorded
# measure. Residuals at every sweep and at every third, to the cap (the goal out of reach) and
# to the goal; the fast form against itself.
@pytest.mark.parametrize("shape", [(96, 64, 64), (100, 75, 51)])
@pytest.mark.parametrize("every,eps,cap", [(1, 1e-30, 48), (3, 1e-30, 50), (1, 0.01, 2000), (3, 0.01, 2000)])
def test_fp64_on_chip_residuals_are_of_one_state(ib3d, grids, oracle_mod, shape, every, eps, cap):
    x, y, z = (grids.tanh_axis(n) for n in shape)
    b = _rhs(shape)
    o = oracle_mod.Oracle(x, y, z, 100.0, 1.0, omega=1.7, eps=eps, criterion=1, max_sweeps=cap, check_every=every)
    o.no_body()
    o.set_field("b", b)
    r = o.redblack_sor(allow_noconv=True)
    p = ib3d.default_params(re=100.0, deltat=1.0, omega=1.7, eps=eps, max_sweeps=cap)
    p.criterion, p.check_every = 1, every
    with ib3d.Solver(x, y, z, p) as s:
        s.set_field("b", b)
        for _ in range(8):
            g = s.redblack_sor(allow_noconv=True)
            assert (g["sweeps"], g["final_err"]) == (r["sweeps"], r["final_err"])
        s.set_params(precision=ib3d.PREC_FP64_FAST)
        fast = {(f["sweeps"], f["final_err"]) for f in (s.redblack_sor(allow_noconv=True) for _ in range(8))}
        assert len(fast) == 1, fast


@pytest.fixture(scope="module")
def set_polls(ib3d, tmp_path_factory):
    """Sets the loads after which a context's waits for neighbouring rows give up, and what is added
    to the numbers that they wait for."""
    import ctypes as C
    import pathlib
    import subprocess
    from ib3d_gpu_gb300 import buildlib
    d = tmp_path_factory.mktemp("polls")
    (d / "polls.cpp").write_text('#include "ib3d_internal.cuh"\n'
                                 'extern "C" int set_polls(ib3d_ctx* c, int n, unsigned skew) {\n'
                                 '  const int o = c->polls;\n  c->polls = n;\n  c->poll_skew = skew;\n  return o;\n}\n')
    include = pathlib.Path(buildlib.nvcc()).resolve().parent.parent / "include"
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-I", str(include), "-I", str(buildlib.CSRC), "-o",
                    str(d / "polls.so"), str(d / "polls.cpp")], check=True)
    f = C.CDLL(str(d / "polls.so")).set_polls
    f.argtypes, f.restype = [C.c_void_p, C.c_int, C.c_uint], C.c_int
    return f


# blocks split both ways; the words waited for carry numbers that are 2^31 passes away, so every
# wait runs out at its limit of 256 polls. The error is reported, and the next solve on the same exchange buffer
# has the bits of a solve that never failed
@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("criterion", [0, 1])
def test_wait_that_gives_up_ends_the_solve_with_an_error(ib3d, grids, set_polls, precision, criterion):
    shape = (40, 33, 31)
    x, y, z = (grids.tanh_axis(n) for n in shape)
    p = ib3d.default_params(re=100.0, deltat=1.0, omega=1.7, eps=1e-4, max_sweeps=5000)
    p.precision, p.criterion, p.inner_sweeps = precision, 1 if precision == 1 else criterion, 32
    with ib3d.Solver(x, y, z, p) as s:
        s.set_field("b", _rhs(shape))
        want = s.redblack_sor(), s.get_field("pc")
        usual = set_polls(s._h, 0, 1 << 31)
        for _ in range(2):
            with pytest.raises(ib3d.IB3DError) as e:
                s.redblack_sor()
            assert e.value.code == ib3d.ERR_CUDA and "gave up" in str(e.value)
        set_polls(s._h, usual, 0)
        got = s.redblack_sor(), s.get_field("pc")
    assert (got[0]["sweeps"], got[0]["final_err"]) == (want[0]["sweeps"], want[0]["final_err"])
    assert np.array_equal(got[1], want[1])


# kernel 0 beyond the on-chip sizes, and the forms that never run on chip
@pytest.mark.parametrize("kernel,shape", [(3, (40, 33, 31)), (4, (40, 33, 31)), (0, (256, 192, 192))])
def test_captured_sweeps_follow_the_arrays_that_fused_sweeps_swap(ib3d, grids, kernel, shape):
    """An odd number of fused sweeps leaves the corrections in the other pair of arrays; the
    sweeps captured before must not be replayed on the first pair."""
    x, y, z = (grids.tanh_axis(n) for n in shape)
    p = ib3d.default_params(re=100.0, deltat=1.0, omega=1.85, eps=1e-30, max_sweeps=75)
    p.precision, p.criterion, p.inner_sweeps, p.sweep_kernel = ib3d.PREC_FP32DC, 1, 35, kernel
    with ib3d.Solver(x, y, z, p) as s:
        s.set_field("b", _rhs(shape))
        s.redblack_sor(allow_noconv=True)
        want = s.get_field("pc")
        s.set_params(sweep_kernel=2, max_sweeps=35)
        s.redblack_sor(allow_noconv=True)
        s.set_params(sweep_kernel=kernel, max_sweeps=75)
        s.redblack_sor(allow_noconv=True)
        assert np.array_equal(s.get_field("pc"), want)


def _sweeps_by_hand(a, b, pc, fluid, omega, sweeps):
    """The reference's red-black sweeps in numpy, each operation rounded as the kernels round it:
    pc, the last sweep's largest update, the residual's largest value."""
    i = np.s_[1:-1]
    ax, ay, az = ([v[:, q].reshape(s) for q in range(3)] for v, s in zip(a, ((-1, 1, 1), (1, -1, 1), (1, 1, -1))))
    diag = ax[1] + ay[1] + az[1]
    odd = np.indices(fluid.shape).sum(0) % 2 == 1     # 0-based interior indices: i + j + k is odd for the same cells
    pc = pc.copy(order="F")

    def num():
        n = b[i, i, i] - ax[0] * pc[:-2, i, i] - ax[2] * pc[2:, i, i]
        n = n - ay[0] * pc[i, :-2, i] - ay[2] * pc[i, 2:, i]
        return n - az[0] * pc[i, i, :-2] - az[2] * pc[i, i, 2:]
    for _ in range(sweeps):
        largest = 0.0
        for colour in (odd, ~odd):
            c = pc[i, i, i]
            new = np.where(fluid & colour, (1.0 - omega) * c + omega * (num() / diag), c)
            largest = max(largest, np.abs(new - c).max())
            pc[i, i, i] = new
    return pc, largest, np.abs(num() - diag * pc[i, i, i])[fluid].max()


# solid and immersed-boundary cells across the blocks' edges in y and z, and a start from a given
# pc whose ghost, solid and fluid cells are all nonzero; one batch, two, three (the result in
# either array)
@pytest.mark.parametrize("shape", [(37, 18, 25), (64, 47, 40)])
@pytest.mark.parametrize("criterion,cap", [(0, 13), (0, 40), (1, 13), (1, 70)])
def test_fp64_on_chip_sweeps_from_a_given_pc_around_a_body(ib3d, grids, oracle_mod, shape, criterion, cap):
    x, y, z = (grids.tanh_axis(n) for n in shape)
    nodes, tris = grids.icosphere(2, 0.3)
    b = _rhs(shape)
    pc0 = np.asfortranarray(np.random.default_rng(9).standard_normal(b.shape))
    p = ib3d.default_params(re=100.0, deltat=1.0, omega=1.7, eps=1e-30, max_sweeps=cap)
    p.criterion, p.warm_start = criterion, ib3d.WARM_PREV
    with ib3d.Solver(x, y, z, p) as s:
        s.set_mesh(nodes + 0.5, tris)
        counts = s.search([1, s.nx + 2, 1, s.ny + 2, 1, s.nz + 2])
        assert counts["solid"] > 0 and counts["ib"] > 0
        cell = s.get_search()["cell"]
        s.set_field("b", b)
        s.set_field("pc", pc0)
        g, got = s.redblack_sor(allow_noconv=True), s.get_field("pc")
        s.set_params(precision=ib3d.PREC_FP64_FAST)
        s.set_field("pc", pc0)
        f, fast = s.redblack_sor(allow_noconv=True), s.get_field("pc")
    o = oracle_mod.Oracle(x, y, z, 100.0, 1.0)
    want, update, residual = _sweeps_by_hand([np.asarray(o.acoef(q)) for q in range(3)], b, pc0,
                                             cell[1:-1, 1:-1, 1:-1] == 0, 1.7, cap)
    assert (g["sweeps"], g["final_err"]) == (cap, residual if criterion else update)
    assert np.array_equal(got, want)
    # the contracted form: the same cells, within rounding amplified by the sweeps
    assert f["sweeps"] == cap and np.array_equal(fast[cell != 0], pc0[cell != 0])
    assert np.max(np.abs(fast - want)) <= 1e-13 * cap * np.max(np.abs(want))
