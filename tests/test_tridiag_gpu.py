"""Batched tridiagonal solves on the B200 path vs the CPU oracle (Thomas).

Two kernels: strided sweeps (y, z) run Thomas per line; x sweeps split
each line into chunks (partition method), whose rounding differs from
sequential Thomas. FP64 results agree to 1e-12 relative, FP32 to 2e-4; the
FP64 residual of the solved system is checked at full size."""
import ctypes

import numpy as np
import pytest

from ops_b200 import ops as O
from ops_b200 import seeded

pytestmark = pytest.mark.gpu


def oracle_solve(orc, a, b, c, d, solvedim, u=None):
    nd = a.ndim
    dims = (ctypes.c_int * 3)(*list(reversed(a.shape)), *([1] * (3 - nd)))
    f = orc.oracle_trid_batch_d if a.dtype == np.float64 else orc.oracle_trid_batch_s
    f(a.ctypes.data, b.ctypes.data, c.ctypes.data, d.ctypes.data, None if u is None else u.ctypes.data, nd,
      solvedim, dims, dims)


def padded(t, pad):
    """Copy t into a larger zero array (numpy order) and return the device
    tensor plus the offset view description."""
    import torch
    big = np.zeros(tuple(s + p for s, p in zip(t.shape, pad)), dtype=t.dtype)
    big[tuple(slice(0, s) for s in t.shape)] = t
    return torch.from_numpy(big).cuda()


def run_gpu(a, b, c, d, solvedim, u=None, pad=None):
    import torch
    pad = pad or (0,) * a.ndim
    tens = [padded(t, pad) for t in (a, b, c, d)]
    ut = padded(u, pad) if u is not None else None
    shape_p = tens[0].shape
    dims = list(reversed(a.shape))
    pads = list(reversed(shape_p))
    sysd = dict(a=tens[0].data_ptr(), b=tens[1].data_ptr(), c=tens[2].data_ptr(), d=tens[3].data_ptr(),
                u=ut.data_ptr() if ut is not None else None, dims=dims, pads=pads)
    O.trid_batch(a.itemsize, solvedim, [sysd], None)
    torch.cuda.synchronize()
    sl = tuple(slice(0, s) for s in a.shape)
    return tens[3].cpu().numpy()[sl], (ut.cpu().numpy()[sl] if ut is not None else None)


@pytest.mark.parametrize("dtype,rtol", [(np.float64, 1e-12), (np.float32, 2e-4)])
@pytest.mark.parametrize("solvedim", [0, 1, 2])
@pytest.mark.parametrize("shape,pad", [((23, 29, 37), (0, 2, 3)), ((3, 300, 17), (1, 0, 5)), ((9, 8, 256), (0, 0, 0))])
def test_strided_batch_matches_oracle(gpu_runtime, orc, dtype, rtol, solvedim, shape, pad):
    if solvedim == 0 and shape[2] > 512:
        pytest.skip("x line longer than the tile kernel's maximum")
    a, b, c, d = seeded.trid_system(shape, solvedim, 11, dtype)
    x, _ = run_gpu(a, b, c, d, solvedim, pad=pad)
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, solvedim)
    np.testing.assert_allclose(x, ref, rtol=rtol, atol=rtol * np.abs(ref).max())


@pytest.mark.parametrize("dtype,rtol", [(np.float64, 1e-12), (np.float32, 2e-4)])
@pytest.mark.parametrize("n,inc", [(1, False), (8, False), (37, True), (130, False), (16, True)])
def test_many_x_lines_match_oracle(gpu_runtime, orc, dtype, rtol, n, inc):
    """x sweeps over 20012 lines of one to 130 rows (many tiles of the
    partition kernel), padding and the _Inc form against the oracle."""
    shape = (4, 5003, n)
    a, b, c, d = seeded.trid_system(shape, 0, 21 + n, dtype)
    u = seeded.uniform(5, np.arange(d.size, dtype=np.uint64), -1, 1).reshape(d.shape).astype(dtype) if inc else None
    dg, ug = run_gpu(a, b, c, d, 0, u=u, pad=(0, 1, 3))
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, 0)
    if inc:
        assert np.array_equal(dg, d)
        np.testing.assert_allclose(ug, u + ref, rtol=rtol, atol=rtol * np.abs(ref).max())
    else:
        np.testing.assert_allclose(dg, ref, rtol=rtol, atol=rtol * np.abs(ref).max())


@pytest.mark.parametrize("solvedim", [0, 1, 2])
def test_inc_form(gpu_runtime, orc, solvedim):
    a, b, c, d = seeded.trid_system((11, 13, 70), solvedim, 4)
    u = seeded.uniform(9, np.arange(d.size, dtype=np.uint64), -1, 1).reshape(d.shape)
    dg, ug = run_gpu(a, b, c, d, solvedim, u=u)
    assert np.array_equal(dg, d)
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, solvedim)
    np.testing.assert_allclose(ug, u + ref, rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 15, 16, 17, 31, 63, 64, 65, 127, 128, 129, 200, 255, 256, 257, 700])
@pytest.mark.parametrize("solvedim", [0, 1])
@pytest.mark.parametrize("warp", [-1, 0, 1])
def test_line_lengths(gpu_runtime, orc, n, solvedim, warp):
    """x lines: the warp-per-line kernel (4 or 8 rows a lane, lines up to
    256 rows) and the shared-memory tile kernel, each forced and as chosen
    by line length; y lines: the line kernel."""
    if solvedim == 1 and warp != -1:
        pytest.skip("the option steers x sweeps only")
    shape = (5, n) if solvedim == 0 else (n, 7)
    a, b, c, d = seeded.trid_system(shape, solvedim, n)
    O.set_option("trid_warp", warp)
    try:
        x, _ = run_gpu(a, b, c, d, solvedim)
    finally:
        O.set_option("trid_warp", -1)
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, solvedim)
    np.testing.assert_allclose(x, ref, rtol=1e-12, atol=1e-13)


@pytest.mark.parametrize("n", [300, 1000, 4099])
def test_long_strided_lines(gpu_runtime, orc, n):
    """y lines of any length (Thomas per line, scratch sized by the call)."""
    a, b, c, d = seeded.trid_system((n, 33), 1, n)
    x, _ = run_gpu(a, b, c, d, 1, pad=(0, 3))
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, 1)
    np.testing.assert_allclose(x, ref, rtol=1e-12, atol=1e-13)


@pytest.mark.parametrize("solvedim", [0, 1, 2])
def test_uneven_batch_one_launch(gpu_runtime, orc, solvedim):
    """Blocks of different edge sizes solved in a single persistent launch."""
    import torch
    rng_sizes = [(7, 19, 33), (32, 40, 50), (61, 5, 12), (13, 64, 100), (2, 3, 4), (40, 40, 40)]
    systems, host, dev = [], [], []
    for i, shp in enumerate(rng_sizes):
        a, b, c, d = seeded.trid_system(shp, solvedim, 100 + i)
        t = [torch.from_numpy(v).cuda() for v in (a, b, c, d)]
        dev.append(t)
        host.append((a, b, c, d))
        systems.append(dict(a=t[0].data_ptr(), b=t[1].data_ptr(), c=t[2].data_ptr(), d=t[3].data_ptr(), u=None,
                            dims=list(reversed(shp)), pads=list(reversed(shp))))
    O.reset_counters()
    O.trid_batch(8, solvedim, systems, None)
    torch.cuda.synchronize()
    assert O.counters()["kernels"] == 1
    for (a, b, c, d), t in zip(host, dev):
        ref = d.copy()
        oracle_solve(orc, a, b, c, ref, solvedim)
        np.testing.assert_allclose(t[3].cpu().numpy(), ref, rtol=1e-12, atol=1e-13)


def test_dat_api_with_range(gpu_runtime, orc):
    """ops_tridMultiDimBatch on dats over a sub-range (offset from the range
    as ops_tridiag.cpp:109-119 computes it), then _Inc along z."""
    nx, ny, nz = 20, 18, 16
    blk = O.ops_decl_block(3, "adi")
    a, b, c, d = seeded.trid_system((nz, ny, nx), 1, 7)
    mk = lambda v, name: O.ops_decl_dat(blk, 1, [nx, ny, nz], [0, 0, 0], [-1, -1, -1], [1, 1, 1],
                                       np.pad(v, 1), "double", name)
    da, db, dc, dd = mk(a, "a"), mk(b, "b"), mk(c, "c"), mk(d, "d")
    rng = [2, 15, 1, 17, 3, 12]
    O.ops_tridMultiDimBatch(3, 1, rng, da, db, dc, dd)
    got = O.ops_dat_fetch_data(dd)[1:-1, 1:-1, 1:-1]
    sub = (slice(rng[4], rng[5]), slice(rng[2], rng[3]), slice(rng[0], rng[1]))
    ref = d.copy()
    ra, rb, rc, rd = (np.ascontiguousarray(t[sub]) for t in (a, b, c, ref))
    oracle_solve(orc, ra, rb, rc, rd, 1)
    expect = d.copy()
    expect[sub] = rd
    np.testing.assert_allclose(got, expect, rtol=1e-12, atol=1e-13)
    u = mk(np.zeros_like(d), "u")
    O.ops_tridMultiDimBatch_Inc(3, 2, [0, nx, 0, ny, 0, nz], da, db, dc, dd, u)
    gu = O.ops_dat_fetch_data(u)[1:-1, 1:-1, 1:-1]
    ref2 = got.copy()
    oracle_solve(orc, a, b, c, ref2, 2)
    np.testing.assert_allclose(gu, ref2, rtol=1e-11, atol=1e-12)


def test_full_size_256_cube_residual(gpu_runtime):
    """Config-3 single block: 256^3 FP64, each direction; ||Ax - d||_inf / ||d||_inf."""
    import torch
    n = 256
    for solvedim in (0, 1, 2):
        a, b, c, d = seeded.trid_system((n, n, n), solvedim, 3 + solvedim)
        x, _ = run_gpu(a, b, c, d, solvedim)
        ax = 2 - solvedim
        xm = np.moveaxis(x, ax, -1)
        am, bm, cm, dm = (np.moveaxis(t, ax, -1) for t in (a, b, c, d))
        r = bm * xm - dm
        r[..., 1:] += am[..., 1:] * xm[..., :-1]
        r[..., :-1] += cm[..., :-1] * xm[..., 1:]
        assert np.abs(r).max() / np.abs(dm).max() < 1e-14


@pytest.mark.parametrize("dtype,rtol", [(np.float64, 1e-12), (np.float32, 2e-4)])
@pytest.mark.parametrize("inc", [False, True])
def test_more_strided_lines_than_threads(gpu_runtime, orc, dtype, rtol, inc):
    """y sweeps of uneven systems in one launch with more groups of 16 lines
    than the grid has warps (a thread takes several lines and reuses its
    scratch), line counts that leave a group part empty, odd, even and one-row
    lines."""
    import torch
    shapes = [(3, 41, 9001), (1, 1, 333), (2, 40, 16), (5, 7, 5003)]
    sets, systems = [], []
    for i, shape in enumerate(shapes):
        a, b, c, d = seeded.trid_system(shape, 1, 31 + i, dtype)
        u = seeded.uniform(7 + i, np.arange(d.size, dtype=np.uint64), -1, 1).reshape(d.shape).astype(dtype)
        t = [torch.from_numpy(v).cuda() for v in (a, b, c, d, u)]
        sets.append(((a, b, c, d, u), t))
        systems.append(dict(a=t[0].data_ptr(), b=t[1].data_ptr(), c=t[2].data_ptr(), d=t[3].data_ptr(),
                            u=t[4].data_ptr() if inc else None, dims=list(shape[::-1]), pads=list(shape[::-1])))
    O.trid_batch(np.dtype(dtype).itemsize, 1, systems, None)
    torch.cuda.synchronize()
    for (a, b, c, d, u), t in sets:
        ref = d.copy()
        oracle_solve(orc, a, b, c, ref, 1)
        if inc:
            assert np.array_equal(t[3].cpu().numpy(), d)
            ref = u + ref
        np.testing.assert_allclose(t[4 if inc else 3].cpu().numpy(), ref, rtol=rtol, atol=rtol * np.abs(ref).max())


@pytest.mark.parametrize("dtype,rtol", [(np.float64, 1e-12), (np.float32, 2e-4)])
@pytest.mark.parametrize("inc", [False, True])
@pytest.mark.parametrize("solvedim", [1, 2])
@pytest.mark.parametrize("n", [2, 3, 5, 16, 17, 64, 101])
def test_strided_lines_with_pivots_from_the_top_only(gpu_runtime, orc, dtype, rtol, inc, solvedim, n):
    """Lines whose elimination from the last row meets a vanishing or tiny
    pivot (b_{n-1} = 0, b_{n-1} = a rounding unit, a singular trailing 2 x 2
    block), between ordinary ones of the same group of 16. From the top they
    are as well conditioned as the rest: |c'| < 1 up to the last rows."""
    lines = 37
    a, b, c, d = seeded.trid_system((lines, n), 1, 3 + n, dtype)
    k = np.arange(lines) % 4
    a[k > 0, n - 1] = 1.0
    b[k == 1, n - 1] = 0.0
    b[k == 2, n - 1] = np.finfo(dtype).eps
    if n > 3:
        for arr, v in ((b, n - 2), (c, n - 2), (b, n - 1)):
            arr[k == 3, v] = 1.0
    u = seeded.uniform(5, np.arange(d.size, dtype=np.uint64), -1, 1).reshape(d.shape).astype(dtype)
    # the solve dimension along y (z = 1) or z (y = 1), the lines along x
    shape = (1, n, lines) if solvedim == 1 else (n, 1, lines)
    a, b, c, d, u = (np.ascontiguousarray(v.T).reshape(shape) for v in (a, b, c, d, u))
    x, ug = run_gpu(a, b, c, d, solvedim, u=u if inc else None)
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, solvedim)
    assert np.isfinite(ref).all()
    if inc:
        assert np.array_equal(x, d)
        x, ref = ug, u + ref
    np.testing.assert_allclose(x, ref, rtol=rtol, atol=rtol * np.abs(ref).max())


@pytest.mark.parametrize("dtype,rtol,power", [(np.float64, 1e-12, 600), (np.float32, 2e-4, 80)])
@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("solvedim", [0, 1, 2])
def test_rows_of_any_scale(gpu_runtime, orc, dtype, rtol, power, sign, solvedim):
    """Rows scaled by a power of two whose square leaves the type's range: the
    solution is that of the unscaled rows."""
    shape = (9, 14, 33)
    a, b, c, d = seeded.trid_system(shape, solvedim, 17, dtype)
    s = dtype(2.0) ** (sign * power)
    x, _ = run_gpu(a * s, b * s, c * s, d * s, solvedim)
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, solvedim)
    np.testing.assert_allclose(x, ref, rtol=rtol, atol=rtol * np.abs(ref).max())


def test_scratch_of_uneven_strided_batches(gpu_runtime, tmp_path):
    """A few long lines beside many short ones, and systems of three lines:
    the y sweep keeps no more scratch than every line's c' and d' (in a process
    of its own: the scratch outlives a call), and solves them all."""
    import subprocess
    import sys
    code = """
import ctypes, sys
import numpy as np, torch
import oracle
from ops_b200 import ops as O, seeded
shapes = [(1, 256, 65536), (1, 200000, 16)] + [(1, 20001, 3)] * 40
O.ops_init(0, 0)
sets = []
for i, shape in enumerate(shapes):
    h = seeded.trid_system(shape, 1, 50 + i)
    sets.append((h, [torch.from_numpy(v).cuda() for v in h]))
def systems(some):
    return [dict(a=t[0].data_ptr(), b=t[1].data_ptr(), c=t[2].data_ptr(), d=t[3].data_ptr(), u=None,
                 dims=list(h[0].shape[::-1]), pads=list(h[0].shape[::-1])) for h, t in some]
first = seeded.trid_system((1, 8, 16), 1, 1)
O.trid_batch(8, 1, systems([(first, [torch.from_numpy(v).cuda() for v in first])]), None)
torch.cuda.synchronize()
free = torch.cuda.mem_get_info()[0]
O.trid_batch(8, 1, systems(sets), None)
torch.cuda.synchronize()
kept = free - torch.cuda.mem_get_info()[0]
rows = sum(z * y * x for z, y, x in shapes)
assert kept <= 16 * rows + (32 << 20), (kept, 16 * rows)
f = oracle.lib().oracle_trid_batch_d
for (a, b, c, d), t in sets:
    ref = d.copy()
    dims = (ctypes.c_int * 3)(*a.shape[::-1])
    f(a.ctypes.data, b.ctypes.data, c.ctypes.data, ref.ctypes.data, None, 3, 1, dims, dims)
    np.testing.assert_allclose(t[3].cpu().numpy(), ref, rtol=1e-12, atol=1e-12 * np.abs(ref).max())
"""
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("dtype,rtol", [(np.float64, 1e-12), (np.float32, 2e-4)])
@pytest.mark.parametrize("inc", [False, True])
@pytest.mark.parametrize("n", [1, 2, 4, 5, 8, 9, 15, 16, 17, 31, 32, 33])
def test_short_lines_in_great_number(gpu_runtime, orc, dtype, rtol, inc, n):
    """Short strided lines, more than one for every thread of a CTA an SM, at
    the edges of their kernel's sizes, along y and along z, alone and beside
    shorter and longer systems. a_0 and c_{n-1} are not read."""
    import torch
    for solvedim, shapes in ((1, [(3, n, 6500)]), (2, [(n, 200, 100)]),
                             (1, [(1, n, 19000), (2, 70, 33), (1, 1, 5), (1, 3, 700), (1, n, 17)])):
        sets, systems = [], []
        for i, shape in enumerate(shapes):
            a, b, c, d = seeded.trid_system(shape, solvedim, 90 + n + i, dtype)
            u = seeded.uniform(7 + i, np.arange(d.size, dtype=np.uint64), -1, 1).reshape(shape).astype(dtype)
            an, cn, ax = a.copy(), c.copy(), 2 - solvedim
            an[(slice(None),) * ax + (0,)] = np.nan
            cn[(slice(None),) * ax + (-1,)] = np.nan
            t = [torch.from_numpy(v).cuda() for v in (an, b, cn, d, u)]
            sets.append(((a, b, c, d, u), t))
            systems.append(dict(a=t[0].data_ptr(), b=t[1].data_ptr(), c=t[2].data_ptr(), d=t[3].data_ptr(),
                                u=t[4].data_ptr() if inc else None, dims=list(shape[::-1]), pads=list(shape[::-1])))
        O.trid_batch(np.dtype(dtype).itemsize, solvedim, systems, None)
        torch.cuda.synchronize()
        for (a, b, c, d, u), t in sets:
            ref = d.copy()
            oracle_solve(orc, a, b, c, ref, solvedim)
            if inc:
                assert np.array_equal(t[3].cpu().numpy(), d)
                ref = u + ref
            np.testing.assert_allclose(t[4 if inc else 3].cpu().numpy(), ref, rtol=rtol, atol=rtol * np.abs(ref).max())


@pytest.mark.parametrize("dtype,rtol", [(np.float64, 1e-12), (np.float32, 2e-4)])
@pytest.mark.parametrize("inc", [False, True])
@pytest.mark.parametrize("n", [17, 33, 39, 40, 41, 63, 64, 65])
def test_more_than_a_wave_of_lines_of_few_rows(gpu_runtime, orc, dtype, rtol, inc, n):
    """Lines of up to 64 rows, more than a wave of the line kernel's usual
    stages: stages of four rows, at the edges of a half line's."""
    shape = (3, n, 10001)
    a, b, c, d = seeded.trid_system(shape, 1, 60 + n, dtype)
    u = seeded.uniform(5, np.arange(d.size, dtype=np.uint64), -1, 1).reshape(shape).astype(dtype) if inc else None
    x, ug = run_gpu(a, b, c, d, 1, u=u, pad=(0, 0, 3))
    ref = d.copy()
    oracle_solve(orc, a, b, c, ref, 1)
    if inc:
        assert np.array_equal(x, d)
        x, ref = ug, u + ref
    np.testing.assert_allclose(x, ref, rtol=rtol, atol=rtol * np.abs(ref).max())
