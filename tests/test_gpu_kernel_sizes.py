"""GPU kernels at the sizes where their tiles, waves and remainders change.

Reduction loops: grids below and above one wave of CTAs (1 and 4 rows per
thread), odd extents, against the oracle's run of the same program.
"""

import pytest

from tests.apprun import assert_lines_close, result_lines, run_app
from tests.opsdump import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("args", [["-nb=1", "-n=2", "-sweeps=2", "-check=1"],
                                  ["-nb=1", "-n=703", "-sweeps=4", "-check=2"],
                                  ["-nb=1", "-n=1021", "-sweeps=4", "-check=2"],
                                  ["-nb=2", "-n=517", "-sweeps=4", "-check=2"]])
def test_reduction_tiles(args):
    """Max residual and sum over blocks of 2^2 to 1021^2 points: the maxima
    and the printed digits of the sum agree, every dat is bit-identical."""
    gout, gd = run_app("poisson_mb", "b200", args, dump=True)
    cout, cd = run_app("poisson_mb", "oracle", args, dump=True)
    diffs = compare(gd, cd)
    # the boundary values come from sin(): CUDA's and glibc's may differ in
    # the last bit
    assert diffs and max(diffs.values()) <= 1e-12, diffs
    assert_lines_close(result_lines(gout), result_lines(cout), 1e-11)


@pytest.mark.parametrize("n", [5, 9, 20, 70, 700])
def test_reduction_results(n):
    """Every way a result takes to the host (apps/redunit): the oracle's
    lines, digit by digit (the sums are exact in any order)."""
    gout, _ = run_app("redunit", "b200", ["-n=%d" % n])
    cout, _ = run_app("redunit", "oracle", ["-n=%d" % n])
    lines = [l for l in cout.splitlines() if l.startswith("sums")]
    assert len(lines) == 17 + 3 + 3
    assert [l for l in gout.splitlines() if l.startswith("sums")] == lines


@pytest.mark.parametrize("name,args", [
    ("poisson_mb", ["-nb=1", "-n=1921", "-sweeps=2", "-check=1"]),
    ("poisson_mb", ["-nb=1", "-n=2048", "-sweeps=2", "-check=1"]),
    ("heat_cg", ["-n=1301", "-maxit=2", "-prec=both"])])
def test_common_layout_tiles(name, args):
    """Ranges large enough for the kernels of several columns per thread: a
    5-point sweep (4 columns, 2 rows) and the copies, updates and reductions
    of a CG, whole tiles and tiles cut off at the right and upper edge.  The
    sweep's dats equal the oracle's but for the boundary's sin(); the CG's
    dot products are summed in another order, so its FP64 dats agree to 1e-10
    of the field's scale and the mixed form's to 1e-5 (a beta that rounds to
    the other float moves every point by one float ulp)."""
    _, gd = run_app(name, "b200", args, dump=True)
    _, cd = run_app(name, "oracle", args, dump=True)
    diffs = compare(gd, cd, floor_frac=1.0)
    assert diffs
    for dat, d in diffs.items():
        if name == "poisson_mb":
            assert d <= 1e-12, (dat, d)
        else:
            assert d <= (1e-5 if dat in ("x", "r32", "p32", "w32") else 1e-10), (dat, d)


@pytest.mark.parametrize("args", [["-nx=131", "-ny=97", "-nz=151"],
                                  ["-nx=160", "-ny=130", "-nz=100", "-off=1"],
                                  ["-nx=33", "-ny=253", "-nz=239"],
                                  ["-nx=9", "-ny=7", "-nz=5"], ["-nx=1030", "-ny=2", "-nz=70"],
                                  ["-nx=40", "-ny=3", "-nz=900"], ["-nx=3", "-ny=10", "-nz=901"],
                                  ["-nx=257", "-ny=17", "-nz=3"], ["-nx=5000", "-ny=2", "-nz=2"]])
def test_common_layout_rows_in_3d(args):
    """3D loops with several rows per thread (apps/sweep3d: 2 in double, 4 in
    float) over extents that are no multiple of a tile, and thin ones, to which
    the reduction's CTA shape is fitted, through the kernels for dats of one
    layout: dats and reductions as the oracle's, bit for bit."""
    gout, gd = run_app("sweep3d", "b200", args, dump=True)
    cout, cd = run_app("sweep3d", "oracle", args, dump=True)
    diffs = compare(gd, cd)
    assert len(diffs) == 5 and max(diffs.values()) == 0.0, diffs
    lines = [l for l in cout.splitlines() if l.startswith("max")]
    assert lines and [l for l in gout.splitlines() if l.startswith("max")] == lines


LINES = [2, 5, 40, 41, 48, 49, 64, 65, 80, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225, 256,
         257, 511, 1537, 2048, 2049, 4096]


@pytest.mark.parametrize("typ", ["double", "float"])
@pytest.mark.parametrize("solvedim", [0, 1, 2])
@pytest.mark.parametrize("n", LINES)
def test_trid_line_lengths(typ, solvedim, n):
    """Line lengths at the edges of the chunk (5 to 8 points), lane (8, 16,
    32) and segment (256 points, 2 to 16 of them) ranges, unit-stride and
    strided, with and without _Inc, against the numpy Thomas model
    (test_trid_batch: 1e-12 relative, diagonally dominant systems; it solves a
    range of two points less than the shape along x and y)."""
    from tests.test_gpu_cabi import test_trid_batch
    others = [9, 5] if n < 1000 else [9, 4 if solvedim == 0 else 2]
    shape = others[:solvedim] + [n if solvedim == 2 else n + 2] + others[solvedim:]
    for inc in (False, True):
        test_trid_batch(typ, solvedim, inc, tuple(shape))


@pytest.mark.parametrize("typ", ["double", "float"])
@pytest.mark.parametrize("segments", range(2, 17))
def test_trid_segments(typ, segments):
    """Strided lines of 2 to 16 segments (the CTAs of a cluster, which write
    into each other's shared memory), the last segment partly empty and the
    last cluster with fewer lines than it holds, three solves in a row."""
    from tests.test_gpu_cabi import test_trid_batch
    for inc in (False, True, False):
        test_trid_batch(typ, 1, inc, (7, 256 * segments - 35, 2))


@pytest.mark.parametrize("typ", ["double", "float"])
@pytest.mark.parametrize("n", [3, 61, 119, 250, 700, 2500])
def test_trid_offsets_beyond_32_bits(typ, n):
    """Strided lines whose elements lie more than 2^31 apart (the third axis
    strides over 2^31 elements of one sparse buffer that holds every array),
    with and without _Inc, starting at an odd element."""
    import ctypes as C

    import numpy as np
    import torch

    from tests import cabi
    from tests.test_gpu_cabi import thomas
    L = cabi.lib()
    L.ob2_trid_batch.argtypes = [C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int),
                                 C.POINTER(C.c_longlong)] + [C.c_void_p] * 5
    ts, dt = (8, torch.float64) if typ == "double" else (4, torch.float32)
    far, apart, nx = 1 << 31, 1 << 20, 3
    buf = torch.empty(far + 5 * apart, dtype=dt, device="cuda")
    rng = np.random.default_rng(n)
    vals = {k: rng.uniform(-1, 1, (2, n, nx)) + (4.0 if k == "b" else 0.0) for k in "abcdu"}
    view = {k: buf[1 + j * apart:].as_strided((2, n, nx), (far, 7, 1)) for j, k in enumerate("abcdu")}
    strides = (C.c_longlong * 3)(1, 7, far)
    for inc in (False, True):
        for k in "abcdu":
            vals[k] = vals[k].astype(np.float64 if ts == 8 else np.float32)
            view[k].copy_(torch.from_numpy(vals[k]))
        torch.cuda.synchronize()
        p = [view[k].data_ptr() for k in "abcd"] + [view["u"].data_ptr() if inc else None]
        assert L.ob2_trid_batch(ts, 3, 1, cabi.ivec([nx, n, 2]), strides, *p) == 0
        torch.cuda.synchronize()
        got = view["u" if inc else "d"].cpu().numpy()
        want = vals["u"].astype(np.float64) if inc else np.zeros((2, n, nx))
        for z in range(2):
            for x in range(nx):
                want[z, :, x] += thomas(*(vals[k][z, :, x].astype(np.float64) for k in "abcd"))
        if ts == 8:
            np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-13)
        else:  # one rounding to float, after u is added
            np.testing.assert_allclose(got, want, rtol=2.5e-7, atol=1e-6)
    del view, buf
    torch.cuda.empty_cache()


def test_trid_too_long_is_refused():
    """Lines of more than 4096 points: an error, nothing written."""
    import ctypes as C

    from tests import cabi
    L = cabi.lib()
    L.ob2_trid_batch.argtypes = [C.c_int, C.c_int, C.c_int, C.POINTER(C.c_int),
                                 C.POINTER(C.c_longlong)] + [C.c_void_p] * 5
    for dim in (0, 1):
        dims = [3, 3, 1]
        dims[dim] = 4097
        strides = (C.c_longlong * 3)(1, dims[0], dims[0] * dims[1])
        assert L.ob2_trid_batch(8, 3, dim, cabi.ivec(dims), strides, None, None, None, None,
                                None) != 0


BOXES = [(1, 1, 1), (1, 7, 5), (2, 3, 4), (5, 1, 8), (31, 4, 2), (33, 6, 3), (40, 9, 8)]


@pytest.mark.parametrize("soa", [0, 1])
@pytest.mark.parametrize("typ", ["double", "float", "int", "half", "complexd"])
@pytest.mark.parametrize("dim", [1, 2, 3, 5])
def test_slab_fetch_and_set(soa, typ, dim):
    """Boxes of a 3D dat out and back through host buffers: rows from one
    element to the whole width, every component count and element size (2 to
    16 bytes), AoS and SoA; bytes equal to the numpy slice, nothing outside
    the box written."""
    import ctypes as C

    import numpy as np

    from tests import cabi
    L = cabi.lib()
    ts = {"double": 8, "float": 4, "int": 4, "half": 2, "complexd": 16}[typ]
    vp, ip = C.c_void_p, C.POINTER(C.c_int)
    for f in (L.ops_dat_fetch_data_slab_memspace, L.ops_dat_set_data_slab_memspace):
        f.argtypes = [vp, C.c_int, vp, ip, C.c_int]
    n = [40, 9, 8]
    blk = L.ops_decl_block(3, b"box")
    L.ops_set_soa(soa)
    try:
        h = L.ops_decl_dat_char(blk, dim, cabi.ivec(n), cabi.ivec([0] * 3), cabi.ivec([-1] * 3),
                                cabi.ivec([1] * 3), cabi.ivec([1] * 3), None, ts, typ.encode(),
                                b"box")
        rng = np.random.default_rng(dim * 100 + ts)
        model = rng.integers(0, 256, (n[2], n[1], n[0], dim * ts), dtype=np.uint8)
        whole = cabi.ivec([0, n[0], 0, n[1], 0, n[2]])
        L.ops_dat_set_data_slab_memspace(h, 0, model.ctypes.data, whole, 1)
        for k, b in enumerate(BOXES):
            lo = [int(rng.integers(0, n[i] - b[i] + 1)) for i in range(3)]
            r = cabi.ivec([v for i in range(3) for v in (lo[i], lo[i] + b[i])])
            sl = tuple(slice(lo[i], lo[i] + b[i]) for i in (2, 1, 0))
            got = np.empty((b[2], b[1], b[0], dim * ts), np.uint8)
            L.ops_dat_fetch_data_slab_memspace(h, 0, got.ctypes.data, r, 1)
            assert np.array_equal(got, model[sl]), (b, lo)
            new = rng.integers(0, 256, got.shape, dtype=np.uint8)
            L.ops_dat_set_data_slab_memspace(h, 0, new.ctypes.data, r, 1)
            model[sl] = new
            back = np.empty_like(model)
            L.ops_dat_fetch_data_slab_memspace(h, 0, back.ctypes.data, whole, 1)
            assert np.array_equal(back, model), (b, lo)
    finally:
        L.ops_set_soa(0)


def test_slab_of_soa_components_is_one_launch():
    """All components of a SoA dat, and both halves of a complex element, go
    in one launch."""
    import ctypes as C

    import numpy as np
    import torch
    from torch.profiler import ProfilerActivity, profile

    from tests import cabi
    L = cabi.lib()
    vp, ip = C.c_void_p, C.POINTER(C.c_int)
    L.ops_dat_fetch_data_slab_memspace.argtypes = [vp, C.c_int, vp, ip, C.c_int]
    n = [40, 9, 8]
    L.ops_set_soa(1)
    try:
        h = L.ops_decl_dat_char(L.ops_decl_block(3, b"one"), 5, cabi.ivec(n), cabi.ivec([0] * 3),
                                cabi.ivec([-1] * 3), cabi.ivec([1] * 3), cabi.ivec([1] * 3), None,
                                16, b"complexd", b"one")
        out = np.empty((4, 4, 30, 5 * 16), np.uint8)
        torch.zeros(1, device="cuda")
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            L.ops_dat_fetch_data_slab_memspace(h, 0, out.ctypes.data,
                                               cabi.ivec([3, 33, 2, 6, 1, 5]), 1)
            torch.cuda.synchronize()
    finally:
        L.ops_set_soa(0)
    copies = [e for e in prof.events() if "box_copy" in e.name]
    assert len(copies) == 1, [e.name for e in prof.events()]


def test_slab_of_long_rows():
    """Rows of more than one piece (1024 units of 8 bytes), 1D and 2D."""
    import ctypes as C

    import numpy as np

    from tests import cabi
    L = cabi.lib()
    vp, ip = C.c_void_p, C.POINTER(C.c_int)
    for f in (L.ops_dat_fetch_data_slab_memspace, L.ops_dat_set_data_slab_memspace):
        f.argtypes = [vp, C.c_int, vp, ip, C.c_int]
    for n, lo, hi in (([5003], [2], [5001]), ([1025, 3], [0, 1], [1025, 3]),
                      ([4097, 2], [1, 0], [4096, 2])):
        nd = len(n)
        blk = L.ops_decl_block(nd, b"rows")
        d = cabi.Dat(blk, nd, n, [-1] * nd, [1] * nd, "double", "rows")
        a = np.random.default_rng(3).random(n[::-1])
        d.set_interior(a)
        sl = tuple(slice(lo[i], hi[i]) for i in reversed(range(nd)))
        got = np.empty(a[sl].shape)
        r = cabi.ivec([v for i in range(nd) for v in (lo[i], hi[i])])
        L.ops_dat_fetch_data_slab_memspace(d.h, 0, got.ctypes.data, r, 1)
        assert np.array_equal(got, a[sl])
