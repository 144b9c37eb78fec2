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


LINES = [2, 5, 40, 41, 48, 49, 64, 65, 80, 96, 97, 128, 129, 160, 161, 192, 193, 224, 225, 256,
         257, 511, 1537, 2048, 2049, 4096]


@pytest.mark.parametrize("typ", ["double", "float"])
@pytest.mark.parametrize("solvedim", [0, 1, 2])
@pytest.mark.parametrize("n", LINES)
def test_trid_line_lengths(typ, solvedim, n):
    """Line lengths at the edges of the chunk (5 to 8 points), lane (8, 16,
    32) and segment (256 points, 2 to 16 of them) ranges, unit-stride and
    strided, with and without _Inc, against the numpy Thomas model
    (test_trid_batch: 1e-12 relative, diagonally dominant systems)."""
    from tests.test_gpu_cabi import test_trid_batch
    others = [9, 5] if n < 1000 else [9, 2]
    shape = others[:solvedim] + [n] + others[solvedim:]
    for inc in (False, True):
        test_trid_batch(typ, solvedim, inc, tuple(shape))


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
