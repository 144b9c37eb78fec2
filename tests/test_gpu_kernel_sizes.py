"""GPU kernels at the sizes where their tiles, waves and remainders change.

Reduction loops: grids below and above one wave of CTAs (1 and 4 rows per
thread), odd extents, against the oracle's run of the same program.
"""

import pytest

from tests.apprun import assert_lines_close, result_lines, run_app
from tests.opsdump import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("args", [["-nb=1", "-n=1", "-sweeps=2", "-check=1"],
                                  ["-nb=1", "-n=703", "-sweeps=4", "-check=2"],
                                  ["-nb=1", "-n=1021", "-sweeps=4", "-check=2"],
                                  ["-nb=2", "-n=517", "-sweeps=4", "-check=2"]])
def test_reduction_tiles(args):
    """Max residual and sum over blocks of 1 to 1021^2 points: the maxima
    and the printed digits of the sum agree, every dat is bit-identical."""
    gout, gd = run_app("poisson_mb", "b200", args, dump=True)
    cout, cd = run_app("poisson_mb", "oracle", args, dump=True)
    diffs = compare(gd, cd)
    # the boundary values come from sin(): CUDA's and glibc's may differ in
    # the last bit
    assert diffs and max(diffs.values()) <= 1e-12, diffs
    assert_lines_close(result_lines(gout), result_lines(cout), 1e-11)
