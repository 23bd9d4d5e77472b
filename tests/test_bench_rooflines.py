"""The kernels whose roofline the benchmark reports are launches of the library, with work and a limiter stated."""
import glob
import os
import re
import sys

sys.path.insert(0, os.path.join(os.path.dirname(__file__), ".."))
import bench  # noqa: E402


def test_rooflines_are_of_launched_kernels():
    root = os.path.join(os.path.dirname(__file__), "..", "spin_based_neural_network_gb300", "csrc")
    launched = set()
    for f in glob.glob(os.path.join(root, "*.cu")):
        launched |= set(re.findall(r'NQS_LAUNCH\("(\w+)"\)', open(f).read()))
    work = bench.algorithmic_work(4096, 1120)
    for name in bench.ROOFLINES:
        assert name in launched and name in work and name in bench.LIMITERS
    # FP64 Cholesky and two triangular solves of the sample-space system, 2 flops per FMA
    assert work["chol_solve_fp64"] == (4096 ** 3 / 3 + 2 * 4096 ** 2, "fp64")
